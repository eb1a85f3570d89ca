"""What the timing calls report: mhd_time_steps times steps and nothing else."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32])
def test_time_steps_leaves_out_the_building_of_graphs(pkg, lib, n):
    """The first call that runs on the chained graph takes as long as the next ones: capture and
    instantiation come before the timed region (inside it they added 0.22 ms, 11 % of 64 steps at
    16^3).  The limit, 5 %, is half of that; the calls themselves agree to within 0.5 %."""
    with pkg.Problem(pkg.GPU(0), nx=n, nu=1e-3, eta=1e-3, dt=1e-4) as p:
        for _ in range(8):
            pkg.stepforward(p, 1)
        pkg._lib.check(lib.mhd_synchronize(p.handle))
        ms = []
        for _ in range(6):
            out = C.c_double()
            pkg._lib.check(lib.mhd_time_steps(p.handle, 64, C.byref(out)))
            ms.append(out.value)
    assert ms[0] < 1.05 * min(ms[1:]), ms
