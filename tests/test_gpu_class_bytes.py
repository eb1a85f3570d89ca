"""mhd_kernel_class_bytes against the arrays that each kernel class reads and writes.

Per instance, with c = 8 bytes a complex value: S = one field of retained modes, Z = one field after
the z transform, P = the half-spectrum rows of one field; nin fields in and nout product planes out."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _bytes(pkg, lib, prob):
    out = {}
    for c in range(lib.mhd_kernel_class_count()):
        b = C.c_double()
        pkg._lib.check(lib.mhd_kernel_class_bytes(prob.handle, c, C.byref(b)))
        out[lib.mhd_kernel_class_name(c).decode()] = b.value
    return out


@pytest.mark.parametrize("scheme", ["RK4", "LSRK4"])
@pytest.mark.parametrize("form", ["mhd", "hd", "mhdvp", "hdvp"])
@pytest.mark.parametrize("n", [16, 64, 96, 128, 256])
def test_bytes_of_the_launched_kernels(pkg, lib, n, form, scheme):
    hd, vp = form.startswith("hd"), form.endswith("vp")
    kx, kp, kn = C.c_int(), C.c_int(), C.c_int()
    pkg._lib.check(lib.mhd_kept_modes(n, C.byref(kx), C.byref(kp), C.byref(kn)))
    k2, c = kp.value + kn.value, 8.0
    S, Z, P, H = k2 * k2 * kx.value * c, n * k2 * kx.value * c, n * n * kx.value * c, k2 * k2 * c
    nin, nout = (3, 8 if vp else 5) if hd else (6, 14 if vp else 8)
    # state arrays a stage update reads and writes (stage state, solution, accumulator)
    stages = [3, 5, 5, 4] if scheme == "RK4" else [3, 4, 4, 4, 4]
    mean = lambda v: sum(v) / len(v)  # noqa: E731
    with pkg.Problem(pkg.GPU(0), nx=n, nu=1e-3, eta=0.0 if hd else 1e-3, dt=1e-3, stepper=scheme, B_field=not hd,
                     VP_method=vp) as p:
        got = _bytes(pkg, lib, p)
    if n <= 64:    # the stage update and the next inverse transforms in one launch, the last update alone
        want = {"z_inverse": (nout + mean(stages[:-1]) * nin) * S + nin * P, "z_forward": nout * (P + S),
                "rk_epilogue": (nout + stages[-1] * nin) * S, "y_inverse": 0, "y_forward": 0}
    elif n <= 128:  # both transforms of a plane in one launch; the forward one also copies H of the kx = 0 plane
        want = {"z_inverse": nin * (S + P), "z_forward": nout * (P + S) + 2 * nin * H,
                "rk_epilogue": (nout + mean(stages) * nin) * S + nin * H, "y_inverse": 0, "y_forward": 0}
    else:
        want = {"z_inverse": nin * (S + Z), "y_inverse": nin * (Z + P), "y_forward": nout * (P + Z),
                "rk_epilogue": (nout + mean(stages) * nin) * S + nin * H}
    # rows read and written; the hydrodynamic rows that are no tiles (16^3, 256^3) write a sixth slot of zeros
    xout = 6 if form == "hd" and n in (16, 256) else nout
    want["x_fused"] = (nin + xout) * P + (4 * n ** 3 if vp else 0)  # and the mask
    for name, b in want.items():
        assert got[name] == pytest.approx(b, rel=1e-12), name
