"""Plane passes and x-row tiles of the small grids: every kernel variant of every form, at every
size they are compiled for, against the FP64 oracle's right-hand side (relative L2 <= 1e-5 on the
retained band, the tolerance of the other right-hand-side tests), and the fused stage update of
both schemes against the oracle's steps.  The kept counts of these sizes end inside, at and next
to the transform groups, rows and column rounds of the kernels."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _problem(pkg, mo, n, form, scheme="RK4", dt=1e-3):
    g = mo.Grid(n)
    hd, vp = form.startswith("hd"), form.endswith("vp")
    s = mo.random_spectrum_state(g, seed=300 + n).astype(np.complex64)
    if hd:
        s[3:] = 0
    prob = pkg.Problem(pkg.GPU(0), nx=n, Lx=2 * math.pi, nu=1e-3, eta=0.0 if hd else 2e-3, dt=dt, stepper=scheme,
                       B_field=not hd, VP_method=vp)
    prob.set_sol(s[:prob.nfields].T)
    pen = None
    if vp:
        x, y, z = g.mesh()
        chi = (0.5 * (1 - np.tanh((np.sqrt(x ** 2 + (y - 0.3) ** 2 + z ** 2) - 1.2) / 0.25))).astype(np.float32)
        wall = tuple((0.3 * (i + 1) * np.sin(x + i) * np.cos(y - z)).astype(np.float32) for i in range(3))
        prob.set_vp(chi.T, U0=tuple(a.T for a in wall))
        pen = dict(chi=chi.astype(np.float64), U0=tuple(a.astype(np.float64) for a in wall))
    return g, s, prob, pen


@pytest.mark.parametrize("form", ["mhd", "hd", "mhdvp", "hdvp"])
@pytest.mark.parametrize("n", [16, 32, 48, 64, 96, 128])
def test_every_variant_of_every_form(pkg, mo, n, form):
    g, s, prob, pen = _problem(pkg, mo, n, form)
    ref = np.zeros(s.shape, dtype=np.complex128)
    mo.calcN_fast(ref, s.astype(np.complex128), g, 1e-3, 0.0 if form.startswith("hd") else 2e-3,
                  vp=None if pen is None else dict(pen, dt=1e-3))
    mask, nf = g.retained_mask(), prob.nfields
    with prob:
        for cls, (selected, names) in pkg.variants(prob).items():
            for i, name in enumerate(names):
                try:
                    pkg.select_variant(prob, cls, i)
                except pkg.MHDError:
                    continue  # another form's variant
                got = prob.rhs_c()
                err = mo.rel_l2(got, ref[:nf], mask)
                assert err < TOL, f"{cls} {name}: rel L2 {err:.2e}"
                assert not got[:, ~mask].any()
            pkg.select_variant(prob, cls, names.index(selected))


@pytest.mark.parametrize("scheme", ["RK4", "LSRK4"])
@pytest.mark.parametrize("n", [16, 48, 64, 96, 128])
def test_steps(pkg, mo, n, scheme):
    g, s, prob, _ = _problem(pkg, mo, n, "mhd", scheme)
    with prob:
        pkg.stepforward(prob, 2)
        got = prob.sol_c()
    st = mo.Stepper(g, 1e-3, 2e-3, 1e-3, scheme, literal=False)
    ref = s.astype(np.complex128)
    for _ in range(2):
        st.stepforward(ref)
    assert mo.rel_l2(got, ref, g.retained_mask()) < TOL


@pytest.mark.parametrize("n,scheme,cfl", [(16, "RK4", False), (32, "LSRK4", True), (48, "RK4", True), (64, "LSRK4", False)])
def test_chained_steps_equal_single_ones(pkg, mo, n, scheme, cfl):
    """One call of many steps runs on graphs of several chained steps, single calls on the graph of
    one: the states, clocks and forcing draws agree bit for bit."""
    got = []
    for calls in ((100,), (1,) * 100):
        _, _, prob, _ = _problem(pkg, mo, n, "mhd", scheme, dt=1e-4)
        with prob:
            pkg.SetUpFk(prob, P=1e-6, seed=5)
            if cfl:
                pkg._lib.check(prob._lib.mhd_set_cfl(prob.handle, 1, 0.2))
            for k in calls:
                pkg.stepforward(prob, k)
            got.append((prob.sol_c(), prob.clock.t, prob.clock.step))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


@pytest.mark.parametrize("form,cfl", [("mhd", True), ("mhdvp", False), ("mhdvp", True)])
def test_runs_on_kept_graphs_equal_runs_on_new_ones(pkg, mo, form, cfl):
    """Runs after one another keep the step's graphs: states, clocks and recorded diagnostics agree bit
    for bit with those of a handle whose graphs are dropped before every run (by selecting the
    variant it has)."""
    got = []
    for fresh in (False, True):
        _, _, prob, _ = _problem(pkg, mo, 32, form, dt=1e-4)
        with prob:
            out = []
            names = pkg.variants(prob)["x_fused"]
            for steps, freq in ((3, 2), (4, 0), (3, 2), (5, 1), (3, 1)):
                if fresh:
                    pkg.select_variant(prob, "x_fused", names[1].index(names[0]))
                pkg.TimeIntegrator(prob, math.inf, steps - 1, usr_dt=0.0 if cfl else 1e-4, diag_freq=freq)
                if freq:
                    out.append(prob.diagnostic_history())
                pkg.stepforward(prob, 2)
                out += [prob.sol_c(), np.array([prob.clock.t, prob.clock.dt])]
            got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("order,dtype", [("F", np.float32), ("C", np.float32), ("F", np.float64)])
def test_vars_arrays_in_place_and_replaced(pkg, mo, order, dtype):
    """SetUpProblemIC and updatevars fill the vars arrays in place where their memory is the library's
    layout, and through a copy where the caller put another kind of array there: same values, and
    the fields handed in stay as they were (also when they are the vars arrays)."""
    n = 32
    _, s, prob, _ = _problem(pkg, mo, n, "mhd")
    rng = np.random.default_rng(0)
    f = rng.standard_normal((n, n, n)).astype(np.float32)
    with prob:
        for name in ("ux", "bz"):
            setattr(prob.vars, name, np.zeros((n, n, n), dtype=dtype, order=order))
        keep = f.copy()
        pkg.SetUpProblemIC(prob, ux=f, bz=np.asfortranarray(f))
        assert np.array_equal(f, keep) and np.array_equal(prob.vars.ux, f) and np.array_equal(prob.vars.bz, f)
        pkg.SetUpProblemIC(prob, ux=prob.vars.ux)
        assert np.array_equal(prob.vars.ux, f)
        arrays = [prob.vars.ux, prob.vars.by]
        pkg.updatevars(prob)
        assert prob.vars.ux is arrays[0] and prob.vars.by is arrays[1]
        for i, name in enumerate(pkg.FIELDS):
            assert np.array_equal(getattr(prob.vars, name), prob.physical_c(i).T)


@pytest.mark.parametrize("n,cap", [(16, 33), (32, 24), (48, 3), (64, 12), (96, 2), (128, 2)])
def test_single_slot_transforms_of_the_last_slots(pkg, mo, n, cap):
    """Single-slot launches cover the whole capacity: the instances past the slot stay inside the work
    lists and the pools, and the last slots' fields and diagnostics equal a single problem's."""
    g, s, prob, _ = _problem(pkg, mo, n, "mhd")
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, n, n)).astype(np.float32)
    batch = pkg.Batch(n, cap, stepper="RK4")
    with prob:
        for _ in range(cap):
            batch.add(1e-3, 2e-3, 1e-3)
        prob.set_physical_c(0, f)
        for slot in sorted({0, cap // 2, cap - 1}):
            batch.set_state(slot, s)
            batch.set_physical(slot, 0, f)
            assert np.array_equal(batch.get_physical(slot, 0), prob.physical_c(0))
            a, b = batch.diagnostics(slot), prob.diagnostics()
            assert (a.E_u, a.E_B, a.H_c, a.nonfinite) == (b.E_u, b.E_B, b.H_c, b.nonfinite)
    batch.close()
