"""Which entry of the tuning file a handle takes: grid size, precision, penalisation, field set and, where
the defaults of single problems and batches differ (plane passes), the capacity.  Each check runs in a
process of its own, so that no selection of another test is known."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import math, os, sys
sys.path.insert(0, {root!r})
import numpy as np, torch
import __graft_entry__ as ge
pkg = ge.load_package()
gpu = torch.cuda.get_device_properties(0)
def names(o):
    return {{c: v[0] for c, v in pkg.variants(o).items()}}
def other(o, cls, default):
    # a variant of the class that the handle accepts and that is not its default
    v = pkg.variants(o)[cls][1]
    for i, name in enumerate(v):
        if name != default:
            try:
                pkg.select_variant(o, cls, i)
            except pkg.MHDError:
                continue
            pkg.select_variant(o, cls, v.index(default))
            return name
    raise AssertionError("no other variant of " + cls)
def entry(key, sel):
    with open(os.environ["MHDGB_TUNE_CACHE"], "a") as f:
        f.write("|".join([gpu.name, str(gpu.multi_processor_count), key] + [sel[c] for c in pkg.TUNED_CLASSES]) + "\\n")
def entries():
    with open(os.environ["MHDGB_TUNE_CACHE"]) as f:
        return [l.rstrip("\\n").split("|")[2:] for l in f]
single = lambda **kw: pkg.Problem(pkg.GPU(0), nu=1e-3, eta=kw.pop("eta", 1e-3), dt=1e-3, **kw)
"""


def _run(tmp_path, body):
    env = dict(os.environ, MHDGB_TUNE_CACHE=str(tmp_path / "tune.txt"))
    r = subprocess.run([sys.executable, "-c", HEAD.format(root=ROOT) + body], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def test_walls_of_a_hydrodynamic_problem(tmp_path):
    """set_vp with walls looks up the entry of its own field set."""
    _run(tmp_path, """
kw = dict(nx=48, B_field=False, VP_method=True, eta=0.0)
chi, wall = np.ones((48,) * 3, np.float32), np.ones((48,) * 3, np.float32)
with single(**kw) as p:
    p.set_vp(chi, U0=(wall,) * 3)
    sel = names(p)
    sel["x_fused"] = other(p, "x_fused", sel["x_fused"])
entry("48v2h", sel)
with single(**kw) as p:
    p.set_vp(chi, U0=(wall,) * 3)
    assert names(p) == sel, names(p)
""")


@pytest.mark.parametrize("n", [48, 64])
def test_single_problems_and_batches_have_entries_of_their_own(tmp_path, n):
    """A selection of single problems leaves a batch's plane passes at the batch's defaults (and the other
    way round), a batch is timed although the single problem's entry is known, and the x rows, which
    decide the rounding, stay common."""
    _run(tmp_path, f"n = {n}" + """
with single(nx=n) as p, pkg.Batch(n, 8) as b:
    one, many = names(p), names(b)
    assert one["x_fused"] == many["x_fused"] and one["z_inverse"] != many["z_inverse"]
    tuned = dict(one, x_fused=other(p, "x_fused", one["x_fused"]))
entry(str(n), tuned)
with single(nx=n) as p, pkg.Batch(n, 8) as b:
    assert names(p) == tuned
    assert names(b) == dict(many, x_fused=tuned["x_fused"]), names(b)
    for _ in range(8):
        b.add(1e-3, 1e-3, 1e-3)
    got = pkg.autotune(b)
    assert [e[0] for e in entries()] == [str(n), str(n) + "b"], entries()
    assert got == dict(zip(pkg.TUNED_CLASSES, entries()[-1][1:])) and got["x_fused"] == tuned["x_fused"]
    assert pkg.autotune(p) == tuned and len(entries()) == 2
with pkg.Batch(n, 4) as b:
    assert names(b) == got
""")


@pytest.mark.parametrize("n", [48, 64, 96, 128])
def test_plane_variants_give_the_same_bits(pkg, mo, n):
    """What lets single problems and batches differ in their plane variants."""
    s = mo.random_spectrum_state(mo.Grid(n), seed=7).astype("complex64")
    with pkg.Problem(pkg.GPU(0), nx=n, nu=1e-3, eta=2e-3, dt=1e-3) as p:
        p.set_sol(s.T)
        ref = None
        for cls in ("z_inverse", "z_forward"):
            for i in range(len(pkg.variants(p)[cls][1])):
                pkg.select_variant(p, cls, i)
                p.set_sol(s.T)
                pkg.stepforward(p, 2)
                got = p.sol_c().tobytes()
                ref = ref or got
                assert got == ref, (cls, i)


def test_column_passes_share_one_entry(tmp_path):
    """Where the variants of a class round differently (column passes), a batch keeps the single
    problem's selection, so that its slots still give a single problem's bits."""
    _run(tmp_path, """
with single(nx=256) as p:
    sel = names(p)
    for c in ("z_inverse", "x_fused"):
        sel[c] = other(p, c, sel[c])
entry("256", sel)
with pkg.Batch(256, 4) as b:
    assert names(b) == sel
    b.add(1e-3, 1e-3, 1e-3)
    assert pkg.autotune(b) == sel and len(entries()) == 1
""")


def test_forced_tuning_moves_the_common_class_of_both_entries(tmp_path):
    """A forced sweep of one kind keeps the x rows common: the other kind's entry takes them over."""
    _run(tmp_path, """
n = 64
with single(nx=n) as p, pkg.Batch(n, 8) as b:
    one, many = names(p), names(b)
    x = other(p, "x_fused", one["x_fused"])
entry(str(n), dict(one, x_fused=x))
entry(str(n) + "b", dict(many, x_fused=x))
with single(nx=n) as p:
    assert names(p)["x_fused"] == x
    new = pkg.autotune(p, force=True)
with pkg.Batch(n, 8) as b:
    assert names(b) == dict(many, x_fused=new["x_fused"])
""")


@pytest.mark.parametrize("n", [48, 64])
def test_line_between_single_and_batch_defaults(tmp_path, n):
    """Batches of two take the single problem's plane variants, batches of three the batch's."""
    _run(tmp_path, f"n = {n}" + """
with single(nx=n) as p, pkg.Batch(n, 1) as a, pkg.Batch(n, 2) as b, pkg.Batch(n, 3) as c, pkg.Batch(n, 24) as d:
    assert names(p) == names(a) == names(b)
    assert names(c) == names(d) != names(p)
""")
