"""Which entry of the tuning file a handle takes: grid size, precision, penalisation, field set.  Each check runs in a
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
