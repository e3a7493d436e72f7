"""The update kernel's forms in the bounds-checked build, each pinned (left to
the timing, either build may run another one): no index outside its array, no
box coordinate outside its block's planes, and the normal build's states bit
for bit.  Each build runs in a process of its own."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUN = """
import os, sys
sys.path[:0] = [{root!r}, os.path.join({root!r}, "tests")]
import numpy as np
import combustioncodegpu_b200 as cc
from bounds_runner import make_case
name, precision, scheme, form, width, out = sys.argv[1:7]
case = make_case(name)
d = cc.Driver.from_case(case, precision)
d.set_update_tuning(form, int(width))
d.set_tuning("split", 3)
d.initialize_computation()
assert d.update_tuning()["form"] == form and d.update_tuning()["tile"][0] == int(width)
d.simulate(2, scheme)
states = {{"b%d" % b: d.field[b].get_state()[2] for b in range(len(case["blocks"]))}}
np.savez(out, status=d.status(), lib=os.path.basename(cc.LIB_PATH), **states)
""".format(root=ROOT)


def _run(lib, args, out):
    env = dict(os.environ, CC_LIBRARY=os.path.join(ROOT, "combustioncodegpu_b200", lib))
    r = subprocess.run([sys.executable, "-c", RUN, *args, str(out)], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(out)


@pytest.mark.gpu
@pytest.mark.parametrize("name,precision,scheme,form,width", [
    ("multiblock", "mixed", "rk3", "tma", "32"), ("multiblock", "mixed", "rk3", "tma", "16"),
    ("channel", "mixed", "steady", "tma", "32"), ("sod", "fp64", "rk3", "tma", "16"),
    ("mixing", "mixed", "rk3", "tma", "32"), ("multiblock", "mixed", "rk3", "plain-4", "16"),
    ("box", "fp64", "rk3", "plain", "16")])
def test_pinned_update_form_stays_in_bounds(tmp_path, name, precision, scheme, form, width):
    args = [name, precision, scheme, form, width]
    got = _run("libcc_b200_bounds.so", args, tmp_path / "bounds.npz")
    want = _run("libcc_b200.so", args, tmp_path / "normal.npz")
    assert str(got["lib"]) == "libcc_b200_bounds.so" and str(want["lib"]) == "libcc_b200.so"
    assert int(got["status"]) == int(want["status"]) == 0
    for k in want.files:
        if k.startswith("b"):
            np.testing.assert_array_equal(got[k], want[k])
