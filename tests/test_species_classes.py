"""Species counts at the edges of the kernels' classes (at most 4, 8, 11, 16)
against the CPU oracle, on a curvilinear grid: the face kernel reading through
L1 and the one with TMA-staged planes (which the autotuner chooses between),
and the LU-SGS step, whose rows are sized for the class.  Tolerances as in
test_gpu_parity.py."""
import os
import sys

import numpy as np
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases
from oracle.oracle_py import Oracle

sys.path.insert(0, os.path.dirname(__file__))
from gpu_compare import bv_groups, group_errors  # noqa: E402

pytestmark = pytest.mark.gpu

MORE = [("N", {"N": 1}), ("NO", {"N": 1, "O": 1}), ("NO2", {"N": 1, "O": 2}), ("N2O", {"N": 2, "O": 1}),
        ("O3", {"O": 3}), ("NH", {"N": 1, "H": 1}), ("HNO", {"H": 1, "N": 1, "O": 1})]


@pytest.mark.parametrize("count", [1, 4, 5, 8, 10, 11, 12, 16])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("faces", ["2", "3", "lusgs"])
def test_count_matches_oracle(count, precision, faces, monkeypatch):
    sp = cases.synthetic_species((cases.H2O2_N2_SPECIES + MORE)[:count])
    case = cases.case_box_distorted(18, amp=0.2, species=sp, seed=count)
    renorm = precision == "mixed"
    if faces != "lusgs":
        monkeypatch.setenv("CC_AUTOTUNE_VARIANT", faces)
    o = Oracle(case)
    o.init()
    (o.lusgs_step if faces == "lusgs" else o.rk3_step)(1, renorm_y=renorm)
    d = cc.Driver.from_case(case, precision)
    d.initialize_computation()
    if faces != "lusgs":
        assert d.tuning()["variant"] == cc.VARIANTS[int(faces)]
    d.simulate(1, "lusgs" if faces == "lusgs" else "rk3")
    bv, yk, _ = d.field[0].get_state()
    assert d.status() == 0
    d.close()
    want = o.state(0)
    err = group_errors(bv, want[0], bv_groups())
    err["yk"] = float(np.abs(yk - want[1]).max())
    assert all(e < (1e-10 if precision == "fp64" else 1e-4) for e in err.values()), err
