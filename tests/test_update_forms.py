"""The update kernel's forms (plain, plain at higher occupancy, conserved
state staged by TMA), pinned one by one, against the CPU oracle: extents below
and beyond a tile, remainders in every direction, walls with the per-point
time step, a runtime species count and the air model.  Tolerances as in
test_gpu_parity.py."""
import os
import sys

import numpy as np
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases
from oracle.oracle_py import Oracle

sys.path.insert(0, os.path.dirname(__file__))
from gpu_compare import bv_groups, cv_groups, group_errors  # noqa: E402

pytestmark = pytest.mark.gpu


def _case(name):
    if name == "blocks":  # 33 and 17 points: one past a 32- and a 16-wide tile
        return cases.case_multiblock(([33, 5], [17, 9], [6]), seed=3)
    if name == "channel":
        return cases.case_channel((34, 10, 7))
    if name == "four":
        return cases.case_box_distorted(13, amp=0.2, species=cases.synthetic_species(cases.H2O2_N2_SPECIES[:4]))
    return cases.case_sod(40, 6, 6)


@pytest.mark.parametrize("form", ["0", "1", "2"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["blocks", "channel", "four", "sod"])
def test_form_matches_oracle(form, precision, name, monkeypatch):
    monkeypatch.setenv("CC_UPDATE_OCC", form)
    case = _case(name)
    steady = name == "channel"
    renorm = precision == "mixed" and case["params"].get("species") is not None
    o = Oracle(case)
    o.init()
    (o.steady_step if steady else o.rk3_step)(2, renorm_y=renorm)
    d = cc.Driver.from_case(case, precision)
    d.set_tuning("split", 2)
    d.initialize_computation()
    d.simulate(2, "steady" if steady else "rk3")
    tol = 1e-10 if precision == "fp64" else 1e-4
    for b in range(len(case["blocks"])):
        bv, yk, cv = d.field[b].get_state()
        obv, oyk, ocv = o.state(b)
        err = group_errors(bv, obv, bv_groups()) | {"cv." + k: v for k, v in
                                                   group_errors(cv, ocv, cv_groups(o.ns)).items()}
        if o.ns:
            err["yk"] = float(np.abs(yk - oyk).max())
        assert all(e < tol for e in err.values()), err
    assert d.status() == 0
    d.close()
