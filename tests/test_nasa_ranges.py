"""Mixture thermodynamics with the species in one NASA-7 range, in different
ranges at the same temperature, and below t_low, against the CPU oracle.

The kernels sum the species' coefficients before evaluating one polynomial,
with one range test for all species where their tables allow it and one per
species elsewhere.  Tolerances as in test_gpu_parity.py (FP64 rounding 1e-10;
FP32 fluxes and transport 1e-4), one RK3 step and one steady step."""
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


def _species(ranges, count):
    sp = dict(cases.synthetic_species() if count == 9 else cases.synthetic_species(cases.H2O2_N2_SPECIES[:count]))
    k = np.arange(count)
    if ranges == "spread":  # t_low and t_mid differ from species to species inside the field's 300..1500 K
        sp["t_low"] = 250.0 + 60.0 * k
        sp["t_mid"] = 1000.0 + 10.0 * (k - count // 2)
    elif ranges == "low":  # every point below t_low: the linear continuation
        sp["t_low"] = np.full(count, 1600.0)
        sp["t_mid"] = np.full(count, 1700.0)
    return sp


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ranges", ["common", "spread", "low"])
@pytest.mark.parametrize("count", [9, 3])
@pytest.mark.parametrize("scheme", ["rk3", "steady"])
def test_species_ranges(precision, ranges, count, scheme):
    case = cases.case_box(11, species=_species(ranges, count), seed=5)
    renorm = precision == "mixed"
    o = Oracle(case)
    o.init()
    (o.rk3_step if scheme == "rk3" else o.steady_step)(1, renorm_y=renorm)
    d = cc.Driver.from_case(case, precision)
    d.initialize_computation()
    d.simulate(1, scheme)
    bv, yk, _ = d.field[0].get_state()
    assert d.status() == 0
    d.close()
    want = o.state(0)
    tol = 1e-10 if precision == "fp64" else 1e-4
    err = group_errors(bv, want[0], bv_groups())
    err["yk"] = float(np.abs(yk - want[1]).max())
    assert all(e < tol for e in err.values()), err
