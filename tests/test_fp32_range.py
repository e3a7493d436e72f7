"""Small operands of the FP32 approximations.  Density in the FP32 denormal range (2e-41 kg/m3; times the gas constant
still below 1.2e-38): the mixed path's FP32 divisions take denormal operands
instead of flushing them to zero, so a uniform stream stays as it is, as in
FP64.  Tolerance 5e-4: a few of the relative steps in which FP32 resolves such
a density (1.4e-45 / 2e-41 = 7e-5)."""
import numpy as np
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu


def _uniform(kind, rho=2e-41):
    case = cases.case_box(8, species=cases.synthetic_species()) if kind == "mixture" else cases.case_sod(12, 6, 6)
    blk = case["blocks"][0]
    bv = np.empty_like(blk["bv"])
    if kind == "mixture":
        blk["yk"] = np.repeat(blk["yk"][:, :1], bv.shape[1], axis=1)
        gas = cases.R_U * (blk["yk"][:, 0] / np.asarray(case["params"]["species"]["mw"])).sum()
    else:
        gas = cases.R_U / 28.9647
    bv[:] = np.array([rho, 30.0, -20.0, 10.0, rho * gas * 900.0, 900.0])[:, None]
    blk["bv"] = bv
    return case


@pytest.mark.parametrize("temperature", [1e-3, 1.0, 40.0, 900.0, 2e4])
@pytest.mark.parametrize("trace", [1e-3, 1e-30, 1e-41])
def test_transport_of_traces_and_extreme_temperatures(temperature, trace):
    """The transport's FP32 approximations flush denormal operands; none is
    denormal over temperatures beyond any flow's and down to denormal mass
    fractions: as in FP64 within 1e-5, the path's error budget."""
    props = []
    for precision in ("fp64", "mixed"):
        case = _uniform("mixture", rho=1.0)
        blk = case["blocks"][0]
        y = np.full(9, trace)
        y[8] = 1.0 - y[:8].sum()
        blk["yk"][:] = y[:, None]
        gas = cases.R_U * (y / np.asarray(case["params"]["species"]["mw"])).sum()
        blk["bv"][5] = temperature
        blk["bv"][4] = gas * temperature
        d = cc.Driver.from_case(case, precision)
        d.set_tuning("split", 2)
        d.initialize_computation()
        d.simulate(1)
        assert d.status() == 0
        props.append(d.field[0].get_props())
        d.close()
    for want, got in zip(*props):
        np.testing.assert_allclose(got, want, rtol=1e-5)


@pytest.mark.parametrize("kind", ["air", "mixture"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("variant", ["l1", "tma", "split", "split-tma"])
def test_uniform_stream_of_denormal_density(kind, precision, variant):
    if precision == "fp64" and variant == "tma":
        pytest.skip("the fused TMA variant is for the FP32 bulk precision")
    case = _uniform(kind)
    d = cc.Driver.from_case(case, precision)
    d.set_tuning(variant, 2)
    d.initialize_computation()
    d.simulate(2)
    bv, yk, _ = d.field[0].get_state()
    assert d.status() == 0
    d.close()
    want = case["blocks"][0]["bv"]
    for f in range(6):
        np.testing.assert_allclose(bv[f], want[f], rtol=5e-4)
    if kind == "mixture":
        np.testing.assert_allclose(yk, case["blocks"][0]["yk"], rtol=5e-4)
