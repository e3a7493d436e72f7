"""The update kernel's forms and tile widths give the same states bit for bit:
which of them runs is chosen by timing, and equal runs, restarts and launch
modes have to agree whatever it chooses.  Extents one past a tile's in both
directions, walls with the per-point time step, a curvilinear grid (the
geometric term of the gauge pressure) and the dq variant's residual."""
import numpy as np
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu


def _case(name):
    if name == "blocks":
        return cases.case_multiblock(([33, 5], [17, 9], [6]), seed=3)
    if name == "channel":
        return cases.case_channel((34, 10, 7))
    if name == "four":
        return cases.case_box_distorted(17, amp=0.2, species=cases.synthetic_species(cases.H2O2_N2_SPECIES[:4]))
    if name == "curved":
        return cases.case_box_distorted(17, amp=0.2)
    return cases.case_sod(40, 6, 6)


@pytest.mark.parametrize("name,precision,scheme,variant", [
    ("blocks", "mixed", "rk3", "split"), ("blocks", "fp64", "rk3", "split"), ("channel", "mixed", "steady", "split"),
    ("channel", "fp64", "steady", "split"), ("four", "mixed", "rk3", "split"), ("four", "fp64", "rk3", "split"),
    ("curved", "mixed", "rk3", "split-tma"), ("curved", "fp32", "rk3", "split-tma"), ("curved", "mixed", "rk3", "dq-tma"),
    ("sod", "mixed", "rk3", "split"), ("sod", "fp64", "rk3", "split")])
def test_forms_agree_bit_for_bit(name, precision, scheme, variant):
    case = _case(name)
    want = None
    for form in ("plain", "plain-4", "tma"):
        if form == "plain-4" and precision == "fp64":
            continue
        for width in (32, 16):
            d = cc.Driver.from_case(case, precision)
            d.set_update_tuning(form, width)
            d.set_tuning(variant, 2)
            d.initialize_computation()
            assert d.update_tuning() == {"form": form, "tile": (width, 256 // width, 2)}
            d.simulate(3, scheme)
            assert d.status() == 0
            got = [a for b in range(len(case["blocks"])) for a in d.field[b].get_state() if a is not None]
            d.close()
            if want is None:
                want = got
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
