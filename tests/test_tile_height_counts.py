"""Pinned face tile heights by species count: 16 is for the FP32 bulk
precision; in FP64 a context whose species count has no kernel of its own
(neither 0 nor 9) refuses it at cc_init, whatever the variant."""
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,height,taken", [("mixed", 8, True), ("mixed", 16, True), ("fp64", 8, True),
                                                    ("fp64", 16, False)])
@pytest.mark.parametrize("variant", ["auto", "l1", "split"])
@pytest.mark.parametrize("count", [4, 8, 11])
def test_height_by_species_count(variant, count, precision, height, taken):
    more = [("N", {"N": 1}), ("NO", {"N": 1, "O": 1})]
    sp = cases.synthetic_species((cases.H2O2_N2_SPECIES + more)[:count])
    d = cc.Driver.from_case(cases.case_box(9, species=sp, seed=2), precision)
    d.set_tuning(variant, 2, height)
    if taken:
        d.initialize_computation()
        d.simulate(1)
        assert d.status() == 0
    else:
        with pytest.raises(RuntimeError, match="face tile height"):
            d.initialize_computation()
    d.close()
