"""The update kernel's own bounded wait for its state boxes (k_update_tma),
apart from the face kernel's: the faces come through L1 here, so that the
status bit can only be the update's.  With a limit of 0 a wait checks once;
in the tiles of the last rows, of which the block fills one, whole warps have
no point and reach the wait a few hundred cycles after the request.  The
kernel sets status bit 3, lets its copies land and returns; with the limit
restored and the state set again a step equals a fresh context's."""
import numpy as np
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu

STATUS_TMA_TIMEOUT = 8


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("width", [32, 16])
def test_update_wait_gives_up_and_context_recovers(precision, width):
    case = cases.case_box(49, species=cases.synthetic_species(), seed=7)  # one row past 8- and 16-high tiles
    blk = case["blocks"][0]

    def context():
        d = cc.Driver.from_case(case, precision)
        d.set_update_tuning("tma", width)
        d.set_tuning("split", 4)
        d.initialize_computation()
        assert d.tuning()["variant"] == "split" and d.update_tuning()["form"] == "tma"
        return d

    d = context()
    d.set_wait_limit(0)
    d.simulate(1)
    assert d.status() & STATUS_TMA_TIMEOUT
    d.set_wait_limit(None)
    d.field[0].set_state(blk["bv"], blk["yk"])
    d.simulate(1)
    assert d.status() == 0
    got = d.field[0].get_state()[2]
    d.close()
    e = context()
    e.simulate(1)
    want = e.field[0].get_state()[2]
    assert e.status() == 0
    e.close()
    np.testing.assert_array_equal(got, want)
