"""The update kernel forms that set-up times: every form in the FP32 bulk
precision; in FP64 only the plain one, as the others are slower there or not
built.  A form named for a profiling run still runs where it is built."""
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,pinned,forms", [("fp64", None, {"0"}), ("mixed", None, {"0", "1", "2"}),
                                                    ("fp64", "2", {"2"}), ("fp64", "1", {"0"}), ("mixed", "1", {"1"})])
def test_update_forms_timed(precision, pinned, forms, monkeypatch, capfd):
    monkeypatch.setenv("CC_AUTOTUNE_VERBOSE", "1")
    if pinned:
        monkeypatch.setenv("CC_UPDATE_OCC", pinned)
    d = cc.Driver.from_case(cases.case_sod(40, 6, 6), precision)
    d.initialize_computation()
    d.close()
    lines = [ln for ln in capfd.readouterr().err.splitlines() if "update form" in ln]
    assert {ln.split("update form ")[1].split()[0] for ln in lines} == forms
