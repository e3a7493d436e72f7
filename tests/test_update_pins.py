"""Pinning the update kernel: the form and tile width asked for are the ones
that run (cc_update_tuning), and a form that the context cannot run is an
error at set-up."""
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases


def test_arguments_are_checked():
    d = cc.Driver.from_case(cases.case_sod(12, 6, 6), "fp64")
    for form, width in ((0, 0), (1, 16), (2, 32), (-1, 0)):
        assert d.lib.cc_set_update_tuning(d.ctx, form, width) == 0
    for form, width in ((3, 0), (-2, 0), (0, 8)):
        assert d.lib.cc_set_update_tuning(d.ctx, form, width) == -1
    d.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("form", ["plain", "plain-4", "tma"])
@pytest.mark.parametrize("width", [16, 32])
def test_pinned_form_runs_or_fails(precision, form, width):
    d = cc.Driver.from_case(cases.case_box(9, species=cases.synthetic_species(), seed=2), precision)
    d.set_update_tuning(form, width)
    d.set_tuning("split", 2)
    if form == "plain-4" and precision == "fp64":
        with pytest.raises(RuntimeError, match="update kernel form"):
            d.initialize_computation()
    else:
        d.initialize_computation()
        assert d.update_tuning() == {"form": form, "tile": (width, 256 // width, 2)}
        d.simulate(1)
        assert d.status() == 0
    d.close()


@pytest.mark.gpu
def test_tma_form_without_tensor_maps_fails(monkeypatch):
    monkeypatch.setenv("CC_NO_TMA", "1")
    d = cc.Driver.from_case(cases.case_sod(12, 6, 6), "mixed")
    d.set_update_tuning("tma")
    with pytest.raises(RuntimeError, match="update kernel form"):
        d.initialize_computation()
    d.close()
