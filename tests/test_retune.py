"""Tuning a context again after the dq variant has run, which leaves its
residual where the split variants keep their faces: the update kernel is timed
on faces of the current state, as in a fresh context.  On a residual read as
faces its Newton iterates far longer (tens of times at this size)."""
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu


def _update_ms(text):
    return [float(ln.split()[-2]) for ln in text.splitlines() if "update form 0" in ln]


def test_update_is_timed_on_faces_after_the_dq_variant(monkeypatch, capfd):
    monkeypatch.setenv("CC_AUTOTUNE_VERBOSE", "1")
    d = cc.Driver.from_case(cases.case_box(32, species=cases.synthetic_species()), "mixed")
    d.set_tuning("split", 2)
    d.initialize_computation()
    fresh = min(_update_ms(capfd.readouterr().err))
    d.set_tuning("dq-tma", 2)
    d.simulate(2)
    capfd.readouterr()
    d.set_tuning("split", 2)
    again = min(_update_ms(capfd.readouterr().err))
    d.close()
    assert 0.0 < again < 5.0 * fresh
