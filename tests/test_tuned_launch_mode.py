"""The stage kernels are timed in the launch mode they will run in: per block,
a candidate of 27 small blocks is 27 launches and takes several times the
batched one's single launch."""
import pytest

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases

pytestmark = pytest.mark.gpu


def test_candidates_are_timed_per_block(monkeypatch, capfd):
    monkeypatch.setenv("CC_AUTOTUNE_VERBOSE", "1")
    case = cases.case_multiblock(([6, 5, 7], [5, 6, 5], [5, 5, 6]), seed=3)
    best = {}
    for mode in ("batched", "per_block"):
        d = cc.Driver.from_case(case, "mixed")
        d.set_launch_mode(mode)
        capfd.readouterr()
        d.initialize_computation()
        lines = capfd.readouterr().err.splitlines()
        d.close()
        for what in ("update form", "split tile", "split-tma tile", "fused-l1 tile"):
            best[mode, what] = min(float(ln.split()[-2]) for ln in lines if what in ln)
    for what in ("update form", "split tile", "split-tma tile", "fused-l1 tile"):
        assert best["per_block", what] > 3.0 * best["batched", what]
