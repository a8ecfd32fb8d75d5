"""The azimuth split N = n1 * n2 is a launch shape: the same scene focused with splits whose strided
pass puts one, two, four and eight tiles side by side in a block (n2 a multiple of that and not), with
compiled and run-time block lengths and two-, three- and four-stage schedules, against the oracle and
against each other.

Each transform costs a few float32 roundings per stage, so two splits differ by rounding only: the
detected images agree to 2e-6 relative RMSE (twice the single-precision transforms' error against the
oracle on this scene), and a row moved or missed would show as 1e-3 or more.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import scene as S
from conftest import oracle_focus, rel_rmse, scene_and_raw


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def lib(request):
    return request.getfixturevalue("emu_lib" if request.param == "emu" else "gpu_lib")


# (range, lines, azimuth splits n2): lines 1990 pad to 2000, 1205 to 1215, 2010 to 2016, 2870 to 2880
CASES = [
    (2048, 1990, [0, 125, 100, 250, 40, 16]),
    (768, 1205, [0, 81, 135, 243, 45]),
    (768, 2010, [0, 168, 126, 144, 112, 96, 63]),
    (768, 2870, [0, 160, 180, 240, 90, 64]),
]


@pytest.mark.parametrize("nr,lines,splits", CASES)
def test_splits_agree(lib, nr, lines, splits):
    sc, raw, _ = scene_and_raw(lib, S.tiny, range_size=nr, azimuth_size=lines, seed=21)
    base = None
    for n2 in splits:
        plan = asarf.FocusPlan(sc, lib=lib, az_n2=n2)
        out = plan.focus_host(raw)
        assert plan.results()["errors"] == 0
        if n2:
            assert plan.dims["n2"] == n2
        if base is None:
            base = out
            if nr == 768:
                assert rel_rmse(out, oracle_focus(sc, raw).detected) < 1e-5
        assert out.shape == base.shape
        assert rel_rmse(out, base) < 2e-6, n2
        plan.close()
