"""The autotuner's cache serves shapes timed on this revision of the kernels only, and its azimuth splits are
searched around the planner's.  The timing is a fake, so this runs without a GPU.
"""
from __future__ import annotations

import json

import pytest

from asarf import autotune
from asarf import scene as S


@pytest.fixture
def tuner(monkeypatch):
    import torch

    tried = []

    class Plan:
        dims = {"az_pad": 10000, "n2": 125, "az_tile_width": 64, "strided_tile_width": 32, "rc_fft_len": 1024}
        out_shape = (4, 4)

        def __init__(self, *a, **k):
            pass

        def close(self):
            pass

    def timed(scene, raw_d, out_d, lib, opts, runs):
        tried.append(dict(opts))
        return 1.0 + abs(opts.get("az_n2", 125) - 125) * 0.01

    monkeypatch.setattr(autotune, "FocusPlan", Plan)
    monkeypatch.setattr(autotune, "_time_options", timed)
    monkeypatch.setattr(torch, "empty", lambda *a, **k: None)
    return tried


def _old_key(sc):
    """The key as it was without a revision."""
    return autotune.shape_key(sc).rsplit(":r", 1)[0]


def test_entries_of_other_kernels_are_not_served(tuner, tmp_path):
    sc = S.tiny()
    cache = tmp_path / "tune.json"
    stale = {"options": {"precision": 0, "az_n2": 49}, "ms_default": 2.0, "ms_tuned": 1.0, "timings": []}
    cache.write_text(json.dumps({_old_key(sc): stale}))
    opts = autotune.tune(sc, None, lib=object(), cache=cache)
    assert opts.get("az_n2") != 49 and tuner
    n = len(tuner)
    assert autotune.tune(sc, None, lib=object(), cache=cache) == opts and len(tuner) == n  # its own entry is served
    assert f":r{autotune.REVISION}" in autotune.shape_key(sc)


def test_splits_are_searched_around_the_planned_one(tuner, tmp_path):
    autotune.tune(S.tiny(), None, lib=object(), cache=tmp_path / "tune.json")
    n2 = sorted({o["az_n2"] for o in tuner if "az_n2" in o})
    assert n2 == [80, 100, 200, 250]  # 125 is the planner's, 100 the divisor at the root
