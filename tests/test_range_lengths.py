"""Range compression at every compile-time transform length (its samples decoded by the first pass,
its own radices, threads and resident blocks) against a run-time length on the same records: bytes
and FBAQ4 records, with records that start later and, for FBAQ4, end early.

Any length of at least the range size gives the same compressed samples up to float32 rounding:
the relative RMSE of the detected image stays below 1e-5, the bound the range lengths are held to
elsewhere, and the statistics do not depend on the length at all.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import scene as S
from conftest import rel_rmse, scene_and_raw

LENGTHS = [768, 1024, 1536, 2048, 3072, 4096, 6144, 8192]


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def lib(request):
    return request.getfixturevalue(f"{request.param}_lib")


@pytest.mark.parametrize("fmt", ["bytes", "fbaq4"])
@pytest.mark.parametrize("L", LENGTHS)
def test_every_length_equals_a_run_time_length(lib, L, fmt):
    na, nr = 400, min(L, 1000)
    codes = (np.arange(na) // 150 * (2 if fmt == "bytes" else 8) + 600).astype(np.uint16)
    kw = dict(azimuth_size=na, range_size=nr, swst_codes=codes)
    factory = S.tiny
    if fmt == "fbaq4":
        factory = S.tiny_fbaq
        kw["record_samples"] = np.full(na, nr - 16) - np.arange(na) % 3 * 41
    sc, raw, _ = scene_and_raw(lib, factory, **kw)
    img, res = [], []
    for n in (L, L // 8 * 9):
        plan = asarf.FocusPlan(sc, lib=lib, rc_fft_len=n)
        assert plan.dims["rc_fft_len"] == n
        img.append(plan.focus_host(raw, codes))
        res.append(plan.results())
        plan.close()
    assert res[0]["errors"] == res[1]["errors"] == 0
    for k in ("dc_i", "dc_q", "iq_gain", "phase_error", "first_line", "n_lines"):
        assert res[0][k] == res[1][k], k
    assert np.abs(img[0]).max() > 0
    assert rel_rmse(img[0], img[1]) < 1e-5
