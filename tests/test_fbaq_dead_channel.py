"""A dead channel in FBAQ4 records: every sample of one channel decodes to the same instrument-table value.

The planned path sums squares about zero in FP64 (n v^2 rounded to n v^2 2^-53 sqrt(n) or so, n = 75600
here: 3e-14 of it), so the variance that is left of a constant v is rounding of either sign and its root
at most 2e-7 v, plus the mean's own rounding to float32 (6e-8 v): 1e-6 v bounds the deviation, which
is a number and not NaN; the gain and phase follow from it and from the padding's share.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import fbaq
from asarf import scene as S


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


@pytest.mark.parametrize("block", [3, 40, 77, 101, 128, 150, 203, 255])
@pytest.mark.parametrize("dead", ["i", "q"])
def test_deviation_is_a_number(be, block, dead):
    lib, gpu = be
    nr, lines = 252, 300
    sc = S.tiny_fbaq(range_size=nr, azimuth_size=lines, record_samples=np.full(lines, nr))
    sc.prepare(lib)
    rng = np.random.default_rng(block)
    rec = fbaq.encode(rng.normal(0.0, 8.0, (lines, nr)), rng.normal(0.0, 8.0, (lines, nr)), np.full(lines, nr),
                      sc.raw_line_bytes)
    r = np.arange(nr)
    rec[:, 2 + 64 * (r // 63)] = block
    at = 2 + r + r // 63 + 1
    code = 5
    rec[:, at] = (code << 4 | rec[:, at] & 15) if dead == "i" else (rec[:, at] & 0xF0 | code)
    level = abs(float(sc.fbaq_tables[0 if dead == "i" else 1][fbaq.table_index(np.array([block]), np.array([code]))][0]))
    plan = asarf.FocusPlan(sc, lib=lib, ref_compat_stats=False)
    plan.focus_host(rec)
    res = plan.results()
    plan.close()
    std = res["stddev_" + dead]
    assert 0.0 <= std <= 1e-6 * level, (std, level)
    assert res["stddev_" + ("q" if dead == "i" else "i")] > 0.01 * level
