"""Standard deviations of the per-stage IQ correction where the spread is small beside the level: dead
channels of instrument-table values, large means, blocks whose first pixels are missing, an outlier as
the first pixel, a total that counts more samples than were filled.

The reference value is sqrt(sum (v - dc)^2 / total) in FP64 about the mean that the call itself
reports, so a dead channel gives |v - dc|, at most an ulp of the level.  The call forms the sum in FP64
and rounds it, the quotient and the root to float32: three roundings of at most 2^-24 each, halved by the
root for the first two, so 1.2e-7; the FP64 sums lose at most 1e4 times their own rounding (1e-14 of
120000 pixels), 1e-10, before they are taken again about the mean.  2e-7 covers both.
"""
from __future__ import annotations

import numpy as np
import pytest

from asarf import scene as S
from asarf import stages as st


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


def _image(i, q, pad=37):
    y, x = i.shape
    img = np.zeros((y, x + pad), dtype=np.complex64)
    img[:, :x] = i.astype(np.float32) + 1j * q.astype(np.float32)
    return img


def _run(be, img, x, y, total):
    lib, gpu = be
    data = np.ascontiguousarray(img).copy()
    if gpu:
        import torch
        data = torch.from_numpy(data).cuda()
    return st.raw_data_correction(st.DevicePaddedImage(data, x, y), total, lib=lib)


def _check(res, i, q, total):
    ok = ~(np.isnan(i) | np.isnan(q))
    for v, dc, std in ((i, res["dc_i"], res["stddev_i"]), (q, res["dc_q"], res["stddev_q"])):
        v = v.astype(np.float32).astype(np.float64)[ok]
        want = np.sqrt(np.sum((v - np.float64(np.float32(dc))) ** 2) / total)
        assert std == pytest.approx(want, rel=2e-7, abs=1e-30), (std, want)


LEVELS = [float(np.float32(S.fbaq.SIGMA0 * 10.0 ** (k * S.fbaq.STEP_DB / 20.0) * S.fbaq.LEVELS[k % 8]))
          for k in (3, 17, 40, 77, 101, 150, 203)] + [64.0592, 0.203, 4.712]


@pytest.mark.parametrize("level", LEVELS)
def test_dead_channel(be, level):
    rng = np.random.default_rng(5)
    i = np.full((301, 400), level)
    q = rng.normal(0.0, 3.0, (301, 400))
    _check(_run(be, _image(i, q), 400, 301, 301 * 400), i, q, 301 * 400)
    _check(_run(be, _image(q, i), 400, 301, 301 * 400), q, i, 301 * 400)


@pytest.mark.parametrize("mean,dev", [(1e6, 0.3), (3e6, 0.5), (1e6, 0.1), (-2e5, 0.02), (15.5, 4.0)])
@pytest.mark.parametrize("shape", [(301, 400), (8, 17), (9, 1), (1, 300)])
def test_large_mean(be, mean, dev, shape):
    rng = np.random.default_rng(int(abs(mean)) + shape[0])
    i = (mean + rng.normal(0.0, dev, shape)).astype(np.float32)
    q = (-mean + rng.normal(0.0, 2 * dev, shape)).astype(np.float32)
    _check(_run(be, _image(i, q), shape[1], shape[0], i.size), i, q, i.size)


def test_missing_pixels_and_total(be):
    rng = np.random.default_rng(9)
    i = (4e5 + rng.normal(0.0, 0.2, (133, 700))).astype(np.float32)
    q = (9e5 + rng.normal(0.0, 0.4, (133, 700))).astype(np.float32)
    i[:, :520] = np.where(np.arange(133)[:, None] % 3 == 0, np.nan, i[:, :520])  # rows that begin late
    q[40:56] = np.nan  # whole blocks without a sample
    filled = int(np.sum(~(np.isnan(i) | np.isnan(q))))
    for total in (filled, filled + 1000):
        _check(_run(be, _image(i, q), 700, 133, total), i, q, total)


def test_outlier_first(be):
    rng = np.random.default_rng(11)
    i = (1e6 + rng.normal(0.0, 0.3, (64, 64))).astype(np.float32)
    q = rng.normal(0.0, 1.0, (64, 64)).astype(np.float32)
    i[0, 0], q[0, 0] = 0.0, 5e3
    _check(_run(be, _image(i, q), 64, 64, i.size), i, q, i.size)


def test_infinite_pixel(be):
    """An infinite sample makes its channel's sums infinite or NaN, and the other one's stay."""
    rng = np.random.default_rng(13)
    i = rng.normal(10.0, 1.0, (40, 90)).astype(np.float32)
    q = rng.normal(10.0, 1.0, (40, 90)).astype(np.float32)
    i[0, 0] = np.inf
    res = _run(be, _image(i, q), 90, 40, i.size)
    assert not np.isfinite(res["stddev_i"])
    assert res["stddev_q"] == pytest.approx(np.sqrt(np.mean((q.astype(np.float64) - np.float64(np.float32(res["dc_q"]))) ** 2)), rel=2e-7)
