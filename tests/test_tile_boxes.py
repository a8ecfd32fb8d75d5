"""The range-Doppler tile arrives in TMA boxes of at most 256 rows, each to shared memory at a multiple of its
rows: every box must start on a 128-byte boundary there, whatever the azimuth length (lines above 98000
pad to 100842, 117649 and 129654, whose contiguous lengths 294 and 343 split into boxes of odd rows).

The launch itself is checked against the oracle at 100842 rows; tolerance as in the other comparisons of
this entry point, two float32 transforms (17 octaves: under 1.2e-6 relative RMSE) with the interpolation, 2e-6.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from asarf import stages as st
from oracle import rda


def _sizes():
    out = []
    for n in range(16, 131073):
        m = n
        for q in (2, 3, 5, 7):
            while m % q == 0:
                m //= q
        if m == 1:
            out.append(n)
    return out


@pytest.mark.parametrize("nk,hr", [(17, 10), (100, 12), (1500, 30), (5000, 9), (5000, 60), (300, 110)])
def test_boxes_start_on_128_bytes(emu_lib, nk, hr):
    f = emu_lib.asarf_emu_rd_tile
    f.restype = None
    n2, wt, box = C.c_int(), C.c_int(), C.c_int()
    for n in _sizes():
        hre = hr + hr % 2
        f(n, nk, 8, hre, C.byref(n2), C.byref(wt), C.byref(box))
        b = box.value
        assert n % n2.value == 0 and wt.value % 2 == 0 and 0 <= b <= 256
        if b:
            assert n2.value % b == 0
            assert b == n2.value or b * wt.value * 8 % 128 == 0, (n, n2.value, wt.value, b)
        else:
            assert n2.value > 256


@pytest.mark.gpu
def test_long_column_matches_oracle(gpu_lib):
    import torch

    x, xs, y, ys = 60, 64, 100000, 100842
    rng = np.random.default_rng(3)
    img = np.zeros((ys, xs), dtype=np.complex64)
    img[:y, :x] = (rng.standard_normal((y, x)) + 1j * rng.standard_normal((y, x))).astype(np.complex64)
    vr, dc = (0.0, 0.0, 7100.0), (0.0, 0.0, 300.0)
    want = rda.range_doppler(img, x, y, rda.RdaArgs(1680.0, 0.05656, 0.8, 7.905707, 830000.0, np.array(dc), np.array(vr)))
    out = st.range_doppler_algorithm(1680.0, 0.05656, 7.905707, 830000.0, 0.8, vr, dc,
                                     st.DevicePaddedImage(torch.from_numpy(img).cuda(), x, y),
                                     torch.zeros(ys, xs, dtype=torch.complex64, device="cuda"), lib=gpu_lib)
    got = out.data.cpu().numpy()
    err = np.sqrt(np.mean(np.abs(got[:y, :x] - want[:y, :x]) ** 2) / np.mean(np.abs(want[:y, :x]) ** 2))
    assert err < 2e-6, err
