"""Scenes whose range walk at the PRF is tens to hundreds of samples: the range-Doppler tile carries that
halo, so the contiguous azimuth length must be one whose tile fits shared memory.

Random complex images through the per-stage entry point against the oracle (FP64 with the reference's
float32 decisions).  Tolerance: two float32 transforms of 4032 points and the interpolation, under 1e-6
relative RMSE; 2e-6 leaves a factor of two.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import scene as S
from asarf import stages as st
from oracle import rda


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


# walk at the PRF, samples: 60, 130, 228, 281
@pytest.mark.parametrize("wavelength", [0.0924, 0.136, 0.18, 0.2])
def test_range_doppler(be, wavelength):
    lib, gpu = be
    x, xs, y, ys = 300, 304, 4000, 4032
    rng = np.random.default_rng(7)
    img = np.zeros((ys, xs), dtype=np.complex64)
    img[:y, :x] = (rng.standard_normal((y, x)) + 1j * rng.standard_normal((y, x))).astype(np.complex64)
    prf, frac, spacing, near = 5200.0, 0.2, 7.905707, 830000.0
    dc, vr = (0.0, 0.0, 100.0), (0.0, 0.0, 7100.0)
    want = rda.range_doppler(img, x, y, rda.RdaArgs(prf, wavelength, frac, spacing, near, np.array(dc), np.array(vr)))

    def dev(a):
        if not gpu:
            return np.ascontiguousarray(a).copy()
        import torch
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    out = st.range_doppler_algorithm(prf, wavelength, spacing, near, frac, vr, dc, st.DevicePaddedImage(dev(img), x, y),
                                     dev(np.zeros_like(img)), lib=lib)
    got = out.data.cpu().numpy() if gpu else out.data
    err = np.sqrt(np.mean(np.abs(got[:y, :x] - want[:y, :x]) ** 2) / np.mean(np.abs(want[:y, :x]) ** 2))
    assert err < 2e-6, err


@pytest.mark.parametrize("range_size,lines", [(2048, 4000), (5616, 9973), (700, 12000)])
def test_plans_fit(be, range_size, lines):
    """A plan is made at every walk whose tile fits at some admissible length."""
    lib, _ = be
    for wavelength in (0.1, 0.2, 0.3, 0.36, 0.4):
        sc = S.tiny(range_size=range_size, azimuth_size=lines, wavelength=wavelength, prf=2400.0, slant_range_first=830000.0,
                    altitude=800000.0, az_bw_frac=0.2, vr_poly=(0.0, 0.0, 7100.0))
        plan = asarf.FocusPlan(sc, lib=lib)
        assert plan.dims["n1"] * plan.dims["n2"] == plan.dims["az_pad"]
        plan.close()
