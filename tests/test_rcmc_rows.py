"""Range cell migration and azimuth filter where their row decisions change: Doppler centroids of
either sign, crossing zero inside a tile, at and beyond half the PRF (aliased rows, wrapped filter
frequencies), walks from a fraction of a sample to many (halo), steep Vr across a tile (rows whose
columns do not agree go sample by sample), image widths around the 64-column tile and an odd stride.

Random complex images through the per-stage entry point against the oracle, which works in FP64 with
the reference's float32 decisions.  Tolerance: the two float32 transforms of N <= 1024 points cost about
eps * sqrt(log2 N) each and the interpolation as much again, under 1e-6 relative RMSE together; 2e-6
leaves a factor of two, and a row decided differently moves the image by 1e-3 or more.
"""
from __future__ import annotations

import numpy as np
import pytest

from asarf import stages as st
from oracle import rda


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


def _dev(gpu, a):
    if not gpu:
        return np.ascontiguousarray(a).copy()
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


BASE = dict(prf=1680.0, wavelength=0.05656, az_bw_frac=0.8, range_spacing=7.905707, slant_range=830000.0,
            vr=(3e-9, -1.35e-3, 7123.0), dc=(0.0, 0.0, 300.0))


def _case(**kw):
    d = dict(BASE)
    d.update(kw)
    return d


CASES = {
    "positive": _case(),
    "negative": _case(dc=(0.0, 0.01, -420.0)),
    "zero_crossing": _case(dc=(0.0, 2.5, -300.0)),
    "zero": _case(dc=(0.0, 0.0, 0.0)),
    "half_prf": _case(dc=(0.0, 0.4, 790.0)),
    "beyond_half_prf": _case(dc=(0.0, 0.0, -905.0)),
    "steep_dc": _case(dc=(0.01, -4.0, 350.0)),
    "small_walk": _case(slant_range=100000.0, vr=(0.0, 0.0, 7100.0)),
    "many_samples": _case(prf=5200.0, dc=(0.0, 0.0, 700.0)),
    "steep_vr": _case(vr=(0.0, -3.0, 7600.0), prf=3200.0),
    "narrow_band": _case(az_bw_frac=0.05),
    "full_band": _case(az_bw_frac=1.0, dc=(0.0, 0.0, 200.0)),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("shape", [(233, 240, 500, 504), (130, 131, 250, 250)])
def test_range_doppler_matches_oracle(be, name, shape):
    lib, gpu = be
    p = CASES[name]
    x, xs, y, ys = shape
    rng = np.random.default_rng(len(name) * 1000 + x)
    img = np.zeros((ys, xs), dtype=np.complex64)
    img[:y, :x] = (rng.standard_normal((y, x)) + 1j * rng.standard_normal((y, x))).astype(np.complex64)
    args = rda.RdaArgs(p["prf"], p["wavelength"], p["az_bw_frac"], p["range_spacing"], p["slant_range"],
                       np.array(p["dc"]), np.array(p["vr"]))
    want = rda.range_doppler(img, x, y, args)[:y, :x]
    src = st.DevicePaddedImage(_dev(gpu, img), x, y)
    out = st.range_doppler_algorithm(p["prf"], p["wavelength"], p["range_spacing"], p["slant_range"], p["az_bw_frac"],
                                     p["vr"], p["dc"], src, _dev(gpu, np.zeros_like(img)), lib=lib)
    got = out.data.cpu().numpy() if gpu else out.data
    got = got[:y, :x]
    err = np.sqrt(np.mean(np.abs(got - want) ** 2) / np.mean(np.abs(want) ** 2))
    assert err < 2e-6, err
