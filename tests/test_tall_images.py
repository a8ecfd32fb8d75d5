"""Per-stage calls over images with more rows than a launch grid is high (65535 blocks): 32 rows a block in
the spreading-loss and ground-range kernels, 256 in the Doppler sums.

The images are narrow, so that the rows past the limit are what the tests see: first, middle and last rows
against numpy.  Spreading loss and resampling are one float32 product and one multiply-add each: exact
for the product with the call's own gain table (row 0 against every row), 2e-7 for the resampling.  The Doppler
fit is FP64 over FP64 sums: 1e-9 relative.
"""
from __future__ import annotations

import numpy as np
import pytest

from asarf import stages as st

pytestmark = pytest.mark.gpu
ROWS = 65535 * 32 + 77


def test_range_spreading_loss(gpu_lib):
    import torch

    x = 5
    row = torch.tensor([1.0, 2.0, 3.0, 5.0, 7.0], device="cuda")
    scale = torch.arange(ROWS, device="cuda").remainder(3).add(1).float()
    img = row[None, :] * torch.exp2(scale)[:, None]  # powers of two: the product scales exactly
    st.range_spreading_loss_correction(img, 830000.0, 7.9, 850000.0, lib=gpu_lib)
    ratio = 850000.0 / (830000.0 + np.arange(x) * 7.9)
    want = row.cpu().numpy() * np.float32(1.0 / np.sqrt(ratio ** 3.0)) * 2.0
    assert np.allclose(img[0].cpu().numpy(), want, rtol=2e-7, atol=0)
    assert torch.equal(img, img[0][None, :] * torch.exp2(scale - 1.0)[:, None])


def test_ground_range(gpu_lib):
    import torch

    poly = np.array([0.0, 0.0, 0.0, 0.8, 0.5])
    in_x, out_x = 40, 9
    row = torch.linspace(1.0, 9.0, in_x, device="cuda") ** 2
    k = torch.arange(ROWS, device="cuda").remainder(4).float()
    img = row[None, :] * torch.exp2(k)[:, None]
    out = torch.zeros(ROWS, out_x, device="cuda")
    st.srgr_interpolation(img, poly, 7.9, out, lib=gpu_lib)
    start = torch.zeros(out_x, dtype=torch.int32, device="cuda")
    frac = torch.zeros(out_x, device="cuda")
    st.srgr_index(poly, 7.9, start, frac, lib=gpu_lib)
    r, s, f = row.cpu().double().numpy(), start.cpu().numpy(), frac.cpu().double().numpy()
    assert np.allclose(out[0].cpu().numpy(), r[s] + f * (r[s + 1] - r[s]), rtol=2e-7, atol=0)
    assert torch.equal(out, out[0][None, :] * torch.exp2(k)[:, None])


def test_doppler_centroid(gpu_lib):
    import torch

    x, y, prf = 32, 65535 * 256 + 300, 1680.0  # 4.3 GB
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    img = torch.empty(y, x, dtype=torch.complex64, device="cuda")
    acc = torch.zeros(x, dtype=torch.complex128, device="cuda")
    step = 1 << 20
    f = (100.0 + 2.0 * torch.arange(x, device="cuda").double()) / prf
    for y0 in range(0, y, step):
        n = min(step, y - y0)
        # the centroid drifts along the rows, so that rows left out would move the sums
        t = torch.arange(y0, y0 + n, device="cuda").double()[:, None]
        ph = 2 * np.pi * torch.remainder(t * f[None, :] + 0.5 * (60.0 / prf) * t * t / y, 1.0)
        z = torch.polar(torch.ones_like(ph), ph).to(torch.complex64)
        z += 0.1 * torch.view_as_complex(torch.randn(n, x, 2, generator=gen, device="cuda"))
        img[y0:y0 + n] = z
        lo = max(y0 - 1, 0)
        w = img[lo:y0 + n].to(torch.complex128)
        acc += (w[:-1].conj() * w[1:]).sum(0)
        del t, ph, z, w
    poly = st.calculate_doppler_centroid(st.DevicePaddedImage(img, x, y), prf, lib=gpu_lib)
    hz = prf * np.angle(acc.cpu().numpy()) / (2 * np.pi)
    xs = np.array([(2 * k + 1) // 2 for k in range(x)], dtype=float)
    want = np.polyfit(xs, hz, 2)
    assert np.polyval(poly, xs) == pytest.approx(np.polyval(want, xs), rel=1e-9)
