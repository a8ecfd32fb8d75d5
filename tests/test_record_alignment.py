"""Level-1 records leave the device in 16-byte units whatever the record size and header: every
byte of IMS records against the oracle, of IMP records against the two-byte values of the same
call with no header at an aligned address, at sizes around the units and the staged chunks;
nothing outside the records is written.
"""
from __future__ import annotations

import numpy as np
import pytest

from asarf import stages as st
from oracle import rda

CAL = 3.7


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


def _host(gpu, x):
    return np.asarray(x).copy() if not gpu else x.cpu().numpy()


@pytest.mark.parametrize("x", [1, 3, 4, 5, 8, 9, 63, 2047, 2048, 2049, 2053, 4896])
@pytest.mark.parametrize("hdr", [0, 1, 15, 17])
def test_ims_records_match_oracle(be, x, hdr):
    lib, gpu = be
    rng = np.random.default_rng(x)
    img = ((rng.standard_normal((5, x + 3)) + 1j * rng.standard_normal((5, x + 3))) * 6000).astype(np.complex64)
    img[0, 0] = complex(np.nan, 1e9)
    n = 5 * (hdr + 4 * x)
    dest = _dev(gpu, np.full(n + 40, 0xAB, dtype=np.uint8))
    st.condition_slc(_dev(gpu, img), x, dest[3:], hdr, CAL, lib=lib)
    got = _host(gpu, dest)
    assert np.array_equal(got[3:3 + n].reshape(5, -1), rda.condition_slc(img[:, :x], CAL, hdr))
    assert (got[:3] == 0xAB).all() and (got[3 + n:] == 0xAB).all()


@pytest.mark.parametrize("x", [1, 2, 3, 7, 8, 9, 17, 4095, 4096, 4097, 4105, 7000])
@pytest.mark.parametrize("hdr", [0, 1, 17])
def test_imp_records_have_the_same_values_at_every_alignment(be, x, hdr):
    lib, gpu = be
    rng = np.random.default_rng(x)
    img = (rng.exponential(1.0, (5, x)) * 10.0 ** rng.uniform(-4, 6, (5, x))).astype(np.float32)
    img[0, 0] = np.nan
    # each pixel as an image of its own row length 1: the value path without units or neighbours
    px = _dev(gpu, img.reshape(-1, 1))
    vals = _dev(gpu, np.zeros(2 * img.size, dtype=np.uint8))
    st.condition_detected(px, vals, 0, CAL, lib=lib)
    want = np.zeros((5, hdr + 2 * x), dtype=np.uint8)
    want[:, hdr:] = _host(gpu, vals).reshape(5, -1)
    n = want.size
    dest = _dev(gpu, np.full(n + 40, 0xAB, dtype=np.uint8))
    st.condition_detected(_dev(gpu, img), dest[5:], hdr, CAL, lib=lib)
    got = _host(gpu, dest)
    assert np.array_equal(got[5:5 + n].reshape(want.shape), want)
    assert (got[:5] == 0xAB).all() and (got[5 + n:] == 0xAB).all()
    ref = rda.condition_detected(img, CAL, hdr)[:, hdr:].reshape(5, x, 2).astype(np.int64)
    g = want[:, hdr:].reshape(5, x, 2).astype(np.int64)
    assert np.abs((g[..., 0] | g[..., 1] << 8) - (ref[..., 0] | ref[..., 1] << 8)).max() <= 1
