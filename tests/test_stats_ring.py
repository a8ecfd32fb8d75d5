"""Raw statistics through the shared-memory ring (lines off 8-byte boundaries): every even place of the
raw buffer in a 16-byte unit, line strides with and without bytes between the records, last batches of
one and of seven lines, blocks whose records start at one place (windows checked once) beside blocks
where they do not, and a buffer that ends with its last record.

The sums are integers, so every result equals that of the 8-byte aligned lines bit for bit.
"""
from __future__ import annotations

import copy

import numpy as np
import pytest

import asarf
from asarf import scene as S


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    return request.getfixturevalue(f"{request.param}_lib"), request.param == "gpu"


def _stats(lib, gpu, sc, rows, stride, shift, codes):
    na, spl = rows.shape[0], rows.shape[1] // 2
    sc = copy.copy(sc)
    sc.__class__ = type("Strided", (S.Scene,), {"raw_line_bytes": stride})  # bytes between the records
    plan = asarf.FocusPlan(sc, lib=lib)
    size = shift + (na - 1) * stride + 2 * spl  # ends with the last record
    buf = np.full(size + 64, 255, dtype=np.uint8)
    o = (-buf.ctypes.data) % 16
    view = buf[o + shift:o + size]
    for y in range(na):
        view[y * stride:y * stride + 2 * spl] = rows[y]
    mn = 0 if codes is None else int(codes.min())
    if gpu:
        import torch
        d = torch.from_numpy(buf[o:o + size].copy()).cuda()
        sw = None if codes is None else torch.from_numpy(codes.view(np.int16)).cuda()
        out = torch.zeros(plan.out_shape, dtype=torch.float32, device="cuda")
        plan.focus(d[shift:], out, sw, mn)
        torch.cuda.synchronize()
    else:
        plan.focus(view, np.zeros(plan.out_shape, dtype=np.float32), codes, mn)
    res = plan.results()
    plan.close()
    assert res["errors"] == 0
    return [res[k] for k in ("dc_i", "dc_q", "stddev_i", "stddev_q", "iq_gain", "phase_error")] + list(res["dc_block_hz"])


@pytest.mark.parametrize("na", [257, 263])
@pytest.mark.parametrize("steps", [0, 1])
@pytest.mark.parametrize("nr", [769, 1301])
def test_every_alignment_gives_the_aligned_statistics(be, na, steps, nr):
    lib, gpu = be
    codes = (np.arange(na) // 90 % 3).astype(np.uint16) + 700 if steps else None
    sc = S.tiny(range_size=nr, azimuth_size=na, swst_codes=codes)
    sc.prepare(lib)
    spl = sc.samples_per_line
    rng = np.random.default_rng(na + nr + steps)
    rows = np.clip(np.rint(rng.normal(15.8, 4.0, (na, 2 * spl))), 0, 31).astype(np.uint8)
    want = _stats(lib, gpu, sc, rows, (2 * spl + 7) // 8 * 8, 0, codes)
    for shift in range(0, 16, 2) if gpu else (2, 12):
        for stride in (2 * spl, 2 * spl + 2, 2 * spl + 38):
            assert _stats(lib, gpu, sc, rows, stride, shift, codes) == want, (shift, stride)
