"""The level-0 gathers move 16-byte units between any alignments of packet and record: every
byte against the oracle's parse for packet buffers, raw buffers and record sizes at all
alignments, records shorter than one unit included; nothing outside the records is written.
Bytes are moved, so they must be equal.
"""
from __future__ import annotations

import numpy as np
import pytest

from asarf import l0
from oracle import l0 as ol0


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


def _at(gpu, data: np.ndarray, shift: int):
    """(kept buffer, pointer) of data placed `shift` bytes past a 16-byte boundary."""
    buf = np.zeros(data.size + 64, dtype=np.uint8)
    if gpu:
        import torch
        buf[shift:shift + data.size] = data.reshape(-1)
        t = torch.from_numpy(buf).cuda()
        assert t.data_ptr() % 16 == 0
        return t, t.data_ptr() + shift
    o = (-buf.ctypes.data) % 16 + shift
    buf[o:o + data.size] = data.reshape(-1)
    return buf, buf.ctypes.data + o


def _bytes(gpu, keep, ptr, n):
    whole = keep.cpu().numpy() if gpu else keep
    o = ptr - (keep.data_ptr() if gpu else keep.ctypes.data)
    rest = np.concatenate([whole[:o], whole[o + n:]])
    return whole[o:o + n].copy(), rest


def _u32(gpu):
    keep, ptr = _at(gpu, np.zeros(4, dtype=np.uint8), 0)
    return keep, ptr


@pytest.mark.parametrize("blob_shift", [0, 2, 6, 14])
@pytest.mark.parametrize("raw_shift", [0, 2, 8])
def test_ers_unpack_at_every_alignment(be, blob_shift, raw_shift):
    lib, gpu = be
    rng = np.random.default_rng(11)
    n = 9  # consecutive packets start 10 bytes further into a 16-byte word: all even alignments
    blob = l0.write_packets(rng.integers(0, 256, (n, l0.MEASUREMENT_BYTES), dtype=np.uint8),
                            np.arange(n) + 700, np.full(n, 2820), np.arange(n) + 5, np.arange(n) * 600)
    offs = np.arange(n, dtype=np.int64) * l0.MDSR_BYTES
    offs[4] = offs[3]
    kb, pb = _at(gpu, blob, blob_shift)
    ko, po = _at(gpu, offs.view(np.uint8), 0)
    fill = np.full(n * l0.MEASUREMENT_BYTES, 0xEE, dtype=np.uint8)
    kr, pr = _at(gpu, fill, raw_shift)
    ke, pe = _u32(gpu)
    l0.unpack(pb, po, n, pr, None, None, pe, lib=lib)
    if gpu:
        import torch
        torch.cuda.synchronize()
    got, rest = _bytes(gpu, kr, pr, fill.size)
    ref = ol0.parse(blob, offs)
    assert np.array_equal(got.reshape(n, -1), ref["raw"])
    assert not rest.any()
    assert not _bytes(gpu, ke, pe, 4)[0].any()


@pytest.mark.parametrize("record_bytes", [3, 17, 18, 31, 33, 34, 48, 65, 66, 129, 5288, 5706, 5707])
@pytest.mark.parametrize("shift", [0, 1, 7, 14])
def test_asar_unpack_at_every_alignment(be, record_bytes, shift):
    lib, gpu = be
    rng = np.random.default_rng(record_bytes)
    n = 18
    rec = np.zeros((n, record_bytes), dtype=np.uint8)
    for i in range(n):  # one record in three is shorter than the rest, one of them empty
        ln = record_bytes - 2 if i % 3 else max(0, record_bytes - 2 - 5 * i)
        rec[i, 0], rec[i, 1] = ln & 0xFF, ln >> 8
        rec[i, 2:2 + ln] = rng.integers(0, 256, size=ln, dtype=np.uint8)
    blob, num = l0.write_asar_packets(rec, np.arange(n) + 900, np.full(n, 11628), np.arange(n) * 605)
    src = np.cumsum([0] + [68 + (int(r[0]) | int(r[1]) << 8) for r in rec[:-1]]).astype(np.int64)
    kb, pb = _at(gpu, blob, shift)
    ks, ps = _at(gpu, src.view(np.uint8), 0)
    kr, pr = _at(gpu, np.full(rec.size, 0xEE, dtype=np.uint8), (3 * shift) % 16)
    ke, pe = _u32(gpu)
    l0.asar_unpack(pb, ps, n, record_bytes, pr, None, None, pe, lib=lib)
    if gpu:
        import torch
        torch.cuda.synchronize()
    got, rest = _bytes(gpu, kr, pr, rec.size)
    assert np.array_equal(got.reshape(rec.shape), rec)
    assert not rest.any()
    assert not _bytes(gpu, ke, pe, 4)[0].any()
