"""ERS level-0 gathers into raw buffers at any byte, odd ones included, from packets at any even byte: the
16-byte aligned interior of every line moves by units and its ends by bytes.  Bytes are moved, so they
must be equal, and nothing outside the raw lines is written.
"""
from __future__ import annotations

import numpy as np
import pytest

from asarf import l0
from test_l0_alignment import _at, _bytes, _u32, be  # noqa: F401


@pytest.mark.parametrize("raw_shift", [1, 2, 3, 4, 7, 8, 13, 14, 15])
@pytest.mark.parametrize("blob_shift", [0, 10])
def test_every_byte_of_a_raw_buffer(be, raw_shift, blob_shift):  # noqa: F811
    lib, gpu = be
    rng = np.random.default_rng(raw_shift)
    n = 9
    lines = rng.integers(0, 256, (n, l0.MEASUREMENT_BYTES), dtype=np.uint8)
    blob = l0.write_packets(lines, np.arange(n) + 700, np.full(n, 2820), np.arange(n) + 5, np.arange(n) * 600)
    kb, pb = _at(gpu, blob, blob_shift)
    ko, po = _at(gpu, (np.arange(n, dtype=np.int64) * l0.MDSR_BYTES).view(np.uint8), 0)
    kr, pr = _at(gpu, np.full(lines.size, 0xEE, dtype=np.uint8), raw_shift)
    ke, pe = _u32(gpu)
    l0.unpack(pb, po, n, pr, None, None, pe, lib=lib)
    if gpu:
        import torch
        torch.cuda.synchronize()
    got, rest = _bytes(gpu, kr, pr, lines.size)
    assert np.array_equal(got.reshape(n, -1), lines)
    assert not rest.any()
    assert not _bytes(gpu, ke, pe, 4)[0].any()
