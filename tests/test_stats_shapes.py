"""Raw statistics at the sizes where the block height and the window form change: few lines,
grids below and above one wave, raw buffers and line strides of every even alignment, record
edges inside a 4-column group; and the same plan run twice, since a run leaves its accumulators
zero for the next.  The sums are integers, so the IQ statistics must equal numpy's closed form to
the last bit of the float they are rounded to, whatever the path.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import scene as S


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


def _scene(lib, nr, na, swst=None):
    sc = S.tiny(range_size=nr, azimuth_size=na, swst_codes=swst)
    sc.prepare(lib)
    return sc


def _run(lib, gpu, sc, raw, shift, plan):
    na, lb = raw.shape
    out_n = int(np.prod(plan.out_shape))
    swst = None if sc.swst_codes is None else np.asarray(sc.swst_codes, dtype=np.uint16)
    mn = 0 if swst is None else int(swst.min())
    buf = np.zeros(na * lb + 32, dtype=np.uint8)
    if gpu:
        import torch
        buf[shift:shift + na * lb] = raw.reshape(-1)
        d = torch.from_numpy(buf).cuda()
        out = torch.zeros(out_n, dtype=torch.float32, device="cuda")
        sw = None if swst is None else torch.from_numpy(swst.view(np.int16)).cuda()
        plan.focus(d[shift:], out, sw, mn)
        torch.cuda.synchronize()
        img = out.cpu().numpy()
    else:
        buf = np.zeros(na * lb + 64, dtype=np.uint8)
        o = (-buf.ctypes.data) % 16 + shift
        buf[o:o + na * lb] = raw.reshape(-1)
        out = np.zeros(out_n, dtype=np.float32)
        plan.focus(buf[o:], out, swst, mn)
        img = out
    return img, plan.results()


@pytest.mark.parametrize("nr,na", [(515, 300), (768, 1024), (1037, 409), (773, 2500)])
@pytest.mark.parametrize("steps", [0, 1])
def test_statistics_equal_the_closed_form(be, nr, na, steps):
    lib, gpu = be
    if not gpu and na > 1100:
        na = 1111
    codes = (np.arange(na) // 97 % 3).astype(np.uint16) + 700 if steps else None
    sc = _scene(lib, nr, na, codes)
    rng = np.random.default_rng(nr + na)
    spl = sc.samples_per_line
    iq = np.clip(np.rint(rng.normal(15.8, 4.0, (na, spl, 2))), 0, 31).astype(np.uint8)
    raw = iq.reshape(na, -1)
    i, q = iq[..., 0].astype(np.float64), iq[..., 1].astype(np.float64)
    total = np.float32(i.size)
    dci, dcq = np.float32(i.sum()) / total, np.float32(q.sum()) / total
    sd = [float(np.sqrt(np.float32(((v - float(d)) ** 2).sum()) / total)) for v, d in ((i, dci), (q, dcq))]
    plan = asarf.FocusPlan(sc, lib=lib)
    first = None
    for shift in (0, 2, 4, 6, 0):  # the same plan each time
        img, res = _run(lib, gpu, sc, raw, shift, plan)
        assert res["errors"] == 0
        assert (res["dc_i"], res["dc_q"]) == (float(dci), float(dcq))
        # the closed form's FP64 cancellation (about 1e-13) can move the float by its last bit
        assert res["stddev_i"] == pytest.approx(sd[0], rel=2e-7) and res["stddev_q"] == pytest.approx(sd[1], rel=2e-7)
        got = (res["iq_gain"], res["phase_error"], tuple(res["dc_block_hz"]), tuple(res["doppler_centroid_poly"]))
        if first is None:
            first = (got, img)
        assert got == first[0]
        assert np.array_equal(img, first[1])
    poly = np.polyfit([(b * (nr // 32) + (b + 1) * (nr // 32)) // 2 for b in range(res["n_dc_blocks"])],
                      res["dc_block_hz"], 2)
    x = np.arange(nr)
    assert np.allclose(np.polyval(res["doppler_centroid_poly"], x), np.polyval(poly, x), rtol=0, atol=1e-8)
    plan.close()
