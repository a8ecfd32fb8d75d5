"""FBAQ4 statistics at the edges of their tiles: line counts around the tile height and the warps'
shares of it, tile rows whose records all have one shift and length (one place per column) beside
rows with one odd record (the masked path), record lengths of whole blocks and of partial ones; and
the records at every alignment, which range compression stages from.

The sums are FP64 in a fixed order: against numpy's FP64 sums they agree to the order's rounding,
n * 2^-53 at most (n <= 4200 * 300 products: 2e-10), and the corrected constants that follow to two
roundings to float32 (2.4e-7); the image must not depend on the records' address.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import fbaq
from asarf import scene as S


@pytest.fixture(params=["emu", pytest.param("gpu", marks=pytest.mark.gpu)])
def be(request):
    if request.param == "emu":
        return request.getfixturevalue("emu_lib"), False
    return request.getfixturevalue("gpu_lib"), True


def _decode(rec, sc):
    ti, tq = sc.fbaq_tables
    na, nr = sc.azimuth_size, sc.range_size
    iv, qv, ok = np.zeros((na, nr)), np.zeros((na, nr)), np.zeros((na, nr), dtype=bool)
    off = np.zeros(na, int) if sc.swst_codes is None else (sc.swst_codes.astype(int) - int(sc.swst_codes.min()))
    for y in range(na):
        length = int(rec[y, 0]) | int(rec[y, 1]) << 8
        n = fbaq.record_samples(length)
        r = np.arange(n)
        ids, cw = rec[y, 2 + 64 * (r // 63)].astype(int), rec[y, 2 + r + r // 63 + 1].astype(int)
        x = r + off[y]
        keep = x < nr
        iv[y, x[keep]] = ti[fbaq.table_index(ids, cw >> 4)][keep]
        qv[y, x[keep]] = tq[fbaq.table_index(ids, cw & 15)][keep]
        ok[y, x[keep]] = True
    return iv, qv, ok


@pytest.mark.parametrize("lines,odd", [(2048, None), (2049, None), (2300, 2100), (4100, 5), (300, None), (300, 299)])
@pytest.mark.parametrize("nr", [252, 263])
def test_statistics_match_numpy(be, lines, odd, nr):
    lib, gpu = be
    if not gpu and lines > 2300:
        pytest.skip("the emulation takes one thread")
    codes = np.full(lines, 700, dtype=np.uint16)
    counts = np.full(lines, nr - 2 if odd is not None else nr)
    if odd is not None:
        codes[odd] = 702          # one record starts two samples later
        counts[odd // 2] = 40     # and one is short
    sc = S.tiny_fbaq(range_size=nr, azimuth_size=lines, swst_codes=codes if odd is not None else None,
                     record_samples=counts)
    sc.prepare(lib)
    rng = np.random.default_rng(lines + nr)
    spl = sc.samples_per_line
    rec = fbaq.encode(rng.normal(0.4, 8.0, (lines, spl)), rng.normal(0.2, 7.5, (lines, spl)), counts, sc.raw_line_bytes)
    iv, qv, ok = _decode(rec, sc)
    n = np.float32(ok.sum())
    dci, dcq = np.float32(iv.sum()) / n, np.float32(qv.sum()) / n
    plan = asarf.FocusPlan(sc, lib=lib, ref_compat_stats=False)
    first = None
    for shift in (0, 1, 7):
        buf = np.zeros(rec.size + 32, dtype=np.uint8)
        sw = None if odd is None else codes
        if gpu:
            import torch
            buf[shift:shift + rec.size] = rec.reshape(-1)
            d = torch.from_numpy(buf).cuda()
            out = torch.zeros(plan.out_shape, dtype=torch.float32, device="cuda")
            s = None if sw is None else torch.from_numpy(sw.view(np.int16)).cuda()
            plan.focus(d[shift:], out, s, 700 if odd is not None else 0)
            torch.cuda.synchronize()
            img = out.cpu().numpy()
        else:
            buf[shift:shift + rec.size] = rec.reshape(-1)
            img = np.zeros(plan.out_shape, dtype=np.float32)
            plan.focus(buf[shift:], img, sw, 700 if odd is not None else 0)
        res = plan.results()
        assert res["errors"] == 0
        assert res["dc_i"] == pytest.approx(float(dci), rel=2.4e-7) and res["dc_q"] == pytest.approx(float(dcq), rel=2.4e-7)
        ci, cq = (iv - res["dc_i"]) * ok, (qv - res["dc_q"]) * ok
        gain = np.sqrt((ci ** 2).sum() / (cq ** 2).sum())
        assert res["iq_gain"] == pytest.approx(gain, rel=1e-9)
        g = float(np.float32(gain))
        delta = ((ci * cq).sum() / g) / ((ci ** 2).sum() / (g * g))
        assert res["phase_error"] == pytest.approx(np.degrees(np.arcsin(delta)), abs=1e-8)
        # lag-1 angle of every Doppler block from the corrected samples
        z = ci / g + 1j * (cq - ci / g * float(np.float32(delta))) / float(np.float32(1 - delta * delta)) * ok
        acc = (np.conj(z[:-1]) * z[1:]).sum(0)
        step = nr // 32
        for b in range(res["n_dc_blocks"]):
            a = acc[b * step:(b + 1) * step].sum()
            assert res["dc_block_hz"][b] == pytest.approx(sc.prf * np.angle(a) / (2 * np.pi), abs=1e-5)
        if first is None:
            first = img
        assert np.array_equal(img, first)
    plan.close()
