"""The work that users of this framework have it do, as measurable cases.

Each case is one call (or one call chain) through the public entry points of ``asarf``:

* ``focus``    a scene from device-resident raw records to the detected ground-range image,
               and to the complex SLC as well where the caller asks for it (``FocusPlan``);
* ``host``     the same from page-locked host memory to page-locked host memory, the call that
               replaces the processing span of a one-file-per-process host flow;
* ``batch``    uneven segments focused together (``FocusBatch``);
* ``strip``    a long strip in overlapped azimuth blocks (``FocusStrip``);
* ``stages``   the per-stage entry points one after another, as a caller does who keeps the
               original main flow and swaps its stages for these (``asarf.stages``);
* ``l0``       level-0 packets to raw lines or FBAQ4 records (``asarf.l0``);
* ``records``  level-1 MDS records from a complex and a detected image (``asarf.stages``).

Raw data are synthetic: clutter with the beam's azimuth spectrum around the Doppler centroid
and a grid of point targets, through the range and azimuth chirps, plus noise, front-end
impairments and the sensor's quantisation.  Everything is made on the GPU from the seed.
``exact`` restates the processing in 64 bits with torch and numpy; where the processor decides
something by a 32-bit value (range walk, Doppler bin, band edge, aliasing, resampling index,
filter phases) the restatement takes the same 32-bit value, since those define the result.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "asar-focus_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import asarf  # noqa: E402
from asarf import l0, stages  # noqa: E402

DEV = "cuda"
SOL = 299792458.0
R_EARTH = 6378137.0
B_EARTH = 6356752.314245
GM = 3.986004418e14
T0_US = 1_000_000_000
ERS_PACKET, ERS_DATA = 11498, 11232

# Sensor parameters of the repository's workloads: ERS-like, ENVISAT ASAR IM-like, and the small
# low-orbit geometry of its tests (short chirp and aperture).  dc: Doppler centroid in Hz against
# normalised range, sigma: raw clutter deviation in counts.
SENSORS = {
    "ers": dict(fs=18.96e6, pulse=37.12e-6, bw=15.55e6, prf=1680.0, lam=0.05656, near=830000.0, alt=800000.0,
                vr=(3.0e-9, -1.35e-3, 7123.0), dc=(250.0, 100.0), bits=5, sigma=4.0),
    "asar": dict(fs=19.208e6, pulse=27.1e-6, bw=16.0e6, prf=1652.0, lam=0.05624, near=830000.0, alt=800000.0,
                 vr=(3.0e-9, -1.33e-3, 7121.0), dc=(-200.0, 250.0, 100.0), bits=8, sigma=30.0),
    "tiny": dict(fs=18.96e6, pulse=6.0e-6, bw=15.55e6, prf=1680.0, lam=0.05656, near=100000.0, alt=80000.0,
                 vr=(0.0, 0.0, 7100.0), dc=(300.0,), bits=5, sigma=4.0),
}


def listed():
    return [
        # a small quick-look cut: the shortest call, bound by launches and latency
        dict(name="focus_small", kind="focus", sensor="tiny", range=768, lines=1024, fmt="bytes", swst=False,
             slc=False, keep_slc=True, abs_phase=False),
        # a full ERS scene to its detected image, nothing else kept: the headline workload
        dict(name="focus_ers", kind="focus", sensor="ers", range=5616, lines=28000, fmt="bytes", swst=False,
             slc=False, keep_slc=False, abs_phase=False),
        # part of an ERS pass with changes of the sampling window and odd sizes, default options
        dict(name="focus_ers_swst", kind="focus", sensor="ers", range=5644, lines=9973, fmt="bytes", swst=True,
             slc=False, keep_slc=True, abs_phase=False),
        # ASAR 8-bit samples to an SLC with absolute phase, for interferometry, and its quick-look
        dict(name="focus_asar_slc", kind="focus", sensor="asar", range=5193, lines=17011, fmt="bytes", swst=False,
             slc=True, keep_slc=True, abs_phase=True),
        # a full ENVISAT ASAR scene in the instrument's own FBAQ4 records
        dict(name="focus_asar_fbaq", kind="focus", sensor="asar", range=5616, lines=30000, fmt="fbaq4", swst=False,
             slc=False, keep_slc=True, abs_phase=False),
        # one small scene from host memory to host memory, copies included
        dict(name="host_ers", kind="host", sensor="ers", range=2048, lines=4096, fmt="bytes", swst=False),
        # a queue of uneven segments of both sensors in one graph
        dict(name="batch_mixed", kind="batch", segments="ers:2048x4507 asar:5616x6121 ers:5616x4999 asar:2048x11831 "
             "ers:5616x9203 asar:2048x5003"),
        # a long strip with a drifting Doppler centroid in overlapped blocks
        dict(name="strip_asar", kind="strip", range=5616, lines=40000, block=16384, overlap=1400),
        # the main flow stage by stage over padded images
        dict(name="stages_ers", kind="stages", sensor="ers", range=5616, lines=7000),
        # level-0 packets of an ERS pass and of an ASAR pass (calibration packets among them)
        dict(name="l0_ers", kind="l0", sensor="ers", lines=28000, samples=5616),
        dict(name="l0_asar", kind="l0", sensor="asar", lines=30000, samples=5203),
        # product records of an SLC and of a detected image
        dict(name="records", kind="records", rows=5003, cols=4896),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    pick = rng.random()
    if pick < 0.55:
        sensor = rng.choice(["ers", "ers", "asar", "asar", "tiny"])
        if sensor == "tiny":
            nr, na = log_int(512, 1536), log_int(900, 4000)
        else:
            nr, na = rng.choice([5616, rng.randint(2048, 5700)]), log_int(3000, 27000)
        fmt = "fbaq4" if sensor == "asar" and rng.random() < 0.5 else "bytes"
        swst = fmt == "bytes" and sensor == "ers" and rng.random() < 0.3
        slc = rng.random() < 0.3
        return dict(kind="focus", sensor=sensor, range=nr, lines=na, fmt=fmt, swst=swst, slc=slc,
                    keep_slc=slc or rng.random() < 0.5, abs_phase=slc and rng.random() < 0.5)
    if pick < 0.62:
        return dict(kind="host", sensor=rng.choice(["ers", "asar"]), range=rng.randint(1600, 5616),
                    lines=log_int(3000, 9000), fmt="bytes", swst=False)
    if pick < 0.70:
        segs = ["%s:%dx%d" % (rng.choice(["ers", "asar"]), rng.choice([2048, 5616]), rng.randint(4000, 9000))
                for _ in range(rng.randint(2, 6))]
        return dict(kind="batch", segments=" ".join(segs))
    if pick < 0.76:
        return dict(kind="strip", range=rng.randint(2048, 5616), lines=rng.randint(17000, 34000),
                    block=rng.choice([6000, 8192, 16384]), overlap=rng.randint(1400, 1600))
    if pick < 0.86:
        return dict(kind="stages", sensor=rng.choice(["ers", "asar"]), range=rng.randint(1600, 5616),
                    lines=log_int(3000, 7000))
    if pick < 0.94:
        sensor = rng.choice(["ers", "asar"])
        return dict(kind="l0", sensor=sensor, lines=log_int(1500, 28000),
                    samples=5616 if sensor == "ers" else rng.randint(2000, 5616))
    return dict(kind="records", rows=log_int(500, 5000), cols=rng.randint(1000, 5000))


# ---------------------------------------------------------------------------- scene description

def _vr_at(p, x):
    return (p[0] * x + p[1]) * x + p[2]


def _chirp_samples(p):
    return int(round(p["pulse"] * p["fs"]))


def _orbit(p, lines):
    """State vectors 10 s apart on a circular orbit around the scene's middle line."""
    rs = R_EARTH + p["alt"]
    w = math.sqrt(GM / rs ** 3)
    inc, th0 = math.radians(98.5), math.radians(30.0)
    e1 = np.array([1.0, 0.0, 0.0])
    e2 = np.array([0.0, math.cos(inc), math.sin(inc)])
    span = lines / p["prf"]
    n = max(5, int(math.ceil(span / 10.0)) + 3)
    osv = []
    for k in range(n):
        t = -10.0 * ((n - 1) // 2) + 10.0 * k + span / 2
        th = th0 + w * (t - span / 2)
        pos = rs * (math.cos(th) * e1 + math.sin(th) * e2)
        vel = rs * w * (-math.sin(th) * e1 + math.cos(th) * e2)
        osv.append((T0_US + int(round(t * 1e6)), tuple(float(v) for v in pos), tuple(float(v) for v in vel)))
    return osv


def _interp_orbit(osv, time_us):
    t0 = osv[0][0]
    t = (time_us - t0) * 1e-6
    xs = [(o[0] - t0) * 1e-6 for o in osv]
    pos, vel = np.zeros(3), np.zeros(3)
    for i, o in enumerate(osv):
        m = 1.0
        for j in range(len(osv)):
            if j != i:
                m *= (t - xs[j]) / (xs[i] - xs[j])
        pos += m * np.array(o[1])
        vel += m * np.array(o[2])
    return pos, vel


def _geolocate(vel, pos, guess, slant):
    """Zero-Doppler point of the ellipsoid at a slant range (Newton)."""
    r = np.array(guess, dtype=np.float64)
    for _ in range(100):
        d = r - pos
        a = np.array([vel, 2 * d, [2 * r[0] / R_EARTH ** 2, 2 * r[1] / R_EARTH ** 2, 2 * r[2] / B_EARTH ** 2]])
        b = np.array([vel @ d, d @ d - slant * slant,
                      (r[0] / R_EARTH) ** 2 + (r[1] / R_EARTH) ** 2 + (r[2] / B_EARTH) ** 2 - 1.0])
        dx = np.linalg.solve(a, -b)
        r = r + dx
        if np.linalg.norm(dx) < 1e-6:
            break
    return r


def _line_time_us(first, prf, idx):
    return first + (int((1.0 / prf) * idx * 1e6) & 0xFFFFFFFF)


def _swst_codes(lines, seed):
    """Sampling-window codes that step a few times along a pass (ERS: 4 samples a step)."""
    r = np.random.RandomState(1000 + seed % 100000)
    cuts = np.sort(r.randint(1, lines, 3))
    codes = np.zeros(lines, dtype=np.int64)
    for k, c in enumerate(cuts):
        codes[c:] = (3, 7, 5)[k]
    return (codes + 740).astype(np.uint16)


def _scene(sensor, nr, na, fmt="bytes", swst=None, name="case"):
    """The metadata of a scene as a user's program has it, orbit and centre point included."""
    p = SENSORS[sensor]
    osv = _orbit(p, na)
    pos, vel = _interp_orbit(osv, T0_US + int((1.0 / p["prf"]) * (na // 2) * 1e6))
    up = pos / np.linalg.norm(pos)
    right = np.cross(vel / np.linalg.norm(vel), up)
    spacing = SOL / (2 * p["fs"])
    mid = p["near"] + ((nr - _chirp_samples(p)) // 2) * spacing
    g = up + math.sqrt(max(mid ** 2 - p["alt"] ** 2, 1.0)) / R_EARTH * right
    center = _geolocate(vel, pos, g / np.linalg.norm(g) * R_EARTH, mid)
    vp = float(np.linalg.norm(osv[len(osv) // 2][2]))
    return asarf.Scene(
        name=name, range_size=nr, azimuth_size=na, bits=p["bits"], range_sampling_rate=p["fs"],
        pulse_duration=p["pulse"], chirp_bandwidth=p["bw"], prf=p["prf"], wavelength=p["lam"],
        slant_range_first=p["near"], altitude=p["alt"], raw_format="fbaq4" if fmt == "fbaq4" else "ers",
        swst_codes=swst, osv=osv, center_point=tuple(float(v) for v in center), vr_poly=p["vr"],
        vr_poly_init=(0.0, 0.0, math.sqrt(0.88 * vp * vp)), first_line_time_us=T0_US)


# ---------------------------------------------------------------------------- raw data

def _smooth_above(n):
    while True:
        m = n
        for q in (2, 3, 5, 7):
            while m % q == 0:
                m //= q
        if m == 1:
            return n
        n += 1


def _chirp64(p):
    n = _chirp_samples(p)
    t = (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2) / p["fs"]
    return torch.polar(torch.ones_like(t), math.pi * (p["bw"] / p["pulse"]) * t * t)


def _iq(sensor, nr, na, seed, drift=0.0):
    """Analogue I and Q (float32 [na][nr], in counts around zero) of a scene."""
    p = SENSORS[sensor]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + nr * 31 + na)
    nc = _chirp_samples(p)
    npad, mpad = _smooth_above(na), _smooth_above(nr + nc)
    z = torch.randn(npad, nr, 2, generator=gen, device=DEV).mul_(math.sqrt(0.5))
    z = torch.view_as_complex(z)
    # point targets 30 dB above the clutter, on a jittered grid
    jit = torch.rand(2, 6, 8, generator=gen, device=DEV)
    ys = ((torch.arange(6, device=DEV)[:, None] + 0.2 + 0.6 * jit[0]) * (na / 6)).long().clamp(0, na - 1)
    xs = ((torch.arange(8, device=DEV)[None, :] + 0.2 + 0.6 * jit[1]) * ((nr - nc) / 8)).long().clamp(0, nr - 1)
    z[ys.reshape(-1), xs.reshape(-1)] += 10 ** (30 / 20)
    # range: the transmitted chirp
    hr = torch.fft.fft(_chirp64(p), n=mpad).to(torch.complex64)
    rows = 4096
    for r0 in range(0, npad, rows):
        f = torch.fft.fft(z[r0:r0 + rows], n=mpad, dim=1) * hr
        z[r0:r0 + rows] = torch.fft.ifft(f, dim=1)[:, :nr]
    # azimuth: the beam around the Doppler centroid and the quadratic phase
    fb = torch.fft.fftfreq(npad, d=1.0 / p["prf"], device=DEV, dtype=torch.float64)[:, None]
    beam_bw = 0.95 * p["prf"]
    cols = max(64, (1 << 24) // npad)
    for c0 in range(0, nr, cols):
        x = torch.arange(c0, min(nr, c0 + cols), device=DEV, dtype=torch.float64)[None, :]
        u = x / max(1, nr - 1)
        fdc = sum(c * u ** k for k, c in enumerate(p["dc"] if drift == 0.0 else (0.0,))) + 0.0 * u
        ka = 2 * _vr_at(p["vr"], x) ** 2 / (p["lam"] * (p["near"] + x * SOL / (2 * p["fs"])))
        fa = fb + p["prf"] * torch.round((fdc - fb) / p["prf"])
        off = fa - fdc
        beam = torch.where(off.abs() < beam_bw / 2, torch.cos(math.pi * off / beam_bw) ** 2, torch.zeros_like(off))
        h = torch.polar((beam * (p["prf"] / torch.sqrt(ka))).float(),
                        torch.remainder(math.pi * fa * fa / ka, 2 * math.pi).float())
        z[:, c0:c0 + cols] = torch.fft.ifft(torch.fft.fft(z[:, c0:c0 + cols], dim=0) * h, dim=0)
    z = z[:na]
    if drift:
        ph = 2 * math.pi * torch.cumsum(drift * torch.sin(2 * math.pi * torch.arange(na, device=DEV).double() / na), 0) / p["prf"]
        z = z * torch.polar(torch.ones_like(ph), torch.remainder(ph, 2 * math.pi)).to(torch.complex64)[:, None]
    std = torch.sqrt(torch.view_as_real(z[:, ::16].contiguous()).square().mean())
    z = torch.view_as_real(z) * (p["sigma"] / std)
    z += torch.randn(z.shape, generator=gen, device=DEV) * (0.25 * p["sigma"])
    skew = math.radians(2.0)
    return z[..., 0] * 1.02, z[..., 1] * math.cos(skew) + z[..., 0] * math.sin(skew)


def _encode_bytes(iv, qv, bits):
    mid, top = 2.0 ** (bits - 1) - 0.5 + 0.3, 2.0 ** bits - 1
    raw = torch.empty(iv.shape[0], iv.shape[1], 2, dtype=torch.uint8, device=DEV)
    raw[..., 0] = (iv + mid).round_().clamp_(0, top).to(torch.uint8)
    raw[..., 1] = (qv + mid).round_().clamp_(0, top).to(torch.uint8)
    return raw.reshape(iv.shape[0], -1)


def _fbaq_scale(ids):
    return asarf.scene.fbaq.SIGMA0 * 10.0 ** (ids * (asarf.scene.fbaq.STEP_DB / 20.0))


def _encode_fbaq(iv, qv, record_bytes):
    """FBAQ4 records: per 63 samples a block id (scale) and one code byte per sample."""
    na, n = iv.shape
    nb = (n + 62) // 63
    lev = torch.as_tensor(asarf.scene.fbaq.LEVELS, device=DEV, dtype=torch.float32)
    thr = (lev[1:] + lev[:-1]) / 2
    data = n + nb
    out = torch.zeros(na, record_bytes, dtype=torch.uint8, device=DEV)
    out[:, 0], out[:, 1] = data & 0xFF, data >> 8
    for y0 in range(0, na, 2048):
        i = torch.nn.functional.pad(iv[y0:y0 + 2048] + 0.3, (0, nb * 63 - n)).view(-1, nb, 63)
        q = torch.nn.functional.pad(qv[y0:y0 + 2048] + 0.3, (0, nb * 63 - n)).view(-1, nb, 63)
        rms = torch.sqrt((i * i + q * q).sum(2) / 126)
        bid = torch.round(20 * torch.log10(rms.clamp_min(1e-6) / asarf.scene.fbaq.SIGMA0) /
                          asarf.scene.fbaq.STEP_DB).clamp(0, 255)
        s = _fbaq_scale(bid)[:, :, None]

        def code(v):
            level = torch.bucketize((v / s).contiguous(), thr)
            return torch.where(level >= 8, level - 8, 15 - level)
        blocks = torch.empty(i.shape[0], nb, 64, dtype=torch.uint8, device=DEV)
        blocks[:, :, 0] = bid.to(torch.uint8)
        blocks[:, :, 1:] = (code(i) * 16 + code(q)).to(torch.uint8)
        out[y0:y0 + 2048, 2:2 + data] = blocks.view(i.shape[0], -1)[:, :data]
    return out


def _raw(c, seed):
    """(scene, raw records on the device, SWST codes or None) of a scene case."""
    na, nr = c["lines"], c["range"]
    codes = _swst_codes(na, seed) if c["swst"] else None
    sc = _scene(c["sensor"], nr, na, c["fmt"], codes)
    iv, qv = _iq(c["sensor"], nr, na, seed)
    if codes is not None:
        spl, off = sc.samples_per_line, torch.as_tensor(4 * (codes.astype(np.int64) - codes.min()), device=DEV)
        idx = off[:, None] + torch.arange(spl, device=DEV)[None, :]
        iv, qv = torch.gather(iv, 1, idx), torch.gather(qv, 1, idx)
    if c["fmt"] == "fbaq4":
        return sc, _encode_fbaq(iv, qv, sc.raw_line_bytes), codes
    return sc, _encode_bytes(iv, qv, sc.bits), codes


def _dev_swst(codes):
    return None if codes is None else torch.from_numpy(codes.astype(np.int16)).to(DEV)


# ---------------------------------------------------------------------------- prepare and run

def _segments(c):
    for k, s in enumerate(c["segments"].split()):
        sensor, size = s.split(":")
        nr, na = size.split("x")
        yield k, dict(sensor=sensor, range=int(nr), lines=int(na), fmt="bytes", swst=False)


def _padded(sc):
    return asarf.fft_size_above(sc.azimuth_size), asarf.fft_size_above(sc.range_size + sc.chirp_samples)


def _chirp_padded(p, padding):
    """The windowed, power-normalised replica a host flow hands to range compression."""
    c = _chirp64(p).cpu().numpy()
    n = c.size
    c = c * (0.54 - 0.46 * np.cos(2 * np.pi * np.arange(n) / n))
    out = np.zeros(padding, dtype=np.complex64)
    out[:n] = (c / math.sqrt(float((np.abs(c) ** 2).sum()))).astype(np.complex64)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("focus", "host"):
        sc, raw, codes = _raw(case, seed)
        if kind == "host":
            plan = asarf.FocusPlan(sc)
            h_raw = torch.empty(raw.shape, dtype=torch.uint8, pin_memory=True)
            h_raw.copy_(raw)
            h_out = torch.empty(plan.out_shape, dtype=torch.float32, pin_memory=True)
            return dict(kind=kind, plan=plan, raw=h_raw, out=h_out)
        plan = asarf.FocusPlan(sc, keep_slc=case["keep_slc"], absolute_phase=case["abs_phase"])
        out = torch.zeros(plan.out_shape, dtype=torch.float32, device=DEV)
        slc = None
        if case["slc"]:
            slc = torch.zeros(sc.azimuth_size - plan.dims["max_aperture"], plan.dims["slc_cols"],
                              dtype=torch.complex64, device=DEV)
        return dict(kind=kind, plan=plan, raw=raw, out=out, slc=slc, swst=_dev_swst(codes),
                    min_swst=0 if codes is None else int(codes.min()))
    if kind == "batch":
        made = [_raw(s, seed * 17 + k) for k, s in _segments(case)]
        batch = asarf.FocusBatch([m[0] for m in made])
        outs = [torch.zeros(p.out_shape, dtype=torch.float32, device=DEV) for p in batch.plans]
        return dict(kind=kind, batch=batch, raws=[m[1] for m in made], outs=outs)
    if kind == "strip":
        sc = _scene("asar", case["range"], case["lines"])
        iv, qv = _iq("asar", case["range"], case["lines"], seed, drift=100.0)
        strip = asarf.FocusStrip(sc, case["block"], case["overlap"])
        return dict(kind=kind, strip=strip, raw=_encode_bytes(iv, qv, sc.bits),
                    out=torch.zeros(strip.out_shape, dtype=torch.float32, device=DEV))
    if kind == "stages":
        sc, raw, _ = _raw(dict(case, fmt="bytes", swst=False), seed)
        p = SENSORS[case["sensor"]]
        az_pad, rg_pad = _padded(sc)
        nx = sc.range_size - sc.chirp_samples - 16
        near = p["near"] + 8 * sc.range_spacing
        rows = sc.azimuth_size - _aperture(sc, p)
        ratio = np.float32(12.5 / sc.azimuth_spacing)
        looks = int(_round_away(float(np.float32(rows) / ratio)))
        poly, ng = stages.srgr_polynomial(sc, near, nx, looks, (1.0 / p["prf"]) * float(ratio))
        return dict(kind=kind, sc=sc, p=p, raw=raw, rows=rows, nx=nx, near=near, poly=poly,
                    chirp=_chirp_padded(p, rg_pad),
                    image=torch.zeros(az_pad, rg_pad, dtype=torch.complex64, device=DEV),
                    work=torch.zeros(az_pad, rg_pad, dtype=torch.complex64, device=DEV),
                    looks=torch.zeros(looks, nx, dtype=torch.float32, device=DEV),
                    ground=torch.zeros(looks, ng, dtype=torch.float32, device=DEV))
    if kind == "l0":
        return _prepare_l0(case, seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    rows, cols = case["rows"], case["cols"]
    # speckle: complex Gaussian pixels of varying local power, some past the 16-bit range
    power = torch.exp(1.5 * torch.randn(rows, cols, generator=gen, device=DEV))
    slc = torch.view_as_complex(torch.randn(rows, cols, 2, generator=gen, device=DEV)) * (900.0 * power)
    return dict(kind=kind, slc=slc, det=(slc.abs() ** 2)[: max(1, rows // 5)].contiguous(),
                ims=torch.zeros(rows, 17 + 4 * cols, dtype=torch.uint8, device=DEV),
                imp=torch.zeros(max(1, rows // 5), 17 + 2 * cols, dtype=torch.uint8, device=DEV), cols=cols)


def _prepare_l0(case, seed):
    n = case["lines"]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    swst = torch.randint(700, 760, (n,), generator=gen, device=DEV)
    if case["sensor"] == "ers":
        pk = torch.randint(0, 32, (n, ERS_PACKET), generator=gen, device=DEV, dtype=torch.uint8)
        pk[:, 24], pk[:, 25], pk[:, 46] = 11465 >> 8, 11465 & 0xFF, 0xAA
        pk[:, 58], pk[:, 59], pk[:, 60], pk[:, 61] = swst >> 8, swst & 0xFF, 2820 >> 8, 2820 & 0xFF
        # a few lost packets are filled by the one before them
        src = torch.arange(n, device=DEV)
        lost = torch.randint(1, n, (max(1, n // 500),), generator=gen, device=DEV)
        src[lost] -= 1
        return dict(kind="l0", sensor="ers", n=n, blob=pk.reshape(-1), src=src * ERS_PACKET,
                    raw=torch.zeros(n, ERS_DATA, dtype=torch.uint8, device=DEV), **_l0_side(n))
    data = case["samples"] + (case["samples"] + 62) // 63
    size = 68 + data
    pk = torch.randint(0, 256, (n, size), generator=gen, device=DEV, dtype=torch.uint8)
    length = data + 29
    for at, v in ((24, length), (36, length), (38, 29), (54, 3300)):
        pk[:, at], pk[:, at + 1] = v >> 8, v & 0xFF
    pk[:, 41], pk[:, 52] = 0x54, 0x80
    pk[:, 56], pk[:, 57] = swst >> 8, swst & 0xFF
    # every 1024th packet is a calibration one: its line repeats the echo before it
    src = torch.arange(n, device=DEV)
    src[1023::1024] -= 1
    return dict(kind="l0", sensor="asar", n=n, blob=pk.reshape(-1), src=src * size,
                raw=torch.zeros(n, 2 + data, dtype=torch.uint8, device=DEV), **_l0_side(n))


def _l0_side(n):
    return dict(swst=torch.zeros(n, dtype=torch.int16, device=DEV), pri=torch.zeros(n, dtype=torch.int16, device=DEV),
                errors=torch.zeros(1, dtype=torch.int32, device=DEV))


def run(s):
    kind = s["kind"]
    if kind == "focus":
        s["plan"].focus(s["raw"], s["out"], s["swst"], s["min_swst"])
        if s["slc"] is None:
            return s["out"]
        s["plan"].slc_into(s["slc"])
        return s["out"], s["slc"]
    if kind == "host":
        s["plan"].focus_host_ptr(s["raw"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if kind == "batch":
        return s["batch"].focus(s["raws"], s["outs"])
    if kind == "strip":
        return s["strip"].focus(s["raw"], s["out"])
    if kind == "stages":
        return _run_stages(s)
    if kind == "l0":
        if s["sensor"] == "ers":
            l0.unpack(s["blob"], s["src"], s["n"], s["raw"], s["swst"], s["pri"], s["errors"])
        else:
            l0.asar_unpack(s["blob"], s["src"], s["n"], s["raw"].shape[1], s["raw"], s["swst"], s["pri"], s["errors"])
        return s["raw"], s["swst"], s["pri"], s["errors"]
    stages.condition_slc(s["slc"], s["cols"], s["ims"], calibration=0.5)
    stages.condition_detected(s["det"], s["imp"], calibration=0.25)
    return s["ims"], s["imp"]


def _run_stages(s):
    """The main flow over padded images: decode to SRGR (the image buffer starts out zeroed)."""
    sc, p = s["sc"], s["p"]
    s["image"].zero_()
    stages.convert_ers_samples(s["raw"], sc.samples_per_line, s["image"], sc.range_size)
    img = stages.DevicePaddedImage(s["image"], sc.range_size, sc.azimuth_size)
    iq = stages.raw_data_correction(img, sc.total_raw_samples)
    stages.zero_nans(img)
    dc = stages.calculate_doppler_centroid(img, p["prf"])
    stages.range_compression(img, s["chirp"], sc.chirp_samples)
    out = stages.range_doppler_algorithm(p["prf"], p["lam"], sc.range_spacing, p["near"], sc.az_bw_frac, p["vr"], dc,
                                         img, s["work"])
    first = sc.azimuth_size - s["rows"] if dc[2] > 0 else 0
    slc = out.data[first:first + s["rows"], 8:8 + s["nx"]].contiguous()
    stages.azimuth_multilook(slc, sc.azimuth_spacing, s["looks"])
    stages.range_spreading_loss_correction(s["looks"], s["near"], sc.range_spacing, 800000.0)
    stages.srgr_interpolation(s["looks"], s["poly"], sc.range_spacing, s["ground"])
    return dict(iq=iq, dc=dc, slc=slc, ground=s["ground"])


# ---------------------------------------------------------------------------- work

def _scene_work(nr, nc, na, raw_bytes, out_bytes):
    nk, npad = nr - nc, _smooth_above(na + 1)
    flops = 2 * na * 5.0 * nr * math.log2(nr) + 2 * nk * 5.0 * npad * math.log2(npad)  # the two transform pairs
    flops += na * nr * 12.0 + npad * nk * (16 * 4 + 12.0) + na * nk * 6.0  # correction, interpolation and filter, looks
    return dict(bytes=float(raw_bytes + out_bytes), flops=flops)


def work(case):
    kind = case["kind"]
    if kind == "records":
        r, c = case["rows"], case["cols"]
        d = max(1, r // 5)
        return dict(bytes=float(r * (8 * c + 17 + 4 * c) + d * (4 * c + 17 + 2 * c)), flops=float(r * c * 6 + d * c * 12))
    if kind == "l0":
        n = case["lines"]
        data = ERS_DATA if case["sensor"] == "ers" else 2 + case["samples"] + (case["samples"] + 62) // 63
        return dict(bytes=float(n * (2 * data + 24)), flops=0.0)
    if kind == "batch":
        parts = [work(dict(s, kind="focus", slc=False)) for _, s in _segments(case)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if kind == "strip":
        # each block works on its overlap too: that is the scheme's own cost, counted here as in the scheme
        nb = len(_strip_layout(case["lines"], case["block"], case["overlap"], 0)[0])
        one = work(dict(kind="focus", sensor="asar", range=case["range"], lines=min(case["block"], case["lines"]),
                        fmt="bytes", slc=False))
        return dict(bytes=one["bytes"] * case["lines"] / min(case["block"], case["lines"]), flops=one["flops"] * nb)
    p = SENSORS[case["sensor"]]
    nr, na, nc = case["range"], case["lines"], _chirp_samples(p)
    nx = nr - nc - 16
    raw = na * nr * 2 if case.get("fmt") != "fbaq4" else na * (2 + nr + (nr + 62) // 63)
    out = na / 5 * nx * 1.6 * 4  # ground-range pixels: about 1.6 per slant sample
    if case.get("slc") or kind == "stages":
        out += na * nx * 8
    return _scene_work(nr, nc, na, raw, out)


# ---------------------------------------------------------------------------- 64-bit restatement

def _round_away(v):
    return math.copysign(math.floor(abs(v) + 0.5), v)


def _aperture(sc, p):
    """Longest synthetic aperture over ten range positions, in lines."""
    nk = sc.range_size - sc.chirp_samples
    fc, best = SOL / p["lam"], 0
    for px in range(0, nk, nk // 10):
        v, r0 = sc.vr_poly_init[2], p["near"] + px * sc.range_spacing
        ka = 2 * fc * v * v / (SOL * r0)
        best = max(best, int(_round_away((p["prf"] * sc.az_bw_frac) / 2 / ka * p["prf"])))
    return best


def _f32(v):
    return v.to(torch.float32) if isinstance(v, torch.Tensor) else np.float32(v)


def _poly32(coeffs, x):
    """Float32 Horner with one rounding per multiply-add, x a float32 tensor."""
    r = torch.zeros_like(x)
    for e in coeffs:
        r = (r.double() * x.double() + float(np.float32(e))).float()
    return r


def _decode(c, raw, codes):
    """(I, Q, filled) as float64 [na][nr]."""
    na, nr = c["lines"], c["range"]
    if c["fmt"] == "fbaq4":
        nb = (nr + 62) // 63
        blk = torch.zeros(na, nb * 64, dtype=torch.uint8, device=DEV)
        blk[:, :raw.shape[1] - 2] = raw[:, 2:]
        blk = blk.view(na, nb, 64)
        lev = np.asarray(asarf.scene.fbaq.LEVELS)
        table = torch.as_tensor((lev[:, None] * _fbaq_scale(np.arange(256))[None, :]).astype(np.float32).reshape(-1),
                                device=DEV).double()
        ids = blk[:, :, :1].long()

        def val(code):
            code = code.long()
            return table[256 * torch.where(code > 7, 15 - code, 8 + code) + ids].view(na, -1)[:, :nr]
        i, q = val(blk[:, :, 1:] >> 4), val(blk[:, :, 1:] & 15)
        return i, q, torch.ones(na, nr, dtype=torch.bool, device=DEV)
    v = raw.view(na, -1, 2).double()
    if codes is None:
        return v[..., 0].contiguous(), v[..., 1].contiguous(), torch.ones(na, nr, dtype=torch.bool, device=DEV)
    off = torch.as_tensor(4 * (codes.astype(np.int64) - codes.min()), device=DEV)
    i = torch.arange(nr, device=DEV)[None, :] - off[:, None]
    ok = (i >= 0) & (i < v.shape[1])
    i = i.clamp(0, v.shape[1] - 1)
    return torch.gather(v[..., 0], 1, i) * ok, torch.gather(v[..., 1], 1, i) * ok, ok


def _corrected(sc, i, q, ok):
    """I/Q correction constants, the corrected image (complex128, zero where nothing was
    recorded) and the Doppler polynomial."""
    na, nr = i.shape
    n = float(ok.sum())
    npad = (asarf.fft_size_above(nr + sc.chirp_samples) - nr) * na
    total = np.float32(n)
    si, sq = float(i.sum()), float(q.sum())
    dci, dcq = float(np.float32(si) / total), float(np.float32(sq) / total)
    ci, cq = (i - dci) * ok, (q - dcq) * ok
    cii, cqq, ciq = float((ci * ci).sum()), float((cq * cq).sum()), float((ci * cq).sum())
    # the zero range padding takes part in the gain and phase sums as 0 - mean
    ii, qq, iq = cii + npad * dci * dci, cqq + npad * dcq * dcq, ciq + npad * dci * dcq
    gain = math.sqrt(ii / qq)
    gf = float(np.float32(gain))
    delta = (iq / gf) / (ii / (gf * gf))
    s, co = float(np.float32(delta)), float(np.float32(1.0 - delta * delta))
    re = ci / gf
    z = torch.complex(re, (cq - re * s) / co * ok)
    pad = complex(-dci / gf, (-dcq + dci / gf * s) / co)
    res = dict(dc_i=dci, dc_q=dcq, iq_gain=gain, phase_error=math.degrees(math.asin(delta)),
               stddev_i=math.sqrt(cii / n), stddev_q=math.sqrt(cqq / n))
    step = nr // 32
    acc = (z[:-1].conj() * z[1:]).sum(0).cpu().numpy()
    xs, hz = [], []
    for xb in range(0, nr, step):
        a = acc[xb:xb + step].sum() + max(0, xb + step - nr) * abs(pad) ** 2 * (na - 1)
        xs.append((xb + xb + step) // 2)
        hz.append(sc.prf * math.atan2(a.imag, a.real) / (2 * math.pi))
    v = np.vander(np.array(xs, dtype=np.float64), 3)
    qm, rm = np.linalg.qr(v[:, ::-1])
    dc = np.linalg.solve(rm, qm.T @ np.array(hz))[::-1]
    return res, z, [float(e) for e in dc]


def _compressed(sc, p, z):
    nr, nc = z.shape[1], sc.chirp_samples
    c = _chirp64(p)
    c = c * (0.54 - 0.46 * torch.cos(2 * math.pi * torch.arange(nc, device=DEV, dtype=torch.float64) / nc))
    c = c / torch.sqrt((c.abs() ** 2).sum())
    n = _smooth_above(nr)
    h = torch.fft.fft(c, n=n).conj()
    out = torch.empty(z.shape[0], nr - nc, dtype=torch.complex128, device=DEV)
    for r0 in range(0, z.shape[0], 4096):
        out[r0:r0 + 4096] = torch.fft.ifft(torch.fft.fft(z[r0:r0 + 4096], n=n, dim=1) * h, dim=1)[:, :nr - nc]
    return out


def _focused(sc, p, rc, dc_poly, abs_phase):
    """Azimuth processing: all lines of the complex image [na][nk] in complex128."""
    na, nk = rc.shape
    n = _smooth_above(na + 1)
    spec = torch.fft.fft(rc, n=n, dim=0)
    x = torch.arange(nk, device=DEV)
    xf = x.float()
    prf, lam = np.float32(p["prf"]), np.float32(p["lam"])
    step, half = np.float32(prf / np.float32(n)), np.float32(prf * np.float32(0.5))
    dc, vr = _poly32(dc_poly, xf), _poly32(p["vr"], xf)
    t = (dc.double() / float(step)).float().double()  # divided in 64 bits: torch multiplies by a scalar's reciprocal
    t = torch.sign(t) * torch.floor(t.abs() + 0.5)
    dc_off = t.float() * float(step)
    r0 = p["near"] + x.double() * sc.range_spacing
    ka = ((2.0 * vr) * vr).double().div(float(lam) * r0).float()
    frac = float(np.float32(sc.az_bw_frac))
    cut_hi = (float(half) * frac + dc_off.double()).float()
    cut_lo = (-float(half) * frac + dc_off.double()).float()
    hi, lo = float(half) + dc, -float(half) + dc
    den = (8.0 * vr) * vr
    dc_ka = dc_off / ka
    win = np.array([0.42 - 0.5 * math.cos(2 * math.pi * k / 15) + 0.08 * math.cos(4 * math.pi * k / 15) for k in range(16)])
    win = [float(np.float32(w)) for w in win]
    pi32 = float(np.float32(math.pi))
    two_pi32 = float(np.float32(2.0) * np.float32(math.pi))
    ph0 = torch.zeros(nk, dtype=torch.float64, device=DEV)
    if abs_phase:
        ph0 = torch.fmod(4 * math.pi * r0 / p["lam"], 2 * math.pi) + \
            torch.fmod(math.pi * dc_off.double() ** 2 / ka.double(), 2 * math.pi)
    wide = torch.nn.functional.pad
    rows = 1024
    for y0 in range(0, n, rows):
        k = torch.arange(y0, min(n, y0 + rows), device=DEV)
        bf = torch.where(k < n // 2, k, k - n).float() * float(step)
        bf = bf[:, None]
        fn = torch.where((dc < 0) & (bf > hi), bf - float(prf), torch.where((dc > 0) & (bf < lo), bf + float(prf), bf + 0 * dc))
        keep = ~((fn < cut_lo) | (fn > cut_hi))
        num = (float(lam * lam) * fn) * fn
        shift = ((num / den).double() * r0 / sc.range_spacing).float()
        walk = torch.floor(shift.double() + 0.5).long()
        inside = (x + walk - 8 >= 0) & (x + walk + 8 < nk)
        off = (shift - walk.float()) + 8.0
        src = wide(spec[y0:y0 + rows], (8, 32))
        acc = torch.zeros(bf.shape[0], nk, dtype=torch.complex128, device=DEV)
        norm = torch.zeros(bf.shape[0], nk, dtype=torch.float64, device=DEV)
        base = (x + walk).clamp(0, nk + 15)
        for i in range(1, 15):
            w = win[i] * torch.special.sinc(off.double() - i)
            acc += torch.gather(src, 1, base + i) * w
            norm += w
        v = torch.where(inside & keep, acc / norm, torch.zeros_like(acc))
        fc = bf - dc_off
        fc = torch.where(fc > float(half), fc - float(prf), torch.where(fc < -float(half), fc + float(prf), fc))
        mf = (pi32 * fc) * fc / ka
        sh = (two_pi32 * dc_ka) * bf
        ph = ph0 - mf.double() - sh.double()
        spec[y0:y0 + rows] = v * torch.polar(torch.ones_like(ph), ph)
    return torch.fft.ifft(spec, dim=0)[:na]


def _detected(sc, p, slc, t0_us):
    """Multilook, range spreading loss and ground range of a complex128 image window."""
    rows, nx = slc.shape
    ratio = np.float32(12.5 / sc.azimuth_spacing)
    n = int(_round_away(float(np.float32(rows) / ratio)))
    power = slc.real ** 2 + slc.imag ** 2
    del slc
    idx = (np.arange(n).astype(np.float32) * ratio).astype(np.float32)
    mu = idx - np.trunc(idx)

    def box(a, b):
        s = np.maximum(np.trunc(idx + np.float32(a)).astype(np.int64), 0)
        e = np.minimum(np.trunc(idx + np.float32(b)).astype(np.int64), rows)
        tot = torch.zeros(n, nx, dtype=torch.float64, device=DEV)
        for k in range(8):  # at most six rows a window
            r = torch.as_tensor(np.minimum(s + k, rows - 1), device=DEV)
            tot += power[r] * torch.as_tensor((s + k < e).astype(np.float64), device=DEV)[:, None]
        cnt = np.maximum(e - s, 0)
        return tot / torch.as_tensor(np.maximum(cnt, 1).astype(np.float64), device=DEV)[:, None], cnt

    a, ca = box(-2, 2)
    b, cb = box(-1, 3)
    ml = a + (b - a) * torch.as_tensor(mu.astype(np.float64), device=DEV)[:, None]
    ml = ml * torch.as_tensor(((ca > 0) & (cb > 0)).astype(np.float64), device=DEV)[:, None]
    near = p["near"] + 8 * sc.range_spacing
    r = near + torch.arange(nx, device=DEV, dtype=torch.float64) * sc.range_spacing
    ml = ml * (r / 800000.0) ** 1.5
    poly, ng = _ground_poly(sc, p, near, nx, n, float(ratio), t0_us)
    xg = torch.arange(ng, device=DEV).float() * 12.5
    pos = (_poly32(poly, xg).double() / float(np.float32(sc.range_spacing))).float()
    i0 = pos.to(torch.int64)
    fr = (pos - i0.float()).double()
    return ml[:, i0] + fr * (ml[:, i0 + 1] - ml[:, i0])


def _ground_poly(sc, p, near, nx, n, ratio, t0_us):
    pos, vel = _interp_orbit(sc.osv, t0_us + (int((1.0 / p["prf"]) * ratio * (n // 2) * 1e6) & 0xFFFFFFFF))
    first = _geolocate(vel, pos, sc.center_point, near)
    gd, sr = [], []
    for i in range(100):
        r = near + (i * (nx // 100)) * sc.range_spacing
        gd.append(float(np.linalg.norm(_geolocate(vel, pos, sc.center_point, r) - first)))
        sr.append(r - near)
    gd = np.array(gd)
    s = gd[-1]
    c = np.linalg.lstsq(np.vander(gd / s, 5), np.array(sr), rcond=None)[0]
    return [float(c[k] / s ** (4 - k)) for k in range(5)], int(s / 12.5)


def _window(sc, p, dc_poly):
    ap = _aperture(sc, p)
    return (ap, sc.azimuth_size) if dc_poly[2] > 0 else (0, sc.azimuth_size - ap)


def _exact_scene(c, seed, abs_phase=False, full=False):
    sc, raw, codes = _raw(c, seed)
    p = SENSORS[c["sensor"]]
    res, z, dc = _corrected(sc, *_decode(c, raw, codes))
    img = _focused(sc, p, _compressed(sc, p, z), dc, abs_phase)
    lo, hi = _window(sc, p, dc)
    slc = img[lo:hi, 8:8 + img.shape[1] - 16]
    det = _detected(sc, p, slc, T0_US)
    return (res, dc, slc, det) if full else (slc, det)


def _strip_layout(na, block, overlap, ap):
    b = min(block, na)
    nb = 1 if na <= b else 1 + (na - b + (b - overlap) - 1) // (b - overlap)
    start = [min(k * (b - overlap), na - b) for k in range(nb)]
    lo = [ap if k == 0 else (start[k - 1] + b + s) // 2 - s for k, s in enumerate(start)]
    hi = [b - ap if k == nb - 1 else (s + b + start[k + 1]) // 2 - s for k, s in enumerate(start)]
    return start, lo, hi


def _exact_strip(c, seed):
    p = SENSORS["asar"]
    sc = _scene("asar", c["range"], c["lines"])
    iv, qv = _iq("asar", c["range"], c["lines"], seed, drift=100.0)
    raw = _encode_bytes(iv, qv, sc.bits)
    del iv, qv
    ap = _aperture(sc, p)
    start, lo, hi = _strip_layout(c["lines"], c["block"], c["overlap"], ap)
    b = min(c["block"], c["lines"])
    parts = []
    for s, a, e in zip(start, lo, hi):
        one = dict(range=c["range"], lines=b, fmt="bytes")
        _, z, dc = _corrected(sc, *_decode(one, raw[s:s + b], None))
        img = _focused(sc, p, _compressed(sc, p, z), dc, False)
        parts.append(img[a:e, 8:img.shape[1] - 8].clone())
    slc = torch.cat(parts)
    return _detected(sc, p, slc, T0_US + int(_round_away(ap * (1.0 / p["prf"]) * 1e6)))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("l0", "records"):
        return None  # bytes: moved or quantised, held to equality
    if kind == "batch":
        return [_exact_scene(s, seed * 17 + k)[1] for k, s in _segments(case)]
    if kind == "strip":
        return _exact_strip(case, seed)
    if kind == "stages":
        res, dc, slc, det = _exact_scene(dict(case, fmt="bytes", swst=False), seed, full=True)
        return dict(iq=res, dc=dc, slc=slc, ground=det)
    slc, det = _exact_scene(case, seed, case.get("abs_phase", False))
    return (det, slc) if case.get("slc") else det
