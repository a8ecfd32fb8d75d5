// Per-stage entry points: the reference's sar/ functions one by one, on its padded complex
// image layout (complex float [y_stride][x_stride], data block [0, y_size) x [0, x_size)
// top-left, cuda_util/device_padded_image.cuh:13-27).  Like the reference's functions they
// allocate what they need, copy results to the host where the reference does, and
// synchronise the stream before returning.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "asarf.h"
#include "backend.h"
#include "bodies.cuh"
#include "internal.h"

using namespace asarf;

namespace {

// A call's device arrays in one allocation (scratch_alloc) on its stream.
struct Scratch {
    void* stream;
    std::vector<size_t> at;
    size_t bytes = 0;
    void* p = nullptr;
    bool pooled = false;
    explicit Scratch(void* s) : stream(s) {}
    ~Scratch() { scratch_free(p, stream, pooled); }
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    int add(size_t n) {
        at.push_back(bytes);
        bytes += (n + 255) / 256 * 256;
        return static_cast<int>(at.size()) - 1;
    }
    bool alloc() { return (p = scratch_alloc(bytes, stream, &pooled)) != nullptr; }
    template <class T>
    T* as(int k) const {
        return reinterpret_cast<T*>(static_cast<unsigned char*>(p) + at[static_cast<size_t>(k)]);
    }
};

int nomem() { return set_error(ASARF_ERR_NOMEM, "device allocation failed"); }

// NaN-aware moments of the data block and of the padding columns, summed on the host in a
// fixed order; about (optional): the value the data block's sums are taken about.
int image_moments(const float2* img, int x_size, int y_size, int x_stride, const double* about, double out[12],
                  void* stream) {
    const int rpb = 8;
    const int blocks = (y_size + rpb - 1) / rpb;
    Scratch part(stream);
    part.add(sizeof(double) * 12 * static_cast<size_t>(blocks));
    if (!part.alloc()) return nomem();
    ImgMomentsArgs a{};
    a.img = img;
    a.x_size = x_size;
    a.y_size = y_size;
    a.x_stride = x_stride;
    a.rows_per_block = rpb;
    if (about) a.about = 1, a.about_i = about[0], a.about_q = about[1];
    a.partial = part.as<double>(0);
    int rc = backend_img_moments(a, blocks, stream);
    if (rc) return rc;
    std::vector<double> h(12 * static_cast<size_t>(blocks));
    rc = mem_d2h(h.data(), part.p, sizeof(double) * h.size(), stream);
    if (rc) return rc;
    rc = stream_sync(stream);
    if (rc) return rc;
    for (int k = 0; k < 12; ++k) out[k] = 0.0;
    for (int b = 0; b < blocks; ++b)
        for (int k = 0; k < 12; ++k) out[k] += h[static_cast<size_t>(b) * 12 + k];
    return ASARF_OK;
}

}  // namespace

extern "C" {

int asarf_convert_ers_samples(const uint8_t* d_raw, int32_t raw_line_bytes, int32_t samples_per_line, int32_t lines,
                              const uint16_t* d_swst, int32_t min_swst, void* d_img, int64_t img_stride,
                              int32_t range_size, void* stream) {
    if (!d_raw || !d_img || lines <= 0 || samples_per_line <= 0 || range_size < samples_per_line ||
        img_stride < range_size || raw_line_bytes < 2 * samples_per_line || (raw_line_bytes & 1))
        return set_error(ASARF_ERR_INVALID, "convert_ers_samples: bad arguments");
    DecodeArgs a{};
    a.raw = d_raw;
    a.line_bytes = raw_line_bytes;
    a.spl = samples_per_line;
    a.lines = lines;
    a.nr = range_size;
    a.swst = d_swst;
    a.min_swst = min_swst;
    a.img = static_cast<float2*>(d_img);
    a.stride = img_stride;
    int rc = backend_decode(a, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int asarf_convert_asar_blocks(const uint8_t* d_raw, int32_t record_bytes, int32_t records, const uint16_t* d_swst,
                              int32_t min_swst, const float* d_lut_i, const float* d_lut_q, void* d_img,
                              int64_t img_stride, int32_t range_size, void* stream) {
    if (!d_raw || !d_img || !d_lut_i || !d_lut_q || records <= 0 || record_bytes < 2 || range_size <= 0 ||
        img_stride < range_size)
        return set_error(ASARF_ERR_INVALID, "convert_asar_blocks: bad arguments");
    DecodeFbaqArgs a{};
    a.raw = d_raw;
    a.line_bytes = record_bytes;
    a.lines = records;
    a.nr = range_size;
    a.swst = d_swst;
    a.min_swst = min_swst;
    a.lut_i = d_lut_i;
    a.lut_q = d_lut_q;
    a.img = static_cast<float2*>(d_img);
    a.stride = img_stride;
    int rc = backend_decode_fbaq(a, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int32_t asarf_fbaq4_index(int32_t block, int32_t code) { return fbaq4_index(block, code); }

int asarf_condition_slc(const void* d_img, int32_t x_size, int32_t y_size, int32_t x_stride,
                        int32_t record_header_bytes, float calibration, void* d_dest, void* stream) {
    if (!d_img || !d_dest || x_size <= 0 || y_size <= 0 || x_stride < x_size || record_header_bytes < 0)
        return set_error(ASARF_ERR_INVALID, "condition_slc: bad arguments");
    ConditionArgs c{};
    c.product = 2;
    c.slc = static_cast<const float2*>(d_img);
    c.stride = x_stride;
    c.x_size = x_size;
    c.y_size = y_size;
    c.hdr = record_header_bytes;
    c.cal = calibration;
    c.dest = static_cast<uint8_t*>(d_dest);
    int rc = backend_condition(c, y_size, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int asarf_condition_detected(const float* d_img, int32_t range_size, int32_t azimuth_size,
                             int32_t record_header_bytes, float calibration, void* d_dest, void* stream) {
    if (!d_img || !d_dest || range_size <= 0 || azimuth_size <= 0 || record_header_bytes < 0)
        return set_error(ASARF_ERR_INVALID, "condition_detected: bad arguments");
    ConditionArgs c{};
    c.product = 1;
    c.img = d_img;
    c.stride = range_size;
    c.x_size = range_size;
    c.y_size = azimuth_size;
    c.hdr = record_header_bytes;
    c.cal = calibration;
    c.dest = static_cast<uint8_t*>(d_dest);
    int rc = backend_condition(c, azimuth_size, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int asarf_raw_data_correction(void* d_img, int32_t x_size, int32_t y_size, int32_t x_stride, int32_t y_stride,
                              int64_t n_total_samples, asarf_iq_results* results, void* stream) {
    if (!d_img || !results || x_size <= 0 || y_size <= 0 || x_stride < x_size || y_stride < y_size)
        return set_error(ASARF_ERR_INVALID, "raw_data_correction: bad arguments");
    float2* img = static_cast<float2*>(d_img);
    double m[12];
    int rc = image_moments(img, x_size, y_size, x_stride, nullptr, m, stream);
    if (rc) return rc;
    const double total = n_total_samples > 0 ? static_cast<double>(n_total_samples) : static_cast<double>(x_size) * y_size;
    const float totf = static_cast<float>(total);
    // CalcMean: float(double sum) / float(total)
    const float dc_i = static_cast<float>(m[1]) / totf;
    const float dc_q = static_cast<float>(m[2]) / totf;
    // sums over x < XStride after the DC step, both regions (closed forms of the FP64 moments)
    const double di = dc_i, dq = dc_q;
    auto sq = [&](int o, int s1, int s2, double d) { return m[o + s2] - 2.0 * d * m[o + s1] + m[o] * d * d; };
    auto cross = [&](int o) { return m[o + 5] - dq * m[o + 1] - di * m[o + 2] + m[o] * di * dq; };
    double cii = sq(0, 1, 3, di), cqq = sq(0, 2, 4, dq), ciq = cross(0);
    // The closed form loses S2 / c of the FP64 sums' digits: where a channel's spread is that small beside its level
    // (a dead channel; never a raw signal), the sums are taken again about the mean itself.
    constexpr double kCancels = 1e-4;
    if (cii <= kCancels * m[3] || cqq <= kCancels * m[4]) {
        const double about[2] = {di, dq};
        double c[12];
        rc = image_moments(img, x_size, y_size, x_stride, about, c, stream);
        if (rc) return rc;
        cii = c[3], cqq = c[4], ciq = c[5];
    }
    const float std_i = std::sqrt(static_cast<float>(cii) / totf);
    const float std_q = std::sqrt(static_cast<float>(cqq) / totf);
    const double i1sq = cii + sq(6, 1, 3, di);
    const double q1sq = cqq + sq(6, 2, 4, dq);
    const double i1q1 = ciq + cross(6);
    const double gain = std::sqrt(i1sq / q1sq);
    const float gf = static_cast<float>(gain);
    const double delta = (i1q1 / gf) / (i1sq / (static_cast<double>(gf) * gf));
    IqApplyArgs ap{};
    ap.img = img;
    ap.x_stride = x_stride;
    ap.y_size = y_size;
    ap.dc_i = dc_i;
    ap.dc_q = dc_q;
    ap.gain = gf;
    ap.sin_c = static_cast<float>(delta);
    ap.cos_c = static_cast<float>(1.0 - delta * delta);
    rc = backend_iq_apply(ap, static_cast<long long>(y_size) * x_stride, stream);
    if (rc) return rc;
    results->dc_i = dc_i;
    results->dc_q = dc_q;
    results->iq_gain = gain;
    results->phase_error = 360.0 * std::asin(delta) / (2.0 * 3.14159265358979323846);
    results->stddev_i = std_i;
    results->stddev_q = std_q;
    return stream_sync(stream);
}

int asarf_zero_nans(void* d_img, int32_t x_stride, int32_t y_stride, void* stream) {
    if (!d_img || x_stride <= 0 || y_stride <= 0) return set_error(ASARF_ERR_INVALID, "zero_nans: bad arguments");
    int rc = backend_zero_nans(static_cast<float2*>(d_img), static_cast<long long>(x_stride) * y_stride, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int asarf_doppler_centroid(const void* d_img, int32_t x_size, int32_t y_size, int32_t x_stride, double prf,
                           double poly[3], void* stream) {
    if (!d_img || !poly || x_size < 32 || y_size < 2 || x_stride < x_size)
        return set_error(ASARF_ERR_INVALID, "doppler_centroid: bad arguments");
    AcccArgs a{};
    a.img = static_cast<const float2*>(d_img);
    a.x_size = x_size;
    a.y_size = y_size;
    a.x_stride = x_stride;
    a.step = x_size / 32;
    a.nblk = (x_size + a.step - 1) / a.step;
    a.rows_per_block = std::max(256, (y_size + kMaxGridY - 1) / kMaxGridY);
    a.xend = std::min(a.nblk * a.step, x_stride);
    a.span = (kAcccCols - 1) / a.step + 2;
    const int gx = (a.xend + kAcccCols - 1) / kAcccCols, gy = (y_size + a.rows_per_block - 1) / a.rows_per_block;
    const size_t count = 2 * static_cast<size_t>(a.span) * gx * gy;
    Scratch part(stream);
    part.add(sizeof(double) * count);
    if (!part.alloc()) return nomem();
    a.partial = part.as<double>(0);
    int rc = backend_accc(a, gx, gy, stream);
    if (rc) return rc;
    std::vector<double> h(count);
    rc = mem_d2h(h.data(), part.p, sizeof(double) * count, stream);
    if (rc) return rc;
    rc = stream_sync(stream);
    if (rc) return rc;
    std::vector<double> re(a.nblk, 0.0), im(a.nblk, 0.0), xs(a.nblk), ys(a.nblk);
    for (int by = 0; by < gy; ++by)
        for (int bx = 0; bx < gx; ++bx)
            for (int k = 0; k < a.span; ++k) {
                const int b = bx * kAcccCols / a.step + k;
                if (b >= a.nblk) break;
                const double* v = &h[2 * (static_cast<size_t>(a.span) * (static_cast<size_t>(by) * gx + bx) + k)];
                re[b] += v[0];
                im[b] += v[1];
            }
    for (int k = 0; k < a.nblk; ++k) {
        ys[k] = prf * (std::atan2(im[k], re[k]) / (2.0 * 3.14159265358979323846));
        xs[k] = static_cast<double>((k * a.step + (k + 1) * a.step) / 2);
    }
    if (a.nblk > kMaxDcBlocks || !polyfit_qr<kMaxDcBlocks, 3>(xs.data(), ys.data(), a.nblk, 2, poly))
        return set_error(ASARF_ERR_NUMERIC, "doppler_centroid: fit failed");
    return ASARF_OK;
}

int asarf_range_compression(void* d_img, int32_t x_size, int32_t y_size, int32_t x_stride, const float* chirp_padded,
                            int32_t chirp_len, int32_t chirp_samples, int32_t* new_x_size, void* stream) {
    if (!d_img || !chirp_padded || x_size <= 0 || y_size <= 0 || chirp_samples <= 0 || chirp_samples >= x_size)
        return set_error(ASARF_ERR_INVALID, "range_compression: bad arguments");
    if (chirp_len != x_stride) return set_error(ASARF_ERR_INVALID, "Range padding and chirp size mismatch");
    HostFft fft;
    const int L = choose_rc_len(x_size);
    int ct[3];
    const int n_ct = L >= x_size ? ct_radices(L, ct) : 0;
    if (L < x_size || !(n_ct ? build_fft_radices(L, std::vector<int>(ct, ct + n_ct), fft, false) : build_fft(L, fft)))
        return set_error(ASARF_ERR_INVALID, "range_compression: no FFT length");
    const LaunchShape sh{512, sizeof(float2) * static_cast<size_t>(n_ct ? ct_smem_elems_of(L) : L)};
    if (sh.smem > smem_optin_limit())
        return set_error(ASARF_ERR_INVALID, "range_compression: range FFT of %d samples exceeds shared memory", L);
    TwiddleArgs tw = n_ct ? ct_twiddle_args(L, nullptr) : TwiddleArgs{nullptr, L, {0, 0, 0}};
    Scratch m(stream);
    const int k_chirp = m.add(sizeof(float2) * chirp_samples), k_mf = m.add(sizeof(float2) * L),
              k_tw = m.add(sizeof(float2) * twiddle_count(tw));
    if (!m.alloc()) return nomem();
    tw.out = m.as<float2>(k_tw);
    int rc = mem_h2d(m.as<float2>(k_chirp), chirp_padded, sizeof(float2) * chirp_samples, stream);
    if (!rc) rc = backend_matched_filter(matched_filter_args(m.as<float2>(k_chirp), chirp_samples, fft, m.as<float2>(k_mf)),
                                         stream);
    if (!rc) rc = backend_twiddles(tw, stream);
    if (rc) return rc;
    RcRowsArgs a{};
    a.img = static_cast<float2*>(d_img);
    a.stride = x_stride;
    a.nr = x_size;
    a.nk = x_size - chirp_samples;
    a.x_zero_end = x_stride;
    a.plan = fft.plan;
    a.plan.tw = n_ct ? nullptr : tw.out;
    a.ctw = n_ct ? tw.out : nullptr;
    a.mf = m.as<float2>(k_mf);
    rc = backend_rc_rows(a, y_size, sh, stream);
    if (rc) return rc;
    if (new_x_size) *new_x_size = a.nk;
    return stream_sync(stream);
}

int asarf_range_doppler(const asarf_rda_params* prm, void* d_src, void* d_out, int32_t x_size, int32_t y_size,
                        int32_t x_stride, int32_t y_stride, void* stream) {
    if (!prm || !d_src || !d_out || x_size < 17 || y_size <= 1 || x_stride < x_size || y_stride < y_size)
        return set_error(ASARF_ERR_INVALID, "range_doppler: bad arguments");
    const int N = y_stride;
    // RCMC halo from the largest walk at |f| <= PRF
    double vr_min = 1e30;
    for (int x = 0; x < x_size; x += std::max(1, x_size / 64)) {
        const double v = (prm->vr_poly[0] * x + prm->vr_poly[1]) * x + prm->vr_poly[2];
        vr_min = std::min(vr_min, std::fabs(v));
    }
    const double rmax = prm->slant_range_first + x_size * prm->range_spacing;
    const double walk =
        prm->wavelength * prm->wavelength * prm->prf * prm->prf * rmax / (8 * vr_min * vr_min) / prm->range_spacing;
    const int hl = kRcmcTaps / 2;
    int hr = rcmc_right_halo(walk);
    if ((hl + hr) & 1) ++hr;  // column-pair transforms need an even tile width
    const int n2 = choose_az_n2(N, x_size, hl, hr, false);
    const int n1 = N / n2;
    HostFft f1, f2;
    if (n2 < 2 || !build_fft_radices(n1, strided_radices(n1), f1) || !build_fft_radices(n2, block_radices(n2), f2))
        return set_error(ASARF_ERR_INVALID, "range_doppler: azimuth size %d is not 2^a3^b5^c7^d", N);
    // tables + a finalised state carrying the Doppler polynomial
    Scratch m(stream);
    const int k_tw1 = m.add(sizeof(float2) * n1), k_dr1 = m.add(sizeof(int) * n1), k_tw2 = m.add(sizeof(float2) * n2),
              k_dr2 = m.add(sizeof(int) * n2), k_twn = m.add(sizeof(float2) * N), k_st = m.add(sizeof(FocusState)),
              k_rcmc = m.add(sizeof(float) * static_cast<size_t>(kRcmcNodes + 1) * kRcmcRowFloats);
    if (!m.alloc()) return nomem();
    float2* tw1 = m.as<float2>(k_tw1);
    int* dr1 = m.as<int>(k_dr1);
    float2* tw2 = m.as<float2>(k_tw2);
    int* dr2 = m.as<int>(k_dr2);
    float2* twN = m.as<float2>(k_twn);
    float* rcmc = m.as<float>(k_rcmc);
    FocusState hs{};
    for (int k = 0; k < 3; ++k) {
        hs.dc_poly[k] = prm->dc_poly[k];
        hs.dc_poly32[k] = static_cast<float>(prm->dc_poly[k]);
    }
    hs.first_line = 0;
    hs.n_lines = y_size;  // inverse pass stores the data rows only
    FocusState* dstate = m.as<FocusState>(k_st);
    int rc = mem_h2d(tw1, f1.tw.data(), sizeof(float2) * n1, stream);
    if (!rc) rc = mem_h2d(dr1, f1.drev.data(), sizeof(int) * n1, stream);
    if (!rc) rc = mem_h2d(tw2, f2.tw.data(), sizeof(float2) * n2, stream);
    if (!rc) rc = mem_h2d(dr2, f2.drev.data(), sizeof(int) * n2, stream);
    if (!rc) rc = mem_h2d(dstate, &hs, sizeof(hs), stream);
    if (!rc) rc = backend_twiddles(TwiddleArgs{twN, N, {0, 0, 0}}, stream);
    if (!rc) rc = backend_rcmc_table(rcmc, stream);
    if (rc) return rc;
    f1.plan.tw = tw1;
    f2.plan.tw = tw2;
    float2* src = static_cast<float2*>(d_src);
    float2* out = static_cast<float2*>(d_out);
    const int xt1 = (n1 * 32 * 8 <= 160 * 1024) ? 32 : 16;
    AzStridedArgs fwd{};
    fwd.in = src;
    fwd.out = src;
    fwd.pitch = x_stride;
    fwd.n1 = n1;
    fwd.n2 = n2;
    fwd.plan1 = f1.plan;
    fwd.drev1 = dr1;
    fwd.twn = twN;
    fwd.nk = x_size;
    fwd.xt = xt1;
    fwd.valid_rows = N;  // the reference transforms every row of the padded image
    fwd.state = dstate;
    fwd.scale = 1.0f;
    AzStridedArgs inv = fwd;
    inv.in = out;
    inv.out = out;
    inv.valid_rows = N;
    inv.scale = azimuth_scale(N, 2.0 * (transform_gain(f1, false) + transform_gain(f2, false)));
    inv.inverse = 1;
    AzRdArgs d{};
    d.in = src;
    d.out = out;
    d.pitch = x_stride;
    d.n1 = n1;
    d.n2 = n2;
    d.az_pad = N;
    d.plan2 = f2.plan;
    d.drev2 = dr2;
    d.nk = x_size;
    d.hl = hl;
    d.hr = hr;
    d.xt = az_rd_tile_width(n2, d.hl, d.hr, false, smem_optin_limit());
    d.wt = d.xt + d.hl + d.hr;
    d.prf = static_cast<float>(prm->prf);
    d.bin_step = d.prf / static_cast<float>(N);
    d.half_prf = d.prf * 0.5f;
    d.lambda = static_cast<float>(prm->wavelength);
    d.frac = static_cast<float>(prm->az_bw_frac);
    d.slant = prm->slant_range_first;
    d.range_spacing = prm->range_spacing;
    for (int k = 0; k < 3; ++k) d.vr_poly[k] = static_cast<float>(prm->vr_poly[k]);
    d.state = dstate;
    d.rcmc = rcmc;
    const int tiles1 = (x_size + xt1 - 1) / xt1, tiles2 = (x_size + d.xt - 1) / d.xt;
    fwd.nb = inv.nb = xt1 == 32 ? az_strided_tiles_per_block(n1, n2, tiles1) : 1;
    const LaunchShape sh_st{256, az_strided_smem(n1, xt1, fwd.nb)};
    const LaunchShape sh_rd{512, az_rd_smem(n2, d.wt, d.xt, false)};
    if (sh_st.smem > smem_optin_limit() || sh_rd.smem > smem_optin_limit())
        return set_error(ASARF_ERR_INVALID, "range_doppler: tiles exceed shared memory (n1 %d, n2 %d)", n1, n2);
    // tiles by TMA where the caller's rows are 16-byte aligned, as the planned path's always are
    alignas(64) unsigned char map_src3[128], map_out3[128], map_src2[128];
    bool tma = x_stride % 2 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0 &&
               (reinterpret_cast<uintptr_t>(out) & 15) == 0 && 2 * d.wt <= 256;
    d.n2_box = rd_box_rows(n2, d.wt);
    tma = tma && d.n2_box > 0;
    if (tma) {
        fwd.n1_box = inv.n1_box = largest_divisor_le(n1, 256);
        tma = make_azimuth_maps(src, out, x_size, x_stride, n1, n2, xt1, fwd.nb, fwd.n1_box, d.wt, d.n2_box, map_src3,
                                map_out3, map_src2);
    }
    fwd.use_tma = inv.use_tma = d.use_tma = tma ? 1 : 0;
    fwd.compiled = inv.compiled = d.compiled = 1;
    rc = backend_az_strided(fwd, tma ? map_src3 : nullptr, tiles1, sh_st, stream);
    if (!rc) rc = backend_az_rd(d, tma ? map_src2 : nullptr, tiles2, n1, sh_rd, &dstate->errors, stream);
    if (!rc) rc = backend_az_strided(inv, tma ? map_out3 : nullptr, tiles1, sh_st, stream);
    // everything outside the data block is zero: columns past it, and the rows past it, which still
    // hold the spectrum stage's values
    if (!rc) rc = mem_zero_2d(out + x_size, sizeof(float2) * x_stride, sizeof(float2) * (x_stride - x_size), y_size, stream);
    if (!rc && y_size < N)
        rc = mem_zero(out + static_cast<size_t>(y_size) * x_stride,
                      sizeof(float2) * static_cast<size_t>(N - y_size) * x_stride, stream);
    if (rc) return rc;
    unsigned int err = 0;
    rc = mem_d2h(&err, &dstate->errors, sizeof(err), stream);
    if (!rc) rc = stream_sync(stream);
    if (rc) return rc;
    if (err) return set_error(ASARF_ERR_NUMERIC, "range_doppler: kernel error flags %#x", err);
    return ASARF_OK;
}

int asarf_azimuth_multilook(const void* d_slc, int32_t x_size, int32_t y_size, double azimuth_spacing, float* d_out,
                            int32_t* out_y, void* stream) {
    if (!d_slc || !d_out || x_size <= 0 || y_size <= 0 || !(azimuth_spacing > 0))
        return set_error(ASARF_ERR_INVALID, "azimuth_multilook: bad arguments");
    MultilookArgs a{};
    a.slc = static_cast<const float2*>(d_slc);
    a.x_size = x_size;
    a.in_y = y_size;
    a.ratio = static_cast<float>(12.5f / azimuth_spacing);
    a.out_y = static_cast<int>(std::round(static_cast<float>(y_size) / a.ratio));
    a.out = d_out;
    if (a.out_y <= 0) return set_error(ASARF_ERR_INVALID, "azimuth_multilook: no output lines");
    if (out_y) *out_y = a.out_y;
    int rc = backend_multilook(a, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int asarf_range_spreading_loss(float* d_img, int32_t range_size, int32_t azimuth_size, double slant_range_first,
                               double range_spacing, double reference_range, void* stream) {
    if (!d_img || range_size <= 0 || azimuth_size <= 0)
        return set_error(ASARF_ERR_INVALID, "range_spreading_loss: bad arguments");
    RslArgs a{};
    a.img = d_img;
    a.range_size = range_size;
    a.az_size = azimuth_size;
    a.slant_first = slant_range_first;
    a.range_spacing = range_spacing;
    a.ref_range = reference_range;
    int rc = backend_rsl(a, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

static int srgr_common(const float* d_in, int32_t in_x, int32_t y_size, const double poly[5], double range_spacing,
                       int32_t out_x, float* d_out, int32_t* d_start, float* d_frac, void* stream) {
    SrgrArgs a{};
    a.in = d_in;
    a.in_x = in_x;
    a.y_size = y_size;
    a.out_x = out_x;
    for (int k = 0; k < 5; ++k) a.grsr[k] = static_cast<float>(poly[k]);
    a.range_spacing = static_cast<float>(range_spacing);
    a.ground_spacing = 12.5f;
    a.out = d_out;
    a.start = d_start;
    a.frac = d_frac;
    int rc = backend_srgr(a, stream);
    if (rc) return rc;
    return stream_sync(stream);
}

int asarf_srgr(const float* d_in, int32_t in_x, int32_t y_size, const double grsr_poly[5], double range_spacing,
               int32_t out_x, float* d_out, void* stream) {
    if (!d_in || !d_out || !grsr_poly || in_x < 2 || y_size <= 0 || out_x <= 0)
        return set_error(ASARF_ERR_INVALID, "srgr: bad arguments");
    return srgr_common(d_in, in_x, y_size, grsr_poly, range_spacing, out_x, d_out, nullptr, nullptr, stream);
}

int asarf_srgr_index(const double grsr_poly[5], double range_spacing, int32_t out_x, int32_t* d_start, float* d_frac,
                     void* stream) {
    if (!grsr_poly || !d_start || !d_frac || out_x <= 0) return set_error(ASARF_ERR_INVALID, "srgr_index: bad arguments");
    return srgr_common(nullptr, 2, 1, grsr_poly, range_spacing, out_x, nullptr, d_start, d_frac, stream);
}

}  // extern "C"
