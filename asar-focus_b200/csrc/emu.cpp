// Host emulation backend: runs the kernel bodies of bodies.cuh single-threaded on the CPU
// (tid = 0, nthr = 1, one block after another).  Built only into the test library
// libasarf_emu.so so the CPU test suite can check the exact kernel code against the
// oracle; the product library links kernels.cu instead and has no CPU path.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "context_cache.h"
#include "internal.h"
#include "asarf.h"
#include "backend.h"
#include "bodies.cuh"
#include "plan.h"

namespace asarf {

namespace {
// Shared-memory stand-in with the device's 16-byte vector alignment.
struct TileBuf {
    std::vector<float4> v;
    explicit TileBuf(size_t bytes) : v(bytes / sizeof(float4) + 2) {}
    float2* data() { return reinterpret_cast<float2*>(v.data()); }
};

// Test hooks: a finalisation that fails to launch, and a stream under capture, on which the statistics,
// their finalisation and the clearing of their accumulators are recorded and not run.
bool g_fail_finalize = false;
bool g_capturing = false;
}  // namespace

// The lines of a statistics block in slots as the device's ring holds them (all batches at once), filled by the
// same copies; a copy that leaves the raw buffer or its slot, or is misaligned, is an error.
struct StatsRowsSlots {
    static constexpr bool kCollective = true;
    static constexpr int kMargin = 0;
    const StatsBatches& bt;
    std::vector<float4> ring;  // 16-byte aligned
    std::vector<int> sample0;
    bool ok = true;
    unsigned char* slot(int k, int u) {
        return reinterpret_cast<unsigned char*>(ring.data()) + (static_cast<size_t>(k) * kStatsBatch + u) * kStatsSlotBytes;
    }
    StatsRowsSlots(const RawStatsArgs& a, const RawStatsSmem& sm, const StatsBatches& b)
        : bt(b), ring(static_cast<size_t>(b.count) * kStatsBatch * kStatsSlotBytes / sizeof(float4)),
          sample0(static_cast<size_t>(b.count) * kStatsBatch) {
        std::memset(ring.data(), 0xEE, ring.size() * sizeof(float4));  // nothing may count on what a copy leaves out
        const uint8_t* end = a.raw + static_cast<long long>(a.na - 1) * a.line_bytes + 2ll * a.spl;
        for (int k = 0; k < b.count; ++k) {
            int yg, ye;
            b.lines(k, &yg, &ye);
            for (int y = yg; y < ye; ++y) {
                const StatsSlotCopy c(a, y, sm.off[y - b.ys], sm.x_lo, sm.x_hi);
                unsigned char* base = slot(k, y - yg);
                ok = ok && c.lead + (c.b1 - c.b0) <= kStatsSlotBytes;
                if (ok) c.plain(base);
                if (c.c0 < c.c1) {
                    const long long to = c.lead + (c.c0 - c.b0), n = c.c1 - c.c0;
                    ok = ok && c.c0 >= a.raw && c.c1 <= end && to >= 0 && to + n <= kStatsSlotBytes && n % 16 == 0 &&
                         (reinterpret_cast<uintptr_t>(c.c0) & 15) == 0 && (reinterpret_cast<uintptr_t>(base + to) & 15) == 0;
                    if (ok) std::memcpy(base + to, c.c0, static_cast<size_t>(n));
                }
                sample0[static_cast<size_t>(k) * kStatsBatch + (y - yg)] = c.sample0;
            }
        }
    }
    void begin(int) const {}
    void end(int) const {}
    const uint8_t* row(int k, int u, int) const {
        return reinterpret_cast<const unsigned char*>(ring.data()) +
               (static_cast<size_t>(k) * kStatsBatch + u) * kStatsSlotBytes + sample0[static_cast<size_t>(k) * kStatsBatch + u];
    }
};

// staged: unaligned lines through the slots (the planned path); in place otherwise.
static int emu_raw_stats(const RawStatsArgs& a, int gx, int gy, bool staged) {
    RawStatsSmem sm;
    const FastDiv dgpb = make_fastdiv(static_cast<unsigned int>(a.gpb));
    for (int by = 0; by < gy; ++by)
        for (int bx = 0; bx < gx; ++bx) {
            const StatsBatches bt = raw_stats_begin(a, by, 0, 1, &sm);
            if (a.aligned) {
                raw_stats_body<true>(a, StatsRowsInPlace<true>{a}, bt, bx, 0, 1, &sm);
            } else if (!staged) {
                raw_stats_body<false>(a, StatsRowsInPlace<false>{a}, bt, bx, 0, 1, &sm);
            } else {
                sm.x_lo = 0x3fffffff;
                sm.x_hi = 0;
                for (int c = 0; c < kStatsCols; ++c) {
                    const StatsUnit un(a, dgpb, bx * kStatsCols + c);
                    if (!un.colmask) continue;
                    sm.x_lo = un.x0 < sm.x_lo ? un.x0 : sm.x_lo;
                    sm.x_hi = un.x0 + 4 > sm.x_hi ? un.x0 + 4 : sm.x_hi;
                }
                const StatsRowsSlots rows(a, sm, bt);
                if (!rows.ok) return set_error(ASARF_ERR_INVALID, "statistics slots: a copy out of bounds");
                raw_stats_body<false>(a, rows, bt, bx, 0, 1, &sm);
            }
        }
    return ASARF_OK;
}

int backend_raw_stats(const RawStatsArgs& a, int gx, int gy, void*) {
    return g_capturing ? ASARF_OK : emu_raw_stats(a, gx, gy, true);
}

int backend_raw_stats_fbaq(const RawStatsArgs& a, int gx, int gy, void*) {
    std::vector<FbaqStatsSmem> sm(1);
    for (int by = 0; by < gy; ++by) {
        const int ys = fbaq_tile_start(by);
        const int off = a.swst ? static_cast<int>(a.swst[ys]) - a.min_swst : 0;
        const int len = fbaq_len(a.raw + static_cast<long long>(ys) * a.line_bytes, a.line_bytes);
        a.uniform[by] = 1;
        for (int y = ys; y < (by + 1) * kFbaqStatsLines && y < a.na; ++y)
            if (!fbaq_line_like(a, y, off, len)) a.uniform[by] = 0;
    }
    for (int by = 0; by < gy; ++by)
        for (int bx = 0; bx < gx; ++bx) raw_stats_fbaq_body(a, bx, by, 0, 1, sm.data());
    return ASARF_OK;
}

int backend_stats_fold(const RawStatsArgs& a, int tiles_y, void*) {
    std::vector<double> tree(6 * kFoldTree);
    stats_fold_body(a, tiles_y, 0, 1, tree.data());
    return ASARF_OK;
}

int backend_finalize(const FinalizeArgs& a, void*) {
    if (g_fail_finalize) {
        g_fail_finalize = false;
        return set_error(ASARF_ERR_CUDA, "finalize launch: made to fail");
    }
    if (g_capturing) return ASARF_OK;
    finalize_body(a);
    if (!a.facc) *a.acc = StatAccum{};  // as the device finalisation leaves it
    return ASARF_OK;
}

template <int L, int FMT>
static void emu_rc_ct(const RangeCompressArgs& a, int lines, float2* s) {
    for (int y = 0; y < lines; ++y) range_compress_ct_body<L, FMT>(a, y, 0, s, nullptr);
}

template <int FMT>
static void emu_rc(const RangeCompressArgs& a, int lines, LaunchShape sh) {
    std::vector<float2> s(sh.smem / sizeof(float2) + 1);
    switch (a.plan.n) {
        case 768: emu_rc_ct<768, FMT>(a, lines, s.data()); return;
        case 1024: emu_rc_ct<1024, FMT>(a, lines, s.data()); return;
        case 1536: emu_rc_ct<1536, FMT>(a, lines, s.data()); return;
        case 2048: emu_rc_ct<2048, FMT>(a, lines, s.data()); return;
        case 3072: emu_rc_ct<3072, FMT>(a, lines, s.data()); return;
        case 4096: emu_rc_ct<4096, FMT>(a, lines, s.data()); return;
        case 6144: emu_rc_ct<6144, FMT>(a, lines, s.data()); return;
        case 8192: emu_rc_ct<8192, FMT>(a, lines, s.data()); return;
        default: break;
    }
    for (int y = 0; y < lines; ++y) range_compress_body<FMT>(a, y, 0, 1, s.data(), nullptr);
}

int backend_range_compress(const RangeCompressArgs& a, int lines, LaunchShape sh, void*) {
    if (a.format == kRawAsarFbaq4)
        emu_rc<kRawAsarFbaq4>(a, lines, sh);
    else
        emu_rc<kRawErsBytes>(a, lines, sh);
    return ASARF_OK;
}

// The same instantiation choice as the device backend (strided_schedule_compiled).
template <int R0, int R1, int R2, int XT, int NB>
static void emu_az_strided(const AzStridedArgs& a, int tiles, LaunchShape sh) {
    TileBuf s(sh.smem);
    float2* tw = s.data() + static_cast<size_t>(a.n1) * XT * NB;
    int* row = reinterpret_cast<int*>(tw + a.n1 * NB);
    for (int b = 0; b < a.n2; b += NB) {
        az_strided_tables(a, b, 0, 1, tw, row);
        for (int t = 0; t < tiles; ++t) az_strided_body<R0, R1, R2, XT, NB>(a, t, b, 0, 1, s.data(), tw, row, false);
    }
}

int backend_az_strided(const AzStridedArgs& a, const void*, int tiles, LaunchShape sh, void*) {
    if (a.compiled && a.nb == 1 && strided_schedule_compiled(a.plan1, a.xt)) {
#define ASARF_CASE(R0, R1, R2) \
    if (plan_is(a.plan1, R0, R1, R2)) emu_az_strided<R0, R1, R2, 32, 1>(a, tiles, sh);
        ASARF_STRIDED_SCHEDULES(ASARF_CASE)
#undef ASARF_CASE
    } else if (a.xt == 16) {
        emu_az_strided<0, 0, 0, 16, 1>(a, tiles, sh);
    } else if (a.nb == 2) {
        emu_az_strided<0, 0, 0, 32, 2>(a, tiles, sh);
    } else if (a.nb == 4) {
        emu_az_strided<0, 0, 0, 32, 4>(a, tiles, sh);
    } else if (a.nb == 8) {
        emu_az_strided<0, 0, 0, 32, 8>(a, tiles, sh);
    } else {
        emu_az_strided<0, 0, 0, 32, 1>(a, tiles, sh);
    }
    return ASARF_OK;
}

template <int R0, int R1, int R2>
static void emu_az_rd(const AzRdArgs& a, int tiles, int nblocks, LaunchShape sh, unsigned int* err) {
    TileBuf buf(sh.smem + 128);
    float2* s = buf.data();
    const AzRdTables tab(a, s);
    for (int b = 0; b < nblocks; ++b)
        for (int t = 0; t < tiles; ++t) {
            az_rd_tables(a, t, b, 0, 1, tab);
            az_rd_body<true, R0, R1, R2>(a, t, b, 0, 1, s, tab, err, false);
        }
}

int backend_rcmc_table(float* table, void*) {
    for (int n = 0; n <= kRcmcNodes; ++n) rcmc_weight_row(n, table + static_cast<size_t>(n) * kRcmcRowFloats);
    return ASARF_OK;
}

// The same instantiation choice as the device backend (block_schedule_compiled).
int backend_az_rd(const AzRdArgs& a, const void*, int tiles, int nblocks, LaunchShape sh, unsigned int* err, void*) {
    if (a.compiled && block_schedule_compiled(a.plan2)) {
#define ASARF_CASE(R0, R1, R2) \
    if (plan_is(a.plan2, R0, R1, R2)) emu_az_rd<R0, R1, R2>(a, tiles, nblocks, sh, err);
        ASARF_BLOCK_SCHEDULES(ASARF_CASE)
#undef ASARF_CASE
    } else {
        emu_az_rd<0, 0, 0>(a, tiles, nblocks, sh, err);
    }
    return ASARF_OK;
}

int backend_tail(const TailArgs& a, int rows, LaunchShape sh, unsigned int* err, void*) {
    std::vector<float> s(sh.smem / sizeof(float) + 1);
    for (int y = 0; y < rows; ++y) tail_body(a, y, 0, 1, s.data(), err);
    return ASARF_OK;
}

int backend_ers_unpack(const ErsUnpackArgs& a, void*) {
    for (int y = 0; y < a.lines; ++y) ers_unpack_line(a, y, 0, 1);
    return ASARF_OK;
}

int backend_asar_unpack(const AsarUnpackArgs& a, void*) {
    for (int y = 0; y < a.lines; ++y) asar_unpack_line(a, y, 0, 1);
    return ASARF_OK;
}

int backend_decode(const DecodeArgs& a, void*) {
    for (int y = 0; y < a.lines; ++y) decode_row(a, y, 0, 1);
    return ASARF_OK;
}
int backend_product_stats(const ProductStatsArgs& a, void*) {
    std::vector<double> red(5 * 256), tree(5 * kStatsFoldLeaves);
    for (int b = 0; b < a.blocks; ++b) product_stats_body(a, b, 0, 1, red.data());
    product_stats_fold(a, 0, 1, tree.data());
    return ASARF_OK;
}

int backend_condition(const ConditionArgs& a, int rows, void*) {
    for (int y = 0; y < rows; ++y) condition_row(a, y, 0, 1);
    return ASARF_OK;
}

int backend_decode_fbaq(const DecodeFbaqArgs& a, void*) {
    for (int y = 0; y < a.lines; ++y) decode_fbaq_row(a, y, 0, 1);
    return ASARF_OK;
}

int backend_img_moments(const ImgMomentsArgs& a, int blocks, void*) {
    std::vector<double> red(12);
    for (int b = 0; b < blocks; ++b) {
        if (a.about) img_moments_body<true>(a, b, 0, 1, red.data());
        else img_moments_body<false>(a, b, 0, 1, red.data());
    }
    return ASARF_OK;
}
int backend_iq_apply(const IqApplyArgs& a, long long n, void*) {
    for (long long i = 0; i < n; ++i) iq_apply_item(a, i);
    return ASARF_OK;
}
int backend_zero_nans(float2* img, long long n, void*) {
    for (long long i = 0; i < n; ++i) zero_nan_item(img, i);
    return ASARF_OK;
}
int backend_accc(const AcccArgs& a, int grid_x, int grid_y, void*) {
    std::vector<double> cols(2 * kAcccCols);
    for (int by = 0; by < grid_y; ++by)
        for (int bx = 0; bx < grid_x; ++bx) accc_body(a, bx, by, grid_x, 0, 1, cols.data());
    return ASARF_OK;
}
template <int L>
static void emu_rc_rows_ct(const RcRowsArgs& a, int rows, float2* s) {
    for (int y = 0; y < rows; ++y) rc_rows_ct_body<L>(a, y, 0, s);
}
int backend_rc_rows(const RcRowsArgs& a, int rows, LaunchShape sh, void*) {
    std::vector<float2> s(sh.smem / sizeof(float2) + 1);
    switch (a.ctw ? a.plan.n : 0) {
        case 768: emu_rc_rows_ct<768>(a, rows, s.data()); return ASARF_OK;
        case 1024: emu_rc_rows_ct<1024>(a, rows, s.data()); return ASARF_OK;
        case 1536: emu_rc_rows_ct<1536>(a, rows, s.data()); return ASARF_OK;
        case 2048: emu_rc_rows_ct<2048>(a, rows, s.data()); return ASARF_OK;
        case 3072: emu_rc_rows_ct<3072>(a, rows, s.data()); return ASARF_OK;
        case 4096: emu_rc_rows_ct<4096>(a, rows, s.data()); return ASARF_OK;
        case 6144: emu_rc_rows_ct<6144>(a, rows, s.data()); return ASARF_OK;
        case 8192: emu_rc_rows_ct<8192>(a, rows, s.data()); return ASARF_OK;
        default: break;
    }
    for (int y = 0; y < rows; ++y) rc_rows_body(a, y, 0, 1, s.data());
    return ASARF_OK;
}
int backend_matched_filter(const MatchedFilterArgs& a, void*) {
    for (int pos = 0; pos < a.plan.n; ++pos) {
        double re, im;
        matched_filter_sum(a, pos, 0, 1, &re, &im);
        matched_filter_store(a, pos, re, im);
    }
    return ASARF_OK;
}
int backend_twiddles(const TwiddleArgs& a, void*) {
    for (int i = 0, n = twiddle_count(a); i < n; ++i) twiddle_item(a, i);
    return ASARF_OK;
}
int backend_multilook(const MultilookArgs& a, void*) {
    for (int y = 0; y < a.out_y; ++y) multilook_row_body(a, y, 0, 1);
    return ASARF_OK;
}
int backend_rsl(const RslArgs& a, void*) {
    for (int x = 0; x < a.range_size; ++x) rsl_column(a, x, 0, a.az_size);
    return ASARF_OK;
}
int backend_srgr(const SrgrArgs& a, void*) {
    for (int x = 0; x < a.out_x; ++x) srgr_column(a, x, 0, a.y_size);
    return ASARF_OK;
}

void* mem_alloc(size_t bytes) { return std::calloc(1, bytes ? bytes : 1); }
void mem_free(void* p) { std::free(p); }
void* scratch_alloc(size_t bytes, void*, bool* pooled) {
    *pooled = false;
    return mem_alloc(bytes);
}
void scratch_free(void* p, void*, bool) { mem_free(p); }
int mem_h2d(void* dst, const void* src, size_t n, void*) {
    std::memcpy(dst, src, n);
    return ASARF_OK;
}
int mem_d2h(void* dst, const void* src, size_t n, void*) {
    std::memcpy(dst, src, n);
    return ASARF_OK;
}
int mem_d2d(void* dst, const void* src, size_t n, void*) {
    std::memmove(dst, src, n);
    return ASARF_OK;
}
int mem_d2d_2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t rows, void*) {
    for (size_t r = 0; r < rows; ++r)
        std::memcpy(static_cast<char*>(dst) + r * dpitch, static_cast<const char*>(src) + r * spitch, width);
    return ASARF_OK;
}
bool stream_capturing(void*) { return g_capturing; }
int mem_zero(void* dst, size_t n, void*) {
    if (g_capturing) return ASARF_OK;
    std::memset(dst, 0, n);
    return ASARF_OK;
}
int mem_zero_2d(void* dst, size_t pitch, size_t width, size_t rows, void*) {
    for (size_t r = 0; r < rows; ++r) std::memset(static_cast<char*>(dst) + r * pitch, 0, width);
    return ASARF_OK;
}
int stream_sync(void*) { return ASARF_OK; }
void* event_create() { return std::calloc(1, 8); }
void event_destroy(void* e) { std::free(e); }
int event_record(void*, void*) { return ASARF_OK; }
int event_elapsed(void*, void*, float* ms) {
    *ms = 0.0f;
    return ASARF_OK;
}
size_t smem_optin_limit() { return 227 * 1024; }
int backend_sm_count() { return 148; }  // the B200's, so plans take the device build's shapes

}  // namespace asarf

// Host-emulation counterpart of noalloc.cu: the same bodies over a static host array.
namespace {
struct EmuNoallocScratch {
    asarf::StatAccum acc;
    asarf::FocusState state;
};
EmuNoallocScratch g_emu_scratch;
}  // namespace

extern "C" int asarf_raw_statistics_noalloc(const uint8_t* d_raw, int32_t raw_line_bytes, int32_t samples_per_line,
                                            int32_t range_size, int32_t azimuth_size, const uint16_t* d_swst,
                                            int32_t min_swst, int64_t total_raw_samples, int32_t stats_stride,
                                            double prf, asarf_raw_stats* d_out, void*) {
    using namespace asarf;
    if (!d_raw || !d_out || range_size < 32 || azimuth_size < 2 || samples_per_line <= 0 ||
        samples_per_line > range_size || (stats_stride != 0 && stats_stride < range_size))
        return set_error(ASARF_ERR_INVALID, "raw_statistics_noalloc: bad arguments");
    const int dc_step = range_size / 32;
    const int nblk = (range_size + dc_step - 1) / dc_step;
    if (nblk > kMaxDcBlocks) return set_error(ASARF_ERR_INVALID, "raw_statistics_noalloc: too many Doppler blocks");
    std::memset(&g_emu_scratch.acc, 0, sizeof(StatAccum));
    RawStatsArgs st{};
    st.raw = d_raw;
    st.line_bytes = raw_line_bytes;
    st.spl = samples_per_line;
    st.na = azimuth_size;
    st.nr = range_size;
    st.swst = d_swst;
    st.min_swst = min_swst;
    st.dc_step = dc_step;
    st.nblk = nblk;
    st.lines_per_cta = kStatsLinesPerBlock;
    st.acc = &g_emu_scratch.acc;
    emu_raw_stats(st, raw_stats_grid_x(st, d_raw), (azimuth_size + st.lines_per_cta - 1) / st.lines_per_cta, false);
    FinalizeArgs fin{};
    fin.acc = &g_emu_scratch.acc;
    fin.state = &g_emu_scratch.state;
    fin.n_total = total_raw_samples > 0 ? total_raw_samples : static_cast<long long>(samples_per_line) * azimuth_size;
    const int stride = stats_stride > 0 ? stats_stride : range_size;
    fin.n_pad = static_cast<long long>(stride - range_size) * azimuth_size;
    fin.nr = range_size;
    fin.na = azimuth_size;
    fin.rg_stride = stride;
    fin.dc_step = dc_step;
    fin.nblk = nblk;
    fin.prf = prf;
    finalize_body(fin);
    const FocusState& s = g_emu_scratch.state;
    d_out->dc_i = s.dc_i_d;
    d_out->dc_q = s.dc_q_d;
    d_out->iq_gain = s.iq_gain;
    d_out->phase_error = s.phase_error;
    d_out->stddev_i = s.stddev_i;
    d_out->stddev_q = s.stddev_q;
    for (int k = 0; k < 3; ++k) d_out->doppler_centroid_poly[k] = s.dc_est[k];
    d_out->n_dc_blocks = s.nblk;
    for (int b = 0; b < kMaxDcBlocks; ++b) d_out->dc_block_hz[b] = b < s.nblk ? s.dc_blk_hz[b] : 0.0;
    d_out->applied_dc_i = s.dc_i;
    d_out->applied_dc_q = s.dc_q;
    d_out->applied_gain = s.gain;
    d_out->applied_sin = s.sin_c;
    d_out->applied_cos = s.cos_c;
    d_out->errors = s.errors;
    return ASARF_OK;
}

// Test hook of the host emulation only: drives the context-keyed address cache of the
// allocation-free entry point (context_cache.h) with made-up context ids and a resolver that
// hands out a fresh fake address on every call.  For each key i, addrs[i] receives the
// address returned and the function returns how many times the resolver ran.
extern "C" int asarf_emu_context_cache_probe(const unsigned long long* ids, int n, unsigned long long* addrs) {
    static asarf::ContextAddressCache<4> cache;
    static unsigned long long next_fake = 0x1000;
    int resolutions = 0;
    for (int i = 0; i < n; ++i) {
        void* p = nullptr;
        bool resolved = false;
        cache.get(ids[i], [](void** q) { *q = reinterpret_cast<void*>(next_fake); next_fake += 0x1000; return 0; },
                  &p, &resolved);
        resolutions += resolved ? 1 : 0;
        addrs[i] = reinterpret_cast<unsigned long long>(p);
    }
    return resolutions;
}

// Test hook of the host emulation only: radices of a strided or contiguous azimuth length; returns their number.
extern "C" int asarf_emu_radices(int n, int strided, int out[16]) {
    const std::vector<int> r = strided ? asarf::strided_radices(n) : asarf::block_radices(n);
    for (size_t i = 0; i < r.size() && i < 16; ++i) out[i] = r[i];
    return static_cast<int>(r.size());
}

// Test hooks of the host emulation only: the next finalisation fails; the stream is under capture; a
// plan's statistics accumulators are all zero.
extern "C" void asarf_emu_fail_finalize() { asarf::g_fail_finalize = true; }
extern "C" void asarf_emu_capture(int on) { asarf::g_capturing = on != 0; }
extern "C" int asarf_emu_accumulators_clear(const asarf_plan* p) {
    const unsigned char* b = reinterpret_cast<const unsigned char*>(p->acc);
    for (size_t i = 0; i < sizeof(asarf::StatAccum); ++i)
        if (b[i]) return 0;
    return 1;
}

// Test hook of the host emulation only: the range-Doppler tile (length n2, width wt) that the planner takes
// for N = n1 * n2 rows of nk columns, and the rows of its TMA boxes.
extern "C" void asarf_emu_rd_tile(int N, int nk, int hl, int hr, int* n2, int* wt, int* box_rows) {
    using namespace asarf;
    *n2 = choose_az_n2(N, nk, hl, hr, false);
    *wt = az_rd_tile_width(*n2, hl, hr, false, smem_optin_limit()) + hl + hr;
    *box_rows = rd_box_rows(*n2, *wt);
}

namespace asarf {
int backend_az_rd_split(const AzRdArgs&, const AzRdSplit&, const void*, int, int, LaunchShape, unsigned int*, void*) {
    return set_error(ASARF_ERR_INVALID, "split precision runs on the tensor cores only (no host emulation)");
}
int event_sync(void*) { return ASARF_OK; }
void* stream_create() { return std::calloc(1, 8); }
void stream_destroy(void* s) { std::free(s); }
int stream_wait_event(void*, void*) { return ASARF_OK; }
bool graphs_supported() { return false; }
int graph_capture_begin(void*) { return set_error(ASARF_ERR_INVALID, "no graphs in the host emulation"); }
int graph_capture_end(void*, void**) { return set_error(ASARF_ERR_INVALID, "no graphs in the host emulation"); }
int graph_launch(void*, void*) { return set_error(ASARF_ERR_INVALID, "no graphs in the host emulation"); }
void graph_destroy(void*) {}
const char* backend_name() { return "host-emulation"; }
int backend_make_tmap(void*, int, void*, const unsigned long long*, const unsigned long long*, const unsigned int*) {
    return set_error(ASARF_ERR_INVALID, "no tensor maps in host emulation");
}

}  // namespace asarf
