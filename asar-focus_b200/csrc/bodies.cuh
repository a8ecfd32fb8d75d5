// Kernel bodies of the focusing path, written once for the device and the host emulation.
//
// A body is a function of (block coordinates, tid, nthr, shared-memory pointer) made of
// phases separated by ASARF_SYNC(); inside a phase every work item is independent.
// Reference behaviour each body reproduces is cited in its comment
// (paths relative to the asar-focus source tree).
#pragma once

#include <cmath>
#include <cstdint>

#include "fft.cuh"
#include "fft_ct.cuh"
#include "hd.cuh"
#include "params.h"

namespace asarf {

ASARF_HD ASARF_INLINE void atomic_or_u32(unsigned int* p, unsigned int v) {
#if defined(__CUDA_ARCH__)
    atomicOr(p, v);
#else
    *p |= v;
#endif
}

// numpy.blackman(16) in float32, the RCMC tap window (sar/range_doppler_algorithm.cu:46-52):
// 0.42 - 0.5 cos(2 pi n / 15) + 0.08 cos(4 pi n / 15) rounded to float.
#define ASARF_BLACKMAN16                                                                                      \
    {-1.3877787807814457e-17f, 0.016757719218730927f, 0.07707241922616959f, 0.20077013969421387f,             \
     0.3940124213695526f,      0.6299999952316284f,   0.8492298722267151f,  0.9821574091911316f,              \
     0.9821574091911316f,      0.8492298722267151f,   0.6299999952316284f,  0.3940124213695526f,              \
     0.20077013969421387f,     0.07707241922616959f,  0.016757719218730927f, -1.3877787807814457e-17f}

// Device Polyval<N> of the reference (float Horner; nvcc contracts r*x + e into one fma).
template <int N>
ASARF_HD ASARF_INLINE float polyval_f32(const float (&p)[N], float x) {
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) r = fma_rn(r, x, p[i]);
    return r;
}

// ----------------------------------------------------------------------------- least squares
// Householder-QR least-squares polynomial fit, coefficients highest power first
// (Polyfit, util/src/math_utils.cc:23-44).  m <= 128 points, degree <= 4.
template <int kM, int kN>
ASARF_HD inline bool polyfit_qr(const double* x, const double* y, int m, int deg, double* out) {
    const int n = deg + 1;
    if (m > kM || n > kN || m < n) return false;
    double A[kN][kM];  // column-major: A[col][row]
    double b[kM];
    for (int r = 0; r < m; ++r) {
        double v = 1.0;
        for (int c = 0; c < n; ++c) {
            A[c][r] = v;
            v *= x[r];
        }
        b[r] = y[r];
    }
    for (int k = 0; k < n; ++k) {
        double nrm = 0.0;
        for (int r = k; r < m; ++r) nrm += A[k][r] * A[k][r];
        nrm = sqrt(nrm);
        if (nrm == 0.0) return false;
        const double alpha = A[k][k] > 0 ? -nrm : nrm;
        // Householder vector v = A[k][k:] - alpha e_k kept in column k (its head in vk)
        const double vk = A[k][k] - alpha;
        double vn = vk * vk;
        for (int r = k + 1; r < m; ++r) vn += A[k][r] * A[k][r];
        if (vn == 0.0) return false;
        for (int c = k + 1; c < n; ++c) {
            double d = vk * A[c][k];
            for (int r = k + 1; r < m; ++r) d += A[k][r] * A[c][r];
            const double f = 2.0 * d / vn;
            A[c][k] -= f * vk;
            for (int r = k + 1; r < m; ++r) A[c][r] -= f * A[k][r];
        }
        double d = vk * b[k];
        for (int r = k + 1; r < m; ++r) d += A[k][r] * b[r];
        const double f = 2.0 * d / vn;
        b[k] -= f * vk;
        for (int r = k + 1; r < m; ++r) b[r] -= f * A[k][r];
        A[k][k] = alpha;  // R diagonal
    }
    double c[kN];
    for (int k = n - 1; k >= 0; --k) {
        double s = b[k];
        for (int j = k + 1; j < n; ++j) s -= A[j][k] * c[j];
        c[k] = s / A[k][k];
    }
    for (int k = 0; k < n; ++k) out[k] = c[n - 1 - k];
    return true;
}

// ----------------------------------------------------------------------------- raw statistics
// One pass over the raw I/Q bytes.  Replaces, exactly and in integers, the reductions of
// RawDataCorrection (sar/iq_correction.cu:188-274: mean, std-dev, gain and phase sums)
// and of CalculateDopplerCentroid (sar/fractional_doppler_centroid.cu:33-69: lag-1
// azimuth correlation per range block): the IQ correction is affine in the raw bytes,
// so every sum the reference takes over corrected floats is a closed form of these.
// Block (bx, by) covers kStatsCols work units and lines [by*L, (by+1)*L).  A unit is the columns
// of one Doppler block inside an aligned group of 4 (columns 4g .. 4g + 3, one 8-byte window per
// line, byte-lane dot products for all sums; a group that straddles a Doppler block boundary is
// two units, one per block, each masking the other's columns), so every sum a thread keeps
// belongs to a single Doppler block, and kStatsBatch lines are read before any is consumed.
// A window is one aligned 8-byte word when the raw base and line stride are 8-byte aligned,
// otherwise the three aligned 4-byte words around it, funnelled into place.
//
// Unaligned lines' bytes under a block's columns (2 KB a line) arrive in a ring of kStatsStages batches
// in shared memory, a bulk copy per line, the batches ahead in flight while one is summed: 5193 x
// 17011, 10386-byte lines, 212 -> 118 us; batches of 16 lines in two stages 172.  Both forms are bound
// by instructions and the chain of batches (315 MB in 113 us are 2.8 TB/s), so a block whose lines
// have one SWST shift checks its windows once: aligned lines of 5616 x 28000 140 -> 113 us.
constexpr int kStatsCols = 256;
constexpr int kStatsBatch = 8;
constexpr int kStatsMaxLines = 256;
// lines per block of the statistics kernel, with the whole-wave rule below (28000, 30000, 60000 lines of 5616
// samples: 128 -> 114, 135, 250 us; 160 -> 114, 116, 231; 192 -> 114, 115, 213; 256 -> 127, 125, 220)
constexpr int kStatsLinesPerBlock = 192;
constexpr int kStatsBlocksPerSm = 3;  // resident blocks of k_raw_stats (its launch bounds)

// Lines per statistics block for a grid of gx block columns over na lines.  When blocks of
// kStatsLinesPerBlock lines fill the `slots` resident blocks more than once, that height, raised
// in whole batches (at most kStatsMaxLines) when it fits the grid into one wave fewer, since the
// last wave of a grid of equal blocks runs mostly empty (ASAR IM-like 30000 lines, 6 columns, 444
// slots: 942 blocks of 192 lines take three waves, 870 of 208 lines two).  Scenes below that
// get blocks low enough to fill the slots once, at least kStatsMinLines: a block's time is its
// chain of batches, so blocks of 192 lines left a 768 x 1024 scene to 6 of 148 SMs (kernel time
// 41 -> 11 us; 2048 x 4096 47 -> 24, 5644 x 9973 101 -> 76 us).
constexpr int kStatsMinLines = 16;
inline int stats_lines_per_block(int na, int gx, int slots) {
    const long long rows = (na + kStatsLinesPerBlock - 1) / kStatsLinesPerBlock;
    const long long waves = (rows * gx + slots - 1) / slots;
    const long long fit_rows = gx > 0 ? (waves > 1 ? waves - 1 : 1) * slots / gx : 0;
    if (fit_rows > 0) {
        long long l = (na + fit_rows - 1) / fit_rows;
        l = (l + kStatsBatch - 1) / kStatsBatch * kStatsBatch;
        if (l < kStatsMinLines) l = kStatsMinLines;
        if (l <= (waves > 1 ? kStatsMaxLines : kStatsLinesPerBlock)) return static_cast<int>(l);
    }
    return kStatsLinesPerBlock;
}

constexpr int kStatsStages = 4;
// a line's bytes in the ring: at most kStatsCols groups of 4 columns, from a 16-byte boundary on
constexpr int kStatsSlotBytes = 8 * kStatsCols + 32;
constexpr size_t kStatsRingBytes = static_cast<size_t>(kStatsStages) * kStatsBatch * kStatsSlotBytes;

struct RawStatsSmem {
    unsigned long long mom[6];
    unsigned long long lag[kMaxDcBlocks][9];
    int off[kStatsMaxLines + 1];  // SWST shift of the block's lines (and the line before)
    int same;                     // 1: all those shifts are equal
    int x_lo, x_hi;               // columns the block's units read
    int sample0[kStatsStages * kStatsBatch];  // ring offset of the lines' sample 0 (may lie before the slot)
    uint64_t full[kStatsStages];  // mbarriers: a batch's bytes have arrived
};

// Batch k of a statistics block's lines [ys, y1): the line before the block's first (its lag-sum
// partner) is a batch of its own, so every following batch holds kStatsBatch counted lines.
struct StatsBatches {
    int ys, y0, y1, count;
    ASARF_HD ASARF_INLINE StatsBatches(int y0_, int y1_) : ys(y0_ > 0 ? y0_ - 1 : 0), y0(y0_), y1(y1_) {
        count = (ys < y0 ? 1 : 0) + (y1 - y0 + kStatsBatch - 1) / kStatsBatch;
    }
    ASARF_HD ASARF_INLINE void lines(int k, int* yg, int* ye) const {
        const int pre = ys < y0 ? 1 : 0;
        *yg = k < pre ? ys : y0 + (k - pre) * kStatsBatch;
        *ye = k < pre ? y0 : (*yg + kStatsBatch < y1 ? *yg + kStatsBatch : y1);
    }
};

// Lines read in place (the caller-scratch statistics and the host emulation).  kMargin: samples past a window that the words around it reach.
template <bool ALIGNED>
struct StatsRowsInPlace {
    static constexpr bool kCollective = false;
    static constexpr int kMargin = ALIGNED ? 0 : 1;
    const RawStatsArgs& a;
    ASARF_HD ASARF_INLINE void begin(int) const {}
    ASARF_HD ASARF_INLINE void end(int) const {}
    ASARF_HD ASARF_INLINE const uint8_t* row(int, int, int y) const {
        return a.raw + static_cast<long long>(y) * a.line_bytes;
    }
};

// What a ring slot takes of line y: the bytes [b0, b1) of the samples under columns [x_lo, x_hi) (none: b0 =
// b1), b0 at slot offset `lead`.  The 16-byte units [c0, c1) (none: c1 <= c0) move by a bulk copy,
// from the boundary before the first byte to the one after the last; at the two ends of the raw buffer, where
// that would leave it, a unit less, and the bytes it would have brought by plain loads.
struct StatsSlotCopy {
    const uint8_t *b0, *b1, *c0, *c1;
    int lead;
    int sample0;  // slot offset of the line's sample 0 (may lie before the slot)
    ASARF_HD ASARF_INLINE StatsSlotCopy(const RawStatsArgs& a, int y, int off, int x_lo, int x_hi) {
        const int i0 = x_lo > off ? x_lo - off : 0, i1 = x_hi - off < a.spl ? x_hi - off : a.spl;
        const uint8_t* row = a.raw + static_cast<long long>(y) * a.line_bytes;
        b0 = row + 2ll * i0;
        b1 = i1 > i0 ? row + 2ll * i1 : b0;
        lead = static_cast<int>(reinterpret_cast<uintptr_t>(b0) & 15);
        sample0 = lead - 2 * i0;
        c0 = b0 - lead;
        c1 = b1 + (static_cast<int>(-reinterpret_cast<uintptr_t>(b1)) & 15);
        if (c0 < a.raw) c0 += 16;
        if (c1 > a.raw + static_cast<long long>(a.na - 1) * a.line_bytes + 2ll * a.spl) c1 -= 16;
        if (b0 == b1) c1 = c0;
    }
    // the odd bytes, to slot offsets
    ASARF_HD ASARF_INLINE void plain(unsigned char* slot) const {
        for (const uint8_t* p = b0; p < c0 && p < b1; ++p) slot[lead + (p - b0)] = *p;
        for (const uint8_t* p = c1 > b0 ? c1 : b0; p < b1; ++p) slot[lead + (p - b0)] = *p;
    }
};

// Host side: work units and grid width of the statistics kernel for this raw buffer.
inline int raw_stats_grid_x(RawStatsArgs& a, const void* raw) {
    a.gpb = (a.dc_step + 3) / 4 + 1;  // aligned groups a block's columns touch
    a.aligned = (reinterpret_cast<uintptr_t>(raw) % 8 == 0 && a.line_bytes % 8 == 0) ? 1 : 0;
    const int units = a.nblk * a.gpb;
    return (units + kStatsCols - 1) / kStatsCols;
}

// sum over the four byte lanes of a * b, plus c
ASARF_HD ASARF_INLINE unsigned int dp4(unsigned int a, unsigned int b, unsigned int c) {
#if defined(__CUDA_ARCH__)
    return __dp4a(a, b, c);
#else
    for (int k = 0; k < 32; k += 8) c += ((a >> k) & 0xffu) * ((b >> k) & 0xffu);
    return c;
#endif
}

ASARF_HD ASARF_INLINE unsigned int funnel_r(unsigned int lo, unsigned int hi, unsigned int sh) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, sh);
#else
    return sh == 0 ? lo : static_cast<unsigned int>(((static_cast<unsigned long long>(hi) << 32) | lo) >> sh);
#endif
}

// bytes of (x, y) = b0..b7 picked by the low 3 bits of each selector nibble (PRMT default mode)
ASARF_HD ASARF_INLINE unsigned int byte_perm(unsigned int x, unsigned int y, unsigned int s) {
#if defined(__CUDA_ARCH__)
    return __byte_perm(x, y, s);
#else
    const unsigned long long xy = (static_cast<unsigned long long>(y) << 32) | x;
    unsigned int r = 0;
    for (int n = 0; n < 4; ++n) r |= static_cast<unsigned int>((xy >> (8 * ((s >> (4 * n)) & 7u))) & 0xffu) << (8 * n);
    return r;
#endif
}

ASARF_HD ASARF_INLINE int popc_u32(unsigned int v) {
#if defined(__CUDA_ARCH__)
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}

// Reduce this thread's sums into the block's shared accumulators (lag sums of Doppler block blk).
ASARF_HD ASARF_INLINE void raw_stats_reduce(RawStatsSmem* sm, bool valid, int blk, unsigned long long mv[6],
                                            unsigned int lv[9]) {
#if defined(__CUDA_ARCH__)
    // every lane of the block runs exactly one unit (kStatsCols == blockDim.x): warp sums first
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        unsigned long long v = mv[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        mv[k] = v;
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k) atomic_add_u64(&sm->mom[k], mv[k]);
    }
    const int bmin = __reduce_min_sync(0xffffffffu, valid ? blk : 0x7fffffff);
    const int bmax = __reduce_max_sync(0xffffffffu, valid ? blk : -1);
    if (bmin == bmax) {
#pragma unroll
        for (int q = 0; q < 9; ++q) lv[q] = __reduce_add_sync(0xffffffffu, valid ? lv[q] : 0u);
        if ((threadIdx.x & 31) == 0)
            for (int q = 0; q < 9; ++q) atomic_add_u64(&sm->lag[bmin][q], lv[q]);
    } else if (valid) {
        for (int q = 0; q < 9; ++q) atomic_add_u64(&sm->lag[blk][q], lv[q]);
    }
#else
    for (int k = 0; k < 6; ++k) atomic_add_u64(&sm->mom[k], mv[k]);
    if (valid)
        for (int q = 0; q < 9; ++q) atomic_add_u64(&sm->lag[blk][q], lv[q]);
#endif
}

// The columns of `colmask` (bit k: column x0 + k) of the aligned group at x0 (x0 % 4 == 0), all in
// one Doppler block.  A line's four samples are the 8 bytes (I0 Q0 I1 Q1 | I2 Q2 I3 Q3) at
// row + 2*(x0 - off) (the SWST shift is a multiple of 4 samples, so with ALIGNED the window stays
// 8-byte aligned on every line; without, it starts at any even address).  A window that leaves its
// record is read sample by sample.  Samples outside the record or the mask are zero bytes, which
// drop out of every sum.  Where the block's lines have one shift, a window that lies inside one
// record lies inside all: its batches are read with nothing checked per line.  With kCollective rows
// every thread of the block runs the batches, an idle one at another's columns with none its own.
template <bool ALIGNED, class Rows>
ASARF_HD ASARF_INLINE void raw_stats_quad(const RawStatsArgs& a, const RawStatsSmem* sm, const Rows& rows, int x0,
                                          unsigned int colmask, const StatsBatches& bt, unsigned long long mv[6],
                                          unsigned int lv[9]) {
    const int y0 = bt.y0, ys = bt.ys;
    const int i_same = x0 - sm->off[0];
    const bool inside = sm->same && i_same >= Rows::kMargin && i_same + 4 + Rows::kMargin <= a.spl;
    constexpr unsigned int kLo = 0x00ff00ffu, kOnes = 0x01010101u;
    const unsigned int colbits = colmask;
    const int ncol = popc_u32(colmask);
    unsigned int cnt = 0, si = 0, sq = 0, sii = 0, sqq = 0, siq = 0;
    unsigned int l0 = 0, l1 = 0, l2 = 0, l3 = 0, l4 = 0, l5 = 0, l6 = 0, l7 = 0, l8 = 0;
    unsigned int pI0 = 0, pI1 = 0, pQ0 = 0, pQ1 = 0, pfb = 0;
    // byte masks of the group's columns: in the packed I (or Q) word byte k is column k; in the
    // two raw words column k is the 16-bit lane k % 2 of word k / 2
    const unsigned int cm = ((colmask & 1u) ? 0x000000ffu : 0u) | ((colmask & 2u) ? 0x0000ff00u : 0u) |
                            ((colmask & 4u) ? 0x00ff0000u : 0u) | ((colmask & 8u) ? 0xff000000u : 0u);
    for (int k = 0; k < bt.count; ++k) {
        int yg, ye;
        bt.lines(k, &yg, &ye);
        rows.begin(k);
        uint2 w[kStatsBatch];
        unsigned int fbv[kStatsBatch], whole = 0;
        // the whole 8-byte window at p is inside its record
        auto window = [](const uint8_t* p) -> uint2 {
            if constexpr (ALIGNED) {
                return *reinterpret_cast<const uint2*>(p);
            } else {
                const unsigned int odd = static_cast<unsigned int>(reinterpret_cast<uintptr_t>(p) & 2);
                const uint32_t* q = reinterpret_cast<const uint32_t*>(p - odd);
                const uint32_t q0 = q[0], q1 = q[1], q2 = odd ? q[2] : 0u;
                return make_uint2(funnel_r(q0, q1, 8 * odd), funnel_r(q1, q2, 8 * odd));
            }
        };
        bool interior = ye - yg == kStatsBatch && pfb == colbits;
        if (interior && inside) {
#pragma unroll
            for (int u = 0; u < kStatsBatch; ++u) w[u] = window(rows.row(k, u, yg + u) + 2ll * i_same);
        } else {
#pragma unroll
            for (int u = 0; u < kStatsBatch; ++u) {
                const int y = yg + u;
                w[u] = make_uint2(0u, 0u);
                fbv[u] = 0u;
                if (y < ye && colbits) {
                    const int i = x0 - sm->off[y - ys];
                    const uint8_t* p = rows.row(k, u, y) + 2ll * i;
                    if (i >= Rows::kMargin && i + 4 + Rows::kMargin <= a.spl) {
                        w[u] = window(p);
                        fbv[u] = colbits;
                        whole |= 1u << u;
                    } else {
                        // record edge: sample by sample
                        for (int c = 0; c < 4; ++c) {
                            if (!((colbits >> c) & 1u) || i + c < 0 || i + c >= a.spl) continue;
                            const unsigned int v = *reinterpret_cast<const uint16_t*>(p + 2 * c);
                            if (c < 2) w[u].x |= v << (16 * c);
                            else w[u].y |= v << (16 * (c - 2));
                            fbv[u] |= 1u << c;
                        }
                    }
                }
            }
            interior = interior && (whole == (1u << kStatsBatch) - 1u || colbits == 0u);
        }
        rows.end(k);
        // Interior batch: every line and the one before it counted, filled and read through a
        // whole window.  The group's I and Q bytes are packed into one word each, so every sum
        // is one byte-lane dot product and nothing is masked per line (an idle thread takes this path
        // with its warp and sums zeros).
        if (interior) {
            unsigned int pI = byte_perm(pI0, pI1, 0x6420u), pQ = byte_perm(pQ0, pQ1, 0x6420u);
            unsigned int psI = dp4(pI, kOnes, 0u), psQ = dp4(pQ, kOnes, 0u);
#pragma unroll
            for (int u = 0; u < kStatsBatch; ++u) {
                const unsigned int I = byte_perm(w[u].x, w[u].y, 0x6420u) & cm;
                const unsigned int Q = byte_perm(w[u].x, w[u].y, 0x7531u) & cm;
                const unsigned int sI = dp4(I, kOnes, 0u), sQ = dp4(Q, kOnes, 0u);
                si += sI;
                sq += sQ;
                sii = dp4(I, I, sii);
                sqq = dp4(Q, Q, sqq);
                siq = dp4(I, Q, siq);
                l1 += psI;
                l2 += psQ;
                l3 += sI;
                l4 += sQ;
                l5 = dp4(pI, I, l5);
                l6 = dp4(pQ, Q, l6);
                l7 = dp4(pI, Q, l7);
                l8 = dp4(pQ, I, l8);
                pI = I, pQ = Q, psI = sI, psQ = sQ;
            }
            cnt += static_cast<unsigned int>(kStatsBatch * ncol);
            l0 += static_cast<unsigned int>(kStatsBatch * ncol);
            // back to the two-word form the general loop carries (I or Q bytes in lanes 0 and 2)
            pI0 = byte_perm(pI, 0u, 0x4140u), pI1 = byte_perm(pI, 0u, 0x4342u);
            pQ0 = byte_perm(pQ, 0u, 0x4140u), pQ1 = byte_perm(pQ, 0u, 0x4342u);
            continue;
        }
#pragma unroll
        for (int u = 0; u < kStatsBatch; ++u) {
            const int y = yg + u;
            if (y >= ye) break;
            const unsigned int fb = fbv[u];
            const unsigned int m0 = ((fb & 1u) ? 0x0000ffffu : 0u) | ((fb & 2u) ? 0xffff0000u : 0u);
            const unsigned int m1 = ((fb & 4u) ? 0x0000ffffu : 0u) | ((fb & 8u) ? 0xffff0000u : 0u);
            const unsigned int c0 = w[u].x & m0, c1 = w[u].y & m1;
            const unsigned int I0 = c0 & kLo, I1 = c1 & kLo;
            const unsigned int Q0 = (c0 >> 8) & kLo, Q1 = (c1 >> 8) & kLo;
            if (y >= y0) {
                cnt += static_cast<unsigned int>(popc_u32(fb));
                si = dp4(I0, kOnes, dp4(I1, kOnes, si));
                sq = dp4(Q0, kOnes, dp4(Q1, kOnes, sq));
                sii = dp4(I0, I0, dp4(I1, I1, sii));
                sqq = dp4(Q0, Q0, dp4(Q1, Q1, sqq));
                siq = dp4(I0, Q0, dp4(I1, Q1, siq));
                if (y > 0) {
                    // pairs (y-1, y) with both samples filled
                    const unsigned int pb = fb & pfb;
                    if (pb == fb && pb == pfb) {
                        l1 = dp4(pI0, kOnes, dp4(pI1, kOnes, l1));
                        l2 = dp4(pQ0, kOnes, dp4(pQ1, kOnes, l2));
                        l3 = dp4(I0, kOnes, dp4(I1, kOnes, l3));
                        l4 = dp4(Q0, kOnes, dp4(Q1, kOnes, l4));
                    } else {
                        const unsigned int n0 = ((pb & 1u) ? 0x000000ffu : 0u) | ((pb & 2u) ? 0x00ff0000u : 0u);
                        const unsigned int n1 = ((pb & 4u) ? 0x000000ffu : 0u) | ((pb & 8u) ? 0x00ff0000u : 0u);
                        l1 = dp4(pI0 & n0, kOnes, dp4(pI1 & n1, kOnes, l1));
                        l2 = dp4(pQ0 & n0, kOnes, dp4(pQ1 & n1, kOnes, l2));
                        l3 = dp4(I0 & n0, kOnes, dp4(I1 & n1, kOnes, l3));
                        l4 = dp4(Q0 & n0, kOnes, dp4(Q1 & n1, kOnes, l4));
                    }
                    l0 += static_cast<unsigned int>(popc_u32(pb));
                    // products vanish wherever either sample is unfilled (its bytes are zero)
                    l5 = dp4(pI0, I0, dp4(pI1, I1, l5));
                    l6 = dp4(pQ0, Q0, dp4(pQ1, Q1, l6));
                    l7 = dp4(pI0, Q0, dp4(pI1, Q1, l7));
                    l8 = dp4(pQ0, I0, dp4(pQ1, I1, l8));
                }
            }
            pI0 = I0, pI1 = I1, pQ0 = Q0, pQ1 = Q1, pfb = fb;
        }
    }
    mv[0] = cnt, mv[1] = si, mv[2] = sq, mv[3] = sii, mv[4] = sqq, mv[5] = siq;
    lv[0] = l0, lv[1] = l1, lv[2] = l2, lv[3] = l3, lv[4] = l4, lv[5] = l5, lv[6] = l6, lv[7] = l7, lv[8] = l8;
}

// Unit -> first column of its aligned group, its columns and its Doppler block: group k of block blk
// is the aligned group at (block start & ~3) + 4k, the block's columns [xs, xe) in it.
struct StatsUnit {
    int blk, x0;
    unsigned int colmask;
    ASARF_HD ASARF_INLINE StatsUnit(const RawStatsArgs& a, const FastDiv& dgpb, int unit) {
        blk = static_cast<int>(fdiv_u(static_cast<unsigned int>(unit), dgpb));
        const int xs = blk * a.dc_step;
        const int xe = (blk + 1) * a.dc_step < a.nr ? (blk + 1) * a.dc_step : a.nr;
        x0 = (xs & ~3) + 4 * (unit - blk * a.gpb);
        const int c_lo = xs > x0 ? xs - x0 : 0;
        const int c_hi = xe - x0 < 4 ? xe - x0 : 4;
        colmask = blk < a.nblk && c_hi > c_lo ? ((1u << c_hi) - 1u) & ~((1u << c_lo) - 1u) : 0u;
    }
};

// Lines of the block by, their SWST shifts and the block's accumulators in sm (the caller barriers).
ASARF_HD ASARF_INLINE StatsBatches raw_stats_begin(const RawStatsArgs& a, int by, int tid, int nthr, RawStatsSmem* sm) {
    unsigned long long* flat = &sm->mom[0];
    for (int i = tid; i < 6 + kMaxDcBlocks * 9; i += nthr) flat[i] = 0ull;
    const int y0 = by * a.lines_per_cta;
    const StatsBatches bt(y0, y0 + a.lines_per_cta < a.na ? y0 + a.lines_per_cta : a.na);
    bool same = true;
    for (int y = bt.ys + tid; y < bt.y1; y += nthr) {
        sm->off[y - bt.ys] = a.swst ? 4 * (static_cast<int>(a.swst[y]) - a.min_swst) : 0;
        same = same && (!a.swst || a.swst[y] == a.swst[bt.ys]);
    }
#if defined(__CUDA_ARCH__)
    same = __syncthreads_and(same) != 0;
#endif
    if (tid == 0) sm->same = same ? 1 : 0;
    return bt;
}

template <bool ALIGNED, class Rows>
ASARF_HD ASARF_INLINE void raw_stats_body(const RawStatsArgs& a, const Rows& rows, const StatsBatches& bt, int bx, int tid,
                                          int nthr, RawStatsSmem* sm) {
    const unsigned long long* flat = &sm->mom[0];
    const int nflat = 6 + a.nblk * 9;
    const FastDiv dgpb = make_fastdiv(static_cast<unsigned int>(a.gpb));
    for (int c = tid; c < kStatsCols; c += nthr) {
        const StatsUnit un(a, dgpb, bx * kStatsCols + c);
        unsigned long long mv[6] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
        unsigned int lv[9] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        if (un.colmask || Rows::kCollective)
            raw_stats_quad<ALIGNED>(a, sm, rows, un.colmask ? un.x0 : sm->x_lo, un.colmask, bt, mv, lv);
        raw_stats_reduce(sm, un.colmask != 0, un.blk, mv, lv);
    }
    ASARF_SYNC();
    unsigned long long* gflat = &a.acc->mom[0];
    for (int i = tid; i < nflat; i += nthr) {
        const unsigned long long v = flat[i];
        if (v) atomic_add_u64(gflat + i, v);
    }
}

// ----------------------------------------------------------------------------- FBAQ4 records
// ENVISAT ASAR raw records (ConvertAsarImBlocksToComplexKernel,
// envisat_format/src/envisat_format_kernels.cu:160-209): a 2-byte little-endian length L of
// the block data, then 64-byte blocks of one block-id byte and 63 codeword bytes (I code in
// the high nibble, Q code in the low one).  Sample r of a record is codeword byte
// j = r + r / 63 + 1 of the block data and exists when j < L (and j lies inside the record).

// Instrument-file table index of a 4-bit code of block `block`: sign-magnitude codes 0..7 are
// levels 8..15, codes 8..15 levels 7..0 (Fbaq4IndexCalc, envisat_format/include/envisat_parse_util.cuh:75-84).
ASARF_HD ASARF_INLINE int fbaq4_index(int block, int code) { return 256 * (code > 7 ? 15 - code : 8 + code) + block; }

// Usable block-data bytes of a record: its length field, bounded by the record stride.
ASARF_HD ASARF_INLINE int fbaq_len(const uint8_t* rec, long long line_bytes) {
    const int len = rec[0] | (rec[1] << 8);
    const long long room = line_bytes - 2;
    return len < room ? len : static_cast<int>(room);
}

// Sample r >= 0 of a record through the permuted tables lut[16 * block id + code].
ASARF_HD ASARF_INLINE bool fbaq_sample(const uint8_t* rec, int len, int r, const FastDiv& d63,
                                       const float* __restrict__ lut_i, const float* __restrict__ lut_q, float* iv,
                                       float* qv) {
    const int b = static_cast<int>(fdiv_u(static_cast<unsigned int>(r), d63));
    const int j = r + b + 1;
    if (j >= len) return false;
    const int id = rec[2 + 64 * b];
    const int cw = rec[2 + j];
    *iv = ASARF_LDG(lut_i + 16 * id + (cw >> 4));
    *qv = ASARF_LDG(lut_q + 16 * id + (cw & 15));
    return true;
}

// Statistics of FBAQ4 records: the sums of k_raw_stats over the decoded samples, in
// FP64.  Tile (bx, by) = 32 columns x kFbaqStatsLines lines; warp w of the block takes lines
// [y0 + w * sub, y0 + (w + 1) * sub) of the tile, lane = column.  Per-lane sums are combined
// over the warps, then over the lanes (moments: fixed pairwise tree; lag sums: per Doppler
// block in lane order), and the tile's partials are written, not accumulated: the fold sums
// them in a fixed order, so the statistics do not depend on scheduling.
// Where all records of a tile have the same SWST shift and length (nearly all tiles), a lane's
// sample has one place in every record: no index arithmetic per line, no masks, and the sums over
// single samples of the pairs follow from the moments and the range's end samples, so a line costs
// nine FP64 operations instead of fifteen.  The tables hold doubles (the float entries, exactly):
// four conversions a sample went at a sixteenth of the FP32 rate.  The next lines' bytes are
// loaded while these are summed.  176 x 15 tiles of a 5616 x 30000 scene: 632 -> 325 us.
constexpr int kFbaqSums = 15;  // 6 moments + 9 lag sums
constexpr int kFoldTree = 256; // leaves of the moment tree of the fold (column tiles wrap onto them)
struct FbaqStatsSmem {
    int off[kFbaqStatsLines + 1];  // SWST shift of the tile's lines (and the line before)
    int len[kFbaqStatsLines + 1];  // usable block-data bytes of those records
    double red[kFbaqStatsWarps][kFbaqSums][32];
};

// One column over lines [wy0, wy1) of records that hold its sample at code byte j of the block data,
// block id at 64 b: the moments and lag sums, the pair (wy0 - 1, wy0) included when wy0 > 0.
ASARF_HD ASARF_INLINE void fbaq_column(const RawStatsArgs& a, int b, int j, int wy0, int wy1, double v[kFbaqSums]) {
    const uint8_t* base = a.raw + 2;
    auto bytes = [&](int y, int& id, int& cw) {
        const uint8_t* rec = base + static_cast<long long>(y) * a.line_bytes;
        id = ASARF_LDG(rec + 64 * b);
        cw = ASARF_LDG(rec + j);
    };
    auto value = [&](int id, int cw, double& i, double& q) {
        i = ASARF_LDG(a.lut_i + 16 * id + (cw >> 4));
        q = ASARF_LDG(a.lut_q + 16 * id + (cw & 15));
    };
    double pi = 0.0, pq = 0.0, fi = 0.0, fq = 0.0;  // previous sample; the first one, when it ends no pair
    double si = 0.0, sq = 0.0, sii = 0.0, sqq = 0.0, siq = 0.0, lac = 0.0, lbd = 0.0, lad = 0.0, lbc = 0.0;
    auto add = [&](double ci, double cq) {
        si += ci;
        sq += cq;
        sii += ci * ci;
        sqq += cq * cq;
        siq += ci * cq;
        lac += pi * ci;
        lbd += pq * cq;
        lad += pi * cq;
        lbc += pq * ci;
        pi = ci;
        pq = cq;
    };
    int id[kStatsBatch], cw[kStatsBatch], y = wy0;
    if (wy0 > 0) {
        bytes(wy0 - 1, id[0], cw[0]);
        value(id[0], cw[0], pi, pq);
    } else {  // line 0: no pair (its products with the zero predecessor vanish)
        bytes(0, id[0], cw[0]);
        value(id[0], cw[0], fi, fq);
        add(fi, fq);
        y = 1;
    }
    const double ai = wy0 > 0 ? pi : fi, aq = wy0 > 0 ? pq : fq;  // first sample of the first pair
    const double bi = wy0 > 0 ? 0.0 : fi, bq = wy0 > 0 ? 0.0 : fq;
    if (y + kStatsBatch <= wy1) {
#pragma unroll
        for (int u = 0; u < kStatsBatch; ++u) bytes(y + u, id[u], cw[u]);
    }
    for (; y + kStatsBatch <= wy1; y += kStatsBatch) {
        constexpr int kHalf = kStatsBatch / 2;
        double ci[kHalf], cq[kHalf];
#pragma unroll
        for (int u = 0; u < kHalf; ++u) value(id[u], cw[u], ci[u], cq[u]);
#pragma unroll
        for (int u = 0; u < kHalf; ++u) add(ci[u], cq[u]);
#pragma unroll
        for (int u = 0; u < kHalf; ++u) value(id[kHalf + u], cw[kHalf + u], ci[u], cq[u]);
        if (y + 2 * kStatsBatch <= wy1) {
#pragma unroll
            for (int u = 0; u < kStatsBatch; ++u) bytes(y + kStatsBatch + u, id[u], cw[u]);
        }
#pragma unroll
        for (int u = 0; u < kHalf; ++u) add(ci[u], cq[u]);
    }
    for (; y < wy1; ++y) {
        double ci, cq;
        bytes(y, id[0], cw[0]);
        value(id[0], cw[0], ci, cq);
        add(ci, cq);
    }
    const int n = wy1 - wy0, np = wy0 > 0 ? n : n - 1;
    v[0] = n, v[1] = si, v[2] = sq, v[3] = sii, v[4] = sqq, v[5] = siq;
    // over the pairs: second samples are all but an unpaired first one, first samples those less the
    // last plus the one before the range
    const double c = si - bi, d = sq - bq;
    v[6] = np, v[7] = np ? c - pi + ai : 0.0, v[8] = np ? d - pq + aq : 0.0, v[9] = np ? c : 0.0, v[10] = np ? d : 0.0;
    v[11] = lac, v[12] = lbd, v[13] = lad, v[14] = lbc;
}

// The same for records of any shift and length: lane sums of column x straight to red[k][lane].
#if defined(__CUDA_ARCH__)
static __device__ __noinline__
#else
static inline
#endif
void fbaq_column_masked(const RawStatsArgs& a, const FbaqStatsSmem* sm, int x, int ys, int wy0, int wy1,
                        double (*red)[32], int lane) {
    const FastDiv d63 = make_fastdiv(63u);
    double v[kFbaqSums];
    for (int k = 0; k < kFbaqSums; ++k) v[k] = 0.0;
    double pi = 0.0, pq = 0.0;
    bool pf = false;
    for (int y = wy0 > 0 ? wy0 - 1 : 0; y < wy1; ++y) {
        const int r = x - sm->off[y - ys];
        const int b = r > 0 ? static_cast<int>(fdiv_u(static_cast<unsigned int>(r), d63)) : 0;
        const int j = r + b + 1;
        const bool f = r >= 0 && j < sm->len[y - ys];
        double ci = 0.0, cq = 0.0;
        if (f) {
            const uint8_t* rec = a.raw + static_cast<long long>(y) * a.line_bytes + 2;
            const int id = rec[64 * b], cw = rec[j];
            ci = ASARF_LDG(a.lut_i + 16 * id + (cw >> 4));
            cq = ASARF_LDG(a.lut_q + 16 * id + (cw & 15));
        }
        if (y >= wy0 && f) {
            v[0] += 1.0;
            v[1] += ci;
            v[2] += cq;
            v[3] += ci * ci;
            v[4] += cq * cq;
            v[5] += ci * cq;
            if (y > 0 && pf) {
                v[6] += 1.0;
                v[7] += pi;
                v[8] += pq;
                v[9] += ci;
                v[10] += cq;
                v[11] += pi * ci;
                v[12] += pq * cq;
                v[13] += pi * cq;
                v[14] += pq * ci;
            }
        }
        pi = ci;
        pq = cq;
        pf = f;
    }
    for (int k = 0; k < kFbaqSums; ++k) red[k][lane] = v[k];
}

// Lines of tile row by with one shift and length: those of its first line in (*off, *len).
ASARF_HD ASARF_INLINE bool fbaq_line_like(const RawStatsArgs& a, int y, int off, int len) {
    return (a.swst ? static_cast<int>(a.swst[y]) - a.min_swst : 0) == off &&
           fbaq_len(a.raw + static_cast<long long>(y) * a.line_bytes, a.line_bytes) == len;
}
ASARF_HD ASARF_INLINE int fbaq_tile_start(int by) { return by > 0 ? by * kFbaqStatsLines - 1 : 0; }

ASARF_HD ASARF_INLINE void raw_stats_fbaq_body(const RawStatsArgs& a, int bx, int by, int tid, int nthr,
                                               FbaqStatsSmem* sm) {
    const int y0 = by * kFbaqStatsLines;
    const int y1 = (y0 + kFbaqStatsLines < a.na) ? y0 + kFbaqStatsLines : a.na;
    const int ys = fbaq_tile_start(by);
    const bool same = a.uniform[by] != 0;
    const int off0 = a.swst ? static_cast<int>(a.swst[ys]) - a.min_swst : 0;
    const int len0 = fbaq_len(a.raw + static_cast<long long>(ys) * a.line_bytes, a.line_bytes);
    if (!same) {
        for (int y = ys + tid; y < y1; y += nthr) {
            sm->off[y - ys] = a.swst ? static_cast<int>(a.swst[y]) - a.min_swst : 0;
            sm->len[y - ys] = fbaq_len(a.raw + static_cast<long long>(y) * a.line_bytes, a.line_bytes);
        }
        ASARF_SYNC();
    }
    constexpr int sub = kFbaqStatsLines / kFbaqStatsWarps;
    for (int t = tid; t < 32 * kFbaqStatsWarps; t += nthr) {
        const int lane = t & 31, w = t >> 5;
        const int x = bx * 32 + lane;
        const int wy0 = y0 + w * sub;
        const int wy1 = (wy0 + sub < y1) ? wy0 + sub : y1;
        const bool any = x < a.nr && wy0 < wy1;
        if (any && !same) {
            fbaq_column_masked(a, sm, x, ys, wy0, wy1, sm->red[w], lane);
            continue;
        }
        double v[kFbaqSums];
#pragma unroll
        for (int k = 0; k < kFbaqSums; ++k) v[k] = 0.0;
        const int r = x - off0;
        const int b = r >= 0 ? r / 63 : 0;
        if (any && r >= 0 && r + b + 1 < len0) fbaq_column(a, b, r + b + 1, wy0, wy1, v);
#pragma unroll
        for (int k = 0; k < kFbaqSums; ++k) sm->red[w][k][lane] = v[k];
    }
    ASARF_SYNC();
    // over the warps, in warp order (into warp 0's row)
    for (int t = tid; t < kFbaqSums * 32; t += nthr) {
        const int k = t >> 5, lane = t & 31;
        double acc = sm->red[0][k][lane];
        for (int w = 1; w < kFbaqStatsWarps; ++w) acc += sm->red[w][k][lane];
        sm->red[0][k][lane] = acc;
    }
    ASARF_SYNC();
    double* out = a.part + (static_cast<long long>(by) * a.tiles_x + bx) * a.part_slots;
    const int b0 = static_cast<int>((bx * 32) / a.dc_step);
    // lag sums: per Doppler block, lanes in order (before the moment tree reuses the row)
    for (int t = tid; t < 9 * a.span; t += nthr) {
        const int bl = t / 9, q = t - bl * 9;
        double acc = 0.0;
        for (int lane = 0; lane < 32; ++lane) {
            const int x = bx * 32 + lane;
            if (x < a.nr && x / a.dc_step == b0 + bl) acc += sm->red[0][6 + q][lane];
        }
        out[6 + t] = acc;
    }
    ASARF_SYNC();
    // moments: pairwise tree over the 32 lanes
    for (int h = 16; h > 0; h >>= 1) {
        for (int t = tid; t < 6 * h; t += nthr) {
            const int k = t / h, lane = t - k * h;
            sm->red[0][k][lane] += sm->red[0][k][lane + h];
        }
        ASARF_SYNC();
    }
    for (int k = tid; k < 6; k += nthr) out[k] = sm->red[0][k][0];
}

// Fold of the FBAQ4 partials into FloatStatAccum: over the line tiles of every
// column tile, then over the column tiles touching each sum, both in index order.
ASARF_HD ASARF_INLINE void stats_fold_body(const RawStatsArgs& a, int tiles_y, int tid, int nthr, double* tree) {
    const int slots = a.part_slots;
    for (int t = tid; t < a.tiles_x * slots; t += nthr) {
        double acc = a.part[t];
        for (int by = 1; by < tiles_y; ++by) acc += a.part[static_cast<long long>(by) * a.tiles_x * slots + t];
        a.part[t] = acc;
    }
    ASARF_SYNC();
    // moments: pairwise tree over the column tiles (tree holds 6 x kFoldTree doubles)
    for (int t = tid; t < 6 * kFoldTree; t += nthr) {
        const int m = t / kFoldTree, bx = t - m * kFoldTree;
        double acc = 0.0;
        for (int k = bx; k < a.tiles_x; k += kFoldTree) acc += a.part[k * slots + m];
        tree[t] = acc;
    }
    ASARF_SYNC();
    for (int h = kFoldTree / 2; h > 0; h >>= 1) {
        for (int t = tid; t < 6 * h; t += nthr) {
            const int m = t / h, i = t - m * h;
            tree[m * kFoldTree + i] += tree[m * kFoldTree + i + h];
        }
        ASARF_SYNC();
    }
    for (int t = tid; t < 6; t += nthr) a.facc->mom[t] = tree[t * kFoldTree];
    // lag sums: the few column tiles touching each Doppler block, in order
    for (int t = tid; t < 9 * a.nblk; t += nthr) {
        const int b = t / 9, q = t - 9 * b;
        const int lo = (b * a.dc_step) / 32;
        int hi = ((b + 1) * a.dc_step - 1) / 32;
        if (hi > a.tiles_x - 1) hi = a.tiles_x - 1;
        double acc = 0.0;
        for (int bx = lo; bx <= hi; ++bx) {
            const int bl = b - (bx * 32) / a.dc_step;
            if (bl >= 0 && bl < a.span) acc += a.part[bx * slots + 6 + 9 * bl + q];
        }
        a.facc->lag[b][q] = acc;
    }
}

// ----------------------------------------------------------------------------- finalisation
// IQ statistics and correction constants exactly as RawDataCorrection
// derives them (sar/iq_correction.cu:200-273, CalcMean/CalcStdDev of
// cuda_util/device_padded_image.cu:331-414), the Doppler centroid per range block and its
// quadratic fit (sar/fractional_doppler_centroid.cu:98-139), and the results-window choice
// that depends on the sign of the fitted constant term (main_flow.cc:155-178).
// Constants of the corrected-sample map z = (p*I + p0, u*Q + v*I + w) and the statistics
// error bits, shared by the IQ part and the per-block Doppler part of the finalisation.
struct FinalizeMap {
    double p, p0, u, v, w, pad_mag2;
    unsigned int err;
};

// IQ statistics and the correction constants; the FocusState fields are written when st is set.
ASARF_HD inline FinalizeMap finalize_stats(const FinalizeArgs& a, FocusState* st) {
    const StatAccum& s = *a.acc;
    const FloatStatAccum* fs = a.facc;
    auto mom = [&](int k) { return fs ? fs->mom[k] : static_cast<double>(s.mom[k]); };
    const double n = mom(0);
    const double SI = mom(1), SQ = mom(2);
    const double SII = mom(3), SQQ = mom(4);
    const double SIQ = mom(5);
    FinalizeMap m;
    m.err = 0;
    if (n == 0.0) m.err |= kErrStatsEmpty;
    if (!a.facc) m.err |= a.acc->errors;
    const float total = static_cast<float>(a.n_total);
    // mean: float(sum) / float(total)
    const float dc_i = static_cast<float>(SI) / total;
    const float dc_q = static_cast<float>(SQ) / total;
    const double di = dc_i, dq = dc_q;
    // sums over filled of (I - dc_i)^2, (Q - dc_q)^2: a dead channel's may round to just below zero
    auto centred = [&](double s2, double s1, double d) {
        const double c = s2 - 2.0 * d * s1 + n * d * d;
        return c < 0.0 ? 0.0 : c;
    };
    const double cii = centred(SII, SI, di);
    const double cqq = centred(SQQ, SQ, dq);
    const double ciq = SIQ - dq * SI - di * SQ + n * di * dq;
    // padding samples hold 0 - dc after the DC step and enter the gain / phase sums
    const double npad = static_cast<double>(a.n_pad);
    const double i1sq = cii + npad * di * di;
    const double q1sq = cqq + npad * dq * dq;
    const double i1q1 = ciq + npad * di * dq;
    const double gain = sqrt(i1sq / q1sq);
    const float gain_f = static_cast<float>(gain);
    const double gf = gain_f;
    const double delta = (i1q1 / gf) / (i1sq / (gf * gf));
    const float sin_c = static_cast<float>(delta);
    const float cos_c = static_cast<float>(1.0 - delta * delta);
    if (st) {
        st->dc_i = dc_i;
        st->dc_q = dc_q;
        st->gain = gain_f;
        st->sin_c = sin_c;
        st->cos_c = cos_c;
        st->rgain = fdiv_rn(1.0f, gain_f);
        st->rcos = fdiv_rn(1.0f, cos_c);
        st->dc_i_d = dc_i;
        st->dc_q_d = dc_q;
        st->iq_gain = gain;
        st->phase_error = 360.0 * asin(delta) / (2.0 * 3.14159265358979323846);
        st->stddev_i = sqrtf(static_cast<float>(cii) / total);
        st->stddev_q = sqrtf(static_cast<float>(cqq) / total);
    }
    // corrected sample z = (p*I + p0, u*Q + v*I + w)
    m.p = 1.0 / gf;
    m.p0 = -di / gf;
    const double sc = sin_c, cc = cos_c;
    m.u = 1.0 / cc;
    m.v = -sc * m.p / cc;
    m.w = (-dq - sc * m.p0) / cc;
    m.pad_mag2 = m.p0 * m.p0 + m.w * m.w;  // |corrected zero padding sample|^2
    return m;
}

// Doppler centroid of range block b from its lag-1 sums through the correction map.
ASARF_HD inline void finalize_block(const FinalizeArgs& a, const FinalizeMap& m, int b, double* xs, double* ys,
                                    FocusState& st) {
    const StatAccum& s = *a.acc;
    const FloatStatAccum* fs = a.facc;
    auto lag = [&](int q) { return fs ? fs->lag[b][q] : static_cast<double>(s.lag[b][q]); };
    const double p = m.p, p0 = m.p0, u = m.u, v = m.v, w = m.w;
    const double np = lag(0);
    const double sA = lag(1), sB = lag(2);
    const double sC = lag(3), sD = lag(4);
    const double sAC = lag(5), sBD = lag(6);
    const double sAD = lag(7), sBC = lag(8);
    double re = p * p * sAC + p * p0 * (sA + sC) + p0 * p0 * np + u * u * sBD + u * v * (sBC + sAD) +
                u * w * (sB + sD) + v * v * sAC + v * w * (sA + sC) + w * w * np;
    const double im = p * u * (sAD - sBC) + p * w * (sA - sC) + p0 * u * (sD - sB) + p0 * v * (sC - sA);
    const int xb = b * a.dc_step;
    const int xe = xb + a.dc_step;
    // columns of this block beyond the data lie in the range padding (constant rows)
    int pad_lo = xb > a.nr ? xb : a.nr;
    int pad_hi = xe < a.rg_stride ? xe : a.rg_stride;
    // (only when the padding went through the correction, i.e. reference statistics)
    if (a.n_pad > 0 && pad_hi > pad_lo) re += static_cast<double>(pad_hi - pad_lo) * (a.na - 1) * m.pad_mag2;
    const double ang = atan2(im, re);
    const double hz = a.prf * (ang / (2.0 * 3.14159265358979323846));
    xs[b] = static_cast<double>((xb + xe) / 2);
    ys[b] = hz;
    st.dc_blk_hz[b] = hz;
}

// The fitted Doppler polynomial (or the caller's), the DC-sign variant and the error bits.
ASARF_HD inline void finalize_poly(const FinalizeArgs& a, FocusState& st, double poly[3], unsigned int err) {
    if (a.nblk > kMaxDcBlocks) err |= kErrDcBlocks;
    st.nblk = a.nblk < kMaxDcBlocks ? a.nblk : kMaxDcBlocks;
    for (int k = 0; k < 3; ++k) st.dc_est[k] = poly[k];
    if (a.dc_given)
        for (int k = 0; k < 3; ++k) poly[k] = a.dc_in[k];
    for (int k = 0; k < 3; ++k) {
        st.dc_poly[k] = poly[k];
        st.dc_poly32[k] = static_cast<float>(poly[k]);
    }
    st.variant = poly[2] > 0 ? 0 : 1;
    st.first_line = a.first_line[st.variant];
    st.n_lines = a.n_lines[st.variant];
    st.errors = err;
}

// The whole finalisation on one thread.
ASARF_HD inline void finalize_body(const FinalizeArgs& a) {
    FocusState& st = *a.state;
    const FinalizeMap m = finalize_stats(a, &st);
    double xs[kMaxDcBlocks], ys[kMaxDcBlocks];
    const int nblk = a.nblk < kMaxDcBlocks ? a.nblk : kMaxDcBlocks;
    for (int b = 0; b < nblk; ++b) finalize_block(a, m, b, xs, ys, st);
    double poly[3] = {0.0, 0.0, 0.0};
    polyfit_qr<kMaxDcBlocks, 3>(xs, ys, nblk, 2, poly);
    finalize_poly(a, st, poly, m.err);
}

// ----------------------------------------------------------------------------- range compression
// One azimuth line per block: ERS byte decode (envisat_format/src/envisat_format_kernels.cu:116-134),
// IQ correction with the reference's float operation order (sar/iq_correction.cu:140-178),
// forward FFT, chirp matched filter and inverse FFT (sar/range_compression.cu:25-107), keeping
// x < XSize - chirp_samples.  Samples the decoder leaves empty are 0 (ZeroNaNs after the
// correction, main.cc:245).  The FFT length is any L >= XSize: outputs x < Nk only correlate
// data samples [x, x + Nc) so they do not depend on L.
// The IQ correction constants of a run, copied out of the FocusState into registers before a
// line's decode loop (read through the state's pointer, they were reloaded for every sample:
// range compression 1.066 -> 0.996 ms on the ERS scene).
struct IqCorr {
    float dc_i, dc_q, gain, rgain, sin_c, cos_c, rcos;
    ASARF_HD ASARF_INLINE explicit IqCorr(const FocusState& s)
        : dc_i(s.dc_i), dc_q(s.dc_q), gain(s.gain), rgain(s.rgain), sin_c(s.sin_c), cos_c(s.cos_c), rcos(s.rcos) {}
};

ASARF_HD ASARF_INLINE float2 correct_sample_f(float iv, float qv, const IqCorr& st) {
    const float i1 = fsub_rn(iv, st.dc_i);
    const float q1 = fsub_rn(qv, st.dc_q);
    // the reference's two IEEE divisions, correctly rounded through the reciprocals
    const float i2 = div_by_recip_rn(i1, st.gain, st.rgain);
    const float q2 = div_by_recip_rn(fma_rn(-i2, st.sin_c, q1), st.cos_c, st.rcos);
    return make_float2(i2, q2);
}

ASARF_HD ASARF_INLINE float2 correct_sample(int iv, int qv, const IqCorr& st) {
    return correct_sample_f(static_cast<float>(iv), static_cast<float>(qv), st);
}

// Corrected sample at range position l of line y (FMT: RawFormat; row: the line's record).
template <int FMT>
struct LineDecoder {
    int off, len;
    FastDiv d63;
    const uint8_t* row;
    ASARF_HD ASARF_INLINE LineDecoder(const RangeCompressArgs& a, int y, const uint8_t* raw_line) {
        row = raw_line ? raw_line : a.raw + static_cast<long long>(y) * a.line_bytes;
        if constexpr (FMT == kRawAsarFbaq4) {
            off = a.swst ? static_cast<int>(a.swst[y]) - a.min_swst : 0;
            len = fbaq_len(row, a.line_bytes);
            d63 = make_fastdiv(63u);
        } else {
            off = a.swst ? 4 * (static_cast<int>(a.swst[y]) - a.min_swst) : 0;
            len = 0;
        }
    }
    ASARF_HD ASARF_INLINE float2 operator()(const RangeCompressArgs& a, const IqCorr& st, int l) const {
        float2 z = make_float2(0.0f, 0.0f);
        const int i = l - off;
        if constexpr (FMT == kRawAsarFbaq4) {
            float iv, qv;
            if (l < a.nr && i >= 0 && fbaq_sample(row, len, i, d63, a.lut_i, a.lut_q, &iv, &qv))
                z = correct_sample_f(iv, qv, st);
        } else {
            if (l < a.nr && i >= 0 && i < a.spl) {
                const uint16_t wv = *reinterpret_cast<const uint16_t*>(row + 2ll * i);
                z = correct_sample(wv & 0xff, wv >> 8, st);
            }
        }
        return z;
    }
};

template <int FMT = kRawErsBytes>
ASARF_HD ASARF_INLINE void range_compress_body(const RangeCompressArgs& a, int y, int tid, int nthr, float2* s,
                                               const uint8_t* raw_line) {
    const IqCorr st(*a.state);
    const int L = a.plan.n;
    const LineDecoder<FMT> dec(a, y, raw_line);
    for (int l = tid; l < L; l += nthr) s[l] = dec(a, st, l);
    ASARF_SYNC();
    fft_forward(a.plan, s, 1, 1, tid, nthr);
    for (int l = tid; l < L; l += nthr) s[l] = cmul(s[l], ASARF_LDG(a.mf + l));
    ASARF_SYNC();
    fft_inverse(a.plan, s, 1, 1, tid, nthr);
    float2* orow = a.out + static_cast<long long>(y) * a.out_pitch;
    for (int l = tid; l < a.nk; l += nthr) orow[l] = s[l];
}

// Compressed line store of the compile-time transform: sample x < nk to orow[x].
struct RcOut {
    static constexpr bool kActive = true;
    float2* orow;
    int nk;
    ASARF_HD ASARF_INLINE void operator()(int x, float2 v) const {
        if (x < nk) orow[x] = v;
    }
};

// Corrected samples of a raw line.
template <int FMT>
struct RcSource {
    static constexpr bool kActive = true;
    const RangeCompressArgs& a;
    const IqCorr st;
    const LineDecoder<FMT> dec;
    ASARF_HD ASARF_INLINE RcSource(const RangeCompressArgs& args, const FocusState& fs, int y, const uint8_t* raw_line)
        : a(args), st(fs), dec(args, y, raw_line) {}
    ASARF_HD ASARF_INLINE float2 operator()(int l) const { return dec(a, st, l); }
};

// Same transform with a compile-time schedule (lengths in kCtLengths): all loops unrolled,
// all index arithmetic constant.
template <int L, int FMT = kRawErsBytes>
ASARF_HD ASARF_INLINE void range_compress_ct_body(const RangeCompressArgs& a, int y, int tid, float2* s,
                                                  const uint8_t* raw_line) {
    // the first pass decodes the samples it transforms, the last inverse pass stores the kept ones
    ct_fft_mf_ifft<L>(s, a.ctw, a.mf, tid, RcSource<FMT>{a, *a.state, y, raw_line},
                      RcOut{a.out + static_cast<long long>(y) * a.out_pitch, a.nk});
}

// ----------------------------------------------------------------------------- azimuth strided pass
// Four-step azimuth FFT of length N = n1 * n2 along the rows of a [N][pitch] block, columns
// [x0, x0 + xt).  Time index n = a*n2 + b, frequency k = k1 + n1*k2.
//  forward (block b): Y[k1][b] = W_N^{b k1} * FFT_n1(x[a*n2 + b])[k1], stored at row k1*n2 + b.
//  inverse (block b): x[a*n2 + b] = IFFT_n1(conj(W_N^{b k1}) * Z[k1][b])[a] * scale.
// Both read their rows in natural order (one strided tile, TMA-loaded on the device) and
// write the digit-reversed transform output straight to its destination rows.
// Together with the contiguous pass this is the transpose-free equivalent of the reference's
// transpose + batched row FFT + transpose (sar/range_doppler_algorithm.cu:314-326, 381-391).
// A block takes NB adjacent b: their tiles lie side by side as one [n1][NB * XT] tile (one TMA
// box), so that short lengths n1 still give a block's threads and its loads enough to do.
// Per-block tables, staged in shared memory while the tile is in flight: tw[k * n1 + p] =
// W_N^{(b + k) k1} and row[p] = destination row of b, for transform position p (forward:
// k1 = drev1(p), digit-reversed output; inverse: tw indexed by the natural input row k1 = p,
// row by the digit-reversed output position).  b * k1 < N, so no reduction is needed.
ASARF_HD ASARF_INLINE void az_strided_tables(const AzStridedArgs& a, int b, int tid, int nthr, float2* tw, int* row) {
    for (int p = tid; p < a.n1; p += nthr) {
        const int kd = ASARF_LDG(a.drev1 + p);
        for (int k = 0; k < a.nb; ++k)
            if (b + k < a.n2) tw[k * a.n1 + p] = ASARF_LDG(a.twn + (b + k) * (a.inverse ? p : kd));
        row[p] = kd * a.n2 + b;
    }
}

// Tiles of a block: as many as keep n1 * nb at 256 rows of 32 columns (64 KB, three blocks per SM)
// while the grid still has three blocks per SM (5000 lines of 4913 columns, n1 = 40: 147 us forward
// with one, 81 with four; n1 = 225 takes one).
inline int az_strided_tiles_per_block(int n1, int n2, int tiles) {
    int nb = 1;
    while (nb < 8 && 2 * nb * n1 <= 256 && static_cast<long long>(tiles) * (n2 / (2 * nb)) >= 3 * 148) nb *= 2;
    return nb;
}

// XT: the tile width (16 or 32), NB tiles.  R0, R1, R2 > 0: the transform's radix schedule as
// compile-time constants (it must be the plan's: the planner picks this instantiation only when it
// is).  b: the first tile's.
template <int R0, int R1, int R2, int XT, int NB>
ASARF_HD ASARF_INLINE void az_strided_body(const AzStridedArgs& a, int tile, int b, int tid, int nthr, float2* s,
                                           const float2* tw, const int* rowmap, bool preloaded) {
    constexpr int LDC = XT * NB, PAIRS = XT / 2, NPAIR = LDC / 2;
    const int n1 = R0 > 0 ? R0 * R1 * R2 : a.n1;
    const int x0 = tile * XT;
    // tile [r][k][c] = row r*n2 + b + k, column x0 + c (natural order; columns >= nk read as 0)
    if (!preloaded) {
        for (int t = tid; t < n1 * LDC; t += nthr) {
            const int r = t / LDC, k = t % LDC / XT;
            const int row = r * a.n2 + b + k;
            const int x = x0 + t % XT;
            float2 v = make_float2(0.0f, 0.0f);
            if (b + k < a.n2 && row < a.valid_rows && x < a.nk) v = a.in[static_cast<long long>(row) * a.pitch + x];
            s[t] = v;
        }
        ASARF_SYNC();
    } else if (a.valid_rows < n1 * a.n2) {
        // rows past the data hold stale values in memory: they are zero by definition
        const int r0 = a.valid_rows > b + NB - 1 ? (a.valid_rows - (b + NB - 1) + a.n2 - 1) / a.n2 : 0;
        for (int t = r0 * LDC + tid; t < n1 * LDC; t += nthr)
            if (t / LDC * a.n2 + b + t % LDC / XT >= a.valid_rows) s[t] = make_float2(0.0f, 0.0f);
        ASARF_SYNC();
    }
    if (!a.inverse) {
        // (writing the last stage straight to HBM, as the range-Doppler block does, measured
        // slower here: its rows scatter through the digit-reversed row map)
        if constexpr (R0 > 0)
            fft_forward_pairs_ct3<R0, R1, R2, NPAIR, LDC, true>(s, a.plan1.tw, tid, nthr);
        else
            fft_forward_pairs_xt<NPAIR, LDC>(a.plan1, s, tid, nthr);
        const bool aligned = (a.pitch & 1) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
        for (int t = tid; t < n1 * NPAIR; t += nthr) {
            const int p = t / NPAIR, k = t % NPAIR / PAIRS;
            const int x = x0 + 2 * (t % PAIRS);
            if (b + k >= a.n2 || x >= a.nk) continue;
            const float4 v = *reinterpret_cast<const float4*>(s + 2 * t);
            const float2 w = tw[k * n1 + p];
            const float2 u0 = cmul(make_float2(v.x, v.y), w), u1 = cmul(make_float2(v.z, v.w), w);
            float2* dst = a.out + static_cast<long long>(rowmap[p] + k) * a.pitch + x;
            if (aligned && x + 1 < a.nk) {
                *reinterpret_cast<float4*>(dst) = make_float4(u0.x, u0.y, u1.x, u1.y);
            } else {
                dst[0] = u0;
                if (x + 1 < a.nk) dst[1] = u1;
            }
        }
    } else {
        // conj(twiddle) of row k1 applied as the first stage loads the row
        if constexpr (R0 > 0)
            fft_inverse_dif_pairs_ct3<R0, R1, R2, PAIRS, NPAIR, LDC, true>(s, a.plan1.tw, tid, nthr, tw);
        else
            fft_inverse_dif_pairs_xt<PAIRS, NPAIR, LDC>(a.plan1, s, tid, nthr, tw);
        const int lo = a.state ? a.state->first_line : 0;
        const int hi = a.state ? lo + a.state->n_lines : n1 * a.n2;
        const bool aligned = (a.pitch & 1) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 &&
                             (reinterpret_cast<uintptr_t>(a.out_intensity) & 7) == 0;
        for (int t = tid; t < n1 * NPAIR; t += nthr) {
            const int p = t / NPAIR, k = t % NPAIR / PAIRS;
            const int x = x0 + 2 * (t % PAIRS);
            const int row = rowmap[p] + k;
            if (b + k >= a.n2 || x >= a.nk || row < lo || row >= hi) continue;
            const float4 v = *reinterpret_cast<const float4*>(s + 2 * t);
            const float2 u0 = make_float2(fmul_rn(v.x, a.scale), fmul_rn(v.y, a.scale));
            const float2 u1 = make_float2(fmul_rn(v.z, a.scale), fmul_rn(v.w, a.scale));
            const long long o = static_cast<long long>(row - a.out_row0) * a.pitch + x;
            if (a.out_intensity) {
                // the tail's |z|^2, same rounding
                const float i0 = fma_rn(u0.x, u0.x, fmul_rn(u0.y, u0.y)), i1 = fma_rn(u1.x, u1.x, fmul_rn(u1.y, u1.y));
                if (aligned && x + 1 < a.nk) {
                    *reinterpret_cast<float2*>(a.out_intensity + o) = make_float2(i0, i1);
                } else {
                    a.out_intensity[o] = i0;
                    if (x + 1 < a.nk) a.out_intensity[o + 1] = i1;
                }
            } else if (aligned && x + 1 < a.nk) {
                *reinterpret_cast<float4*>(a.out + o) = make_float4(u0.x, u0.y, u1.x, u1.y);
            } else {
                a.out[o] = u0;
                if (x + 1 < a.nk) a.out[o + 1] = u1;
            }
        }
    }
}

// Shared-memory bytes of the strided pass: tiles, twiddle tables, row table.
inline size_t az_strided_smem(int n1, int xt, int nb) {
    return (sizeof(float2) * static_cast<size_t>(n1) * xt + sizeof(float2) * n1) * nb + sizeof(int) * n1;
}

// ----------------------------------------------------------------------------- range-Doppler block
// Block (tile, k1): rows k1*n2 .. k1*n2 + n2 - 1 of the strided-pass output, output columns
// [x0, x0 + xt) plus a range halo (hl left, hr right) for the interpolator.
//   1. contiguous forward FFT_n2 -> range-Doppler rows, frequency bin k1 + n1*drev2(p);
//   2. RCMC: 16-tap Blackman-windowed sinc at the parabolic range walk
//      (RangeCellMigrationCorrection, sar/range_doppler_algorithm.cu:107-195);
//   3. azimuth matched filter with Doppler-centroid band cut and linear phase ramp
//      (AzimuthReferenceMultiply, sar/range_doppler_algorithm.cu:197-309);
//   4. contiguous inverse FFT_n2 of the xt output columns.
// Both use the reference's float32 operation order for every branch-deciding quantity.
ASARF_HD ASARF_INLINE ColParams az_col_params(const AzRdArgs& a, int x) {
    ColParams cp;
    const float xf = static_cast<float>(x);
    float dcp[3] = {a.state->dc_poly32[0], a.state->dc_poly32[1], a.state->dc_poly32[2]};
    float vrp[3] = {a.vr_poly[0], a.vr_poly[1], a.vr_poly[2]};
    cp.dc = polyval_f32(dcp, xf);
    const float vr = polyval_f32(vrp, xf);
    const float step = a.bin_step;
    const float dc_steps = roundf(fdiv_rn(cp.dc, step));
    cp.dc_off = fmul_rn(dc_steps, step);
    const double r0 = a.slant + static_cast<double>(x) * a.range_spacing;
    cp.r0_dr = r0 / a.range_spacing;
    const float kav = fmul_rn(fmul_rn(2.0f, vr), vr);
    cp.ka = static_cast<float>(static_cast<double>(kav) / (static_cast<double>(a.lambda) * r0));
    const float half = fmul_rn(a.prf, 0.5f);
    cp.cut_hi = fma_rn(half, a.frac, cp.dc_off);
    cp.cut_lo = fma_rn(-half, a.frac, cp.dc_off);
    cp.den = fmul_rn(fmul_rn(8.0f, vr), vr);
    cp.dc_off_ka = fdiv_rn(cp.dc_off, cp.ka);
    cp.rden = fdiv_rn(1.0f, cp.den);
    cp.rka = fdiv_rn(1.0f, cp.ka);
    cp.pad = 0.0f;
    return cp;
}

ASARF_HD ASARF_INLINE float bin_frequency(int f, int az_pad, float step) {
    const int k = (f < az_pad / 2) ? f : f - az_pad;
    return fmul_rn(static_cast<float>(k), step);
}

// Absolute-phase factor of column x: exp(j phi), phi = 4 pi R0 / lambda + pi dc_off^2 / Ka, in
// FP64 (4 pi R0 / lambda is about 1.9e8 rad at 850 km; it is reduced modulo 2 pi before the
// cast).  With it the matched filter is exp(-j pi f^2 / Ka) in the unaliased Doppler
// frequency times the removal of the carrier phase -4 pi R0 / lambda, so a point target keeps
// its own phase.  The reference has neither term (sar/range_doppler_algorithm.cu:265-290).
ASARF_HD ASARF_INLINE float2 az_abs_phase(const AzRdArgs& a, const ColParams& cp, int x) {
    const double kTwoPi = 6.283185307179586476925286766559;
    const double r0 = a.slant + static_cast<double>(x) * a.range_spacing;
    const double d = static_cast<double>(cp.dc_off);
    const double ph = fmod(fmod(2.0 * kTwoPi * r0 / a.lambda_d, kTwoPi) +
                           fmod(0.5 * kTwoPi * d * d / static_cast<double>(cp.ka), kTwoPi), kTwoPi);
    return make_float2(static_cast<float>(cos(ph)), static_cast<float>(sin(ph)));
}

// ---- rows that one range walk and one band decision serve
// A row of the tile is one Doppler bin.  Over its xt <= 64 columns the aliased frequency, the band
// test and the integer walk nearly always agree, and the fraction dl of the walk moves by a
// few 1e-4 (lambda^2 f^2 / 8 Vr^2 samples a column).  For such a row the 14 interpolation weights
// and their derivatives come from a table over the fraction (kRcmcNodes steps, FP64 values
// rounded once): w + (dl - node) w' is one multiply-add where forming a weight took a
// multiply-add, a reciprocal and its share of the normaliser, and a lane takes two adjacent
// columns, whose taps are 15 samples read as eight 16-byte loads instead of 28 8-byte ones.  The
// first neglected term is (dl - node)^2 w'' / 2 < 4.2e-7 at the limit kRcmcMaxStep (w'' <= 3.4,
// the sinc's centre), about 1e-8 over a scene, below the 1e-6 the reference's fraction is rounded
// to.  Every branch-deciding quantity keeps the reference's float32 value: a row is taken as
// uniform only when the extremes over its columns prove that each of them decides alike, and any
// other row goes sample by sample (rcmc_mf_samples).  The block is bound by instruction issue and
// shared-memory wavefronts: on the ERS 5616 x 8990 cut 360 -> 296 million warp instructions, 28000
// lines 1462 -> 1320 us, ASAR IM 30000 lines 1606 -> 1450 us (and 272 million, 1241 and 1415 us since the slow
// rows hold their constants).  (With one column per lane and the
// table's weights summed as sum w d + (dl - node) sum w' d, 345 million instructions and 15 % more
// wavefronts, it took 1537 us; weights read straight from the table 1549 us.)
constexpr int kRcmcNodes = 4096;
constexpr int kRcmcRowFloats = 32;                   // per node: (w, w') of taps 1 .. 14, padded to 128 bytes
constexpr int kRcmcBufFloats = 2 * (kRcmcTaps - 2);  // a warp's copy of one node
constexpr float kRcmcMaxStep = 5e-4f;
constexpr int kRowSlow = -1, kRowSkip = -2;          // other codes: rcmc_row

// Weights of tap i = 1 .. 14 at fraction dl = n / kRcmcNodes - 1/2 and their derivatives, as the
// quotients v_i / sum v of v_i = dl (-1)^i W_i / (dl + 8 - i) (v_8 = W_8: finite at dl = 0).
ASARF_HD inline void rcmc_weight_row(int n, float* row) {
    constexpr float kWin[kRcmcTaps] = ASARF_BLACKMAN16;
    const double dl = static_cast<double>(n) / kRcmcNodes - 0.5;
    double v[kRcmcTaps], dv[kRcmcTaps], sum = 0.0, dsum = 0.0;
    for (int i = 1; i < kRcmcTaps - 1; ++i) {
        const double w = (i & 1) ? -static_cast<double>(kWin[i]) : static_cast<double>(kWin[i]);
        const double m = kRcmcTaps / 2 - i;
        v[i] = m == 0.0 ? w : dl * w / (dl + m);
        dv[i] = m == 0.0 ? 0.0 : w * m / ((dl + m) * (dl + m));
        sum += v[i];
        dsum += dv[i];
    }
    for (int k = 0; k < kRcmcRowFloats; ++k) row[k] = 0.0f;
    for (int i = 1; i < kRcmcTaps - 1; ++i) {
        const double w = v[i] / sum;
        row[2 * (i - 1)] = static_cast<float>(w);
        row[2 * (i - 1) + 1] = static_cast<float>((dv[i] - w * dsum) / sum);
    }
}

// What a sample needs of its column.
struct ColUse {
    float den, rden;      // 8 Vr^2 and its rounded reciprocal
    float r0_hi, r0_lo;   // R0 / range spacing as a float pair
    float dc_off, ka, rka, sh;  // sh = 2 pi (dc_off / Ka), rounded as the reference rounds it
    ASARF_HD ASARF_INLINE void set(const ColParams& c) {
        den = c.den, rden = c.rden;
        r0_hi = static_cast<float>(c.r0_dr);
        r0_lo = static_cast<float>(c.r0_dr - static_cast<double>(r0_hi));
        dc_off = c.dc_off, ka = c.ka, rka = c.rka;
        sh = fmul_rn(fmul_rn(2.0f, 3.14159265358979323846f), c.dc_off_ka);
    }
};

// Extremes over a tile's columns of what the row decisions depend on.
struct RowSpan {
    float dc_min, dc_max, lo_min, lo_max, hi_min, hi_max, off_min, off_max;
    float g_min, g_max;  // walk per lambda^2 f^2, widened by the roundings of both sides
    ASARF_HD ASARF_INLINE void set(const ColParams& c) {
        dc_min = dc_max = c.dc;
        lo_min = lo_max = c.cut_lo;
        hi_min = hi_max = c.cut_hi;
        off_min = off_max = c.dc_off;
        const float g = fmul_rn(static_cast<float>(c.r0_dr), c.rden);
        // quotient, products and casts on either side together round by less than 1e-6
        g_min = fmul_rn(g, 1.0f - 2e-6f);
        g_max = fmul_rn(g, 1.0f + 2e-6f);
    }
    ASARF_HD ASARF_INLINE void join(const RowSpan& o) {
        dc_min = o.dc_min < dc_min ? o.dc_min : dc_min;
        dc_max = o.dc_max > dc_max ? o.dc_max : dc_max;
        lo_min = o.lo_min < lo_min ? o.lo_min : lo_min;
        lo_max = o.lo_max > lo_max ? o.lo_max : lo_max;
        hi_min = o.hi_min < hi_min ? o.hi_min : hi_min;
        hi_max = o.hi_max > hi_max ? o.hi_max : hi_max;
        off_min = o.off_min < off_min ? o.off_min : off_min;
        off_max = o.off_max > off_max ? o.off_max : off_max;
        g_min = o.g_min < g_min ? o.g_min : g_min;
        g_max = o.g_max > g_max ? o.g_max : g_max;
    }
#if defined(__CUDA_ARCH__)
    static __device__ __forceinline__ float warp_min(float v) {
        float r;
        asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
        return r;
    }
    static __device__ __forceinline__ float warp_max(float v) {
        float r;
        asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
        return r;
    }
    __device__ __forceinline__ void join_warp() {
        dc_min = warp_min(dc_min), dc_max = warp_max(dc_max);
        lo_min = warp_min(lo_min), lo_max = warp_max(lo_max);
        hi_min = warp_min(hi_min), hi_max = warp_max(hi_max);
        off_min = warp_min(off_min), off_max = warp_max(off_max);
        g_min = warp_min(g_min), g_max = warp_max(g_max);
    }
#endif
};

// lambda^2 fn^2 as rcmc_mf_sample rounds it.
ASARF_HD ASARF_INLINE float rcmc_numerator(const AzRdArgs& a, float fn) {
    return fmul_rn(fmul_rn(fmul_rn(a.lambda, a.lambda), fn), fn);
}

// Range walk in samples, with the reference's roundings: the quotient num / den, times R0 / range spacing as
// a float pair (the product's rounding differs from the FP64 one's only within 2^-45 of a tie).
ASARF_HD ASARF_INLINE float rcmc_shift(const ColUse& c, float num) {
    const float q = div_by_recip_rn(num, c.den, c.rden);
    const float p = fmul_rn(q, c.r0_hi);
    return fadd_rn(p, fma_rn(q, c.r0_lo, fma_rn(q, c.r0_hi, -p)));
}

// ---- rows that go sample by sample
// What one sample decides for itself.  first: tile column of tap 0 (kNoTaps where the taps leave the line, or
// the tile, which sets the error bit).
struct SampleWalk {
    static constexpr int kNoTaps = -2;
    bool band;  // inside the processed band; outside it the reference writes zero whatever RCMC gave
    int first;
    float dl;   // walk past the integer walk
};

// bf: the row's Doppler bin frequency (bin_frequency of its bin, from the block's row table); cs: the
// sample's tile column.
ASARF_HD ASARF_INLINE SampleWalk rcmc_decide(const AzRdArgs& a, const ColUse& c, float dc, int x, float bf, int cs,
                                             unsigned int* err_flag) {
    const float prf = a.prf;
    const float half = a.half_prf;
    SampleWalk s{false, SampleWalk::kNoTaps, 0.0f};
    // --- aliased frequency (the same test decides the matched-filter band and the RCMC walk)
    float fn = bf;
    if (dc < 0.0f) {
        if (bf > fadd_rn(half, dc)) fn = fsub_rn(fn, prf);
    } else if (dc > 0.0f) {
        if (fn < fadd_rn(-half, dc)) fn = fadd_rn(fn, prf);
    }
    if (fn < fma_rn(-half, a.frac, c.dc_off) || fn > fma_rn(half, a.frac, c.dc_off)) return s;
    s.band = true;
    // --- RCMC: walk = lambda^2 fn^2 / (8 Vr^2) [float, IEEE divide] * R0 / range spacing
    const float shift = rcmc_shift(c, rcmc_numerator(a, fn));
    const int walk = static_cast<int>(roundf(shift));
    const int calc_x = x + walk;
    if (calc_x - kRcmcTaps / 2 < 0 || calc_x + kRcmcTaps / 2 >= a.nk) return s;
    const int first = cs + walk - kRcmcTaps / 2;  // smem column of tap 0
    if (first + 1 < 0 || first + kRcmcTaps - 1 > a.wt) {
        atomic_or_u32(err_flag, kErrRcmcHalo);
        return s;
    }
    // off = shift - walk + 8 in [7.5, 8.5] as the reference rounds it; off - 8 is exact
    const float off = fadd_rn(fsub_rn(shift, static_cast<float>(walk)), static_cast<float>(kRcmcTaps / 2));
    s.dl = fsub_rn(off, static_cast<float>(kRcmcTaps / 2));
    s.first = first;
    return s;
}

// Windowed sinc at off - i, off = shift - walk + 8 in [7.5, 8.5]:
// sin(pi (off - i)) = (-1)^i sin(pi off), and the common factor sin(pi off) / pi
// cancels in the normalised sum, leaving weights (-1)^i W_i / (off - i).  The two end
// taps are skipped: their window values W_0 = W_15 = -1.4e-17 (a numpy.blackman
// rounding residue of an exact zero) give terms below half an ulp of every sum.
// With dl = off - 8 (exact) a weight is 1 / fma(dl, c_i, (8 - i) c_i), c_i = (-1)^i / W_i
// (constants): one FMA and one reciprocal per tap, within 2 ulp of the quotient since
// |8 - i| >= 1 wherever the constant term is not zero.  The normaliser sums in pairs.
struct TapSum {
    float2 acc, nrm2;
    ASARF_HD ASARF_INLINE TapSum() : acc(make_float2(0.0f, 0.0f)), nrm2(acc) {}
    // taps i (odd) and i + 1
    ASARF_HD ASARF_INLINE void add(int i, float dl, float2 u, float2 v) {
        constexpr float kWin[kRcmcTaps] = ASARF_BLACKMAN16;
        const float ca = -1.0f / kWin[i], cb = 1.0f / kWin[i + 1];
        const float wa = rcp_approx(fma_rn(dl, ca, static_cast<float>(kRcmcTaps / 2 - i) * ca));
        const float wb = rcp_approx(fma_rn(dl, cb, static_cast<float>(kRcmcTaps / 2 - i - 1) * cb));
        acc = pfma(u, wa, acc);
        acc = pfma(v, wb, acc);
        nrm2 = padd(nrm2, make_float2(wa, wb));
    }
    // centre: the sample at the integer walk, which a walk without fraction takes (a unit impulse)
    ASARF_HD ASARF_INLINE float2 value(float dl, const float2* centre) const {
        if (dl == 0.0f) return *centre;
        const float nrm = fadd_rn(nrm2.x, nrm2.y);
        if (nrm == 0.0f) return make_float2(0.0f, 0.0f);
        const float inv = rcp_approx(nrm);
        return make_float2(fmul_rn(acc.x, inv), fmul_rn(acc.y, inv));
    }
};

ASARF_HD ASARF_INLINE float2 rcmc_taps(const float2* srow, const SampleWalk& w) {
    if (w.first == SampleWalk::kNoTaps) return make_float2(0.0f, 0.0f);
    const float2* s = srow + w.first;
    TapSum t;
#pragma unroll
    for (int i = 1; i < kRcmcTaps - 1; i += 2) t.add(i, w.dl, s[i], s[i + 1]);
    return t.value(w.dl, s + kRcmcTaps / 2);
}

// The taps of two adjacent samples with one integer walk: 15 columns, read as the 16-byte units from the even
// one at or below the first (ODD: tap 1 is the unit's second sample).
template <bool ODD>
ASARF_HD ASARF_INLINE void rcmc_taps_pair(const float2* srow, const SampleWalk& wa, const SampleWalk& wb, float2* va,
                                          float2* vb) {
    const float4* q = reinterpret_cast<const float4*>(srow + (ODD ? wa.first : wa.first + 1));
    TapSum ta, tb;
    float4 d = q[0];
    float2 lo = ODD ? make_float2(d.z, d.w) : make_float2(d.x, d.y);  // first sample's next tap
#pragma unroll
    for (int i = 1; i < kRcmcTaps - 1; i += 2) {
        float2 mid, hi;
        if (ODD) {
            d = q[i / 2 + 1];
            mid = make_float2(d.x, d.y), hi = make_float2(d.z, d.w);
        } else {
            mid = make_float2(d.z, d.w);
            d = q[i / 2 + 1];
            hi = make_float2(d.x, d.y);
        }
        ta.add(i, wa.dl, lo, mid);
        tb.add(i, wb.dl, mid, hi);
        lo = hi;
    }
    *va = ta.value(wa.dl, srow + wa.first + kRcmcTaps / 2);
    *vb = tb.value(wb.dl, srow + wb.first + kRcmcTaps / 2);
}

// Matched filter exp(-j pi fc^2 / Ka) * exp(-j 2 pi (dc_off / Ka) f), both phases
// rounded as the reference rounds them, combined into one reduced exponential.
ASARF_HD ASARF_INLINE float2 mf_sample(const AzRdArgs& a, const ColUse& c, float bf, const SampleWalk& w, float2 v) {
    if (!w.band) return make_float2(0.0f, 0.0f);
    float fc = fsub_rn(bf, c.dc_off);
    if (fc > a.half_prf) fc = fsub_rn(fc, a.prf);
    else if (fc < -a.half_prf) fc = fadd_rn(fc, a.prf);
    const float mf_phase = div_by_recip_rn(fmul_rn(fmul_rn(3.14159265358979323846f, fc), fc), c.ka, c.rka);
    return cmul(v, expj_neg_sum(mf_phase, fmul_rn(c.sh, bf)));
}

// One sample, and two adjacent ones (columns x, x + 1, of which the first lies inside the line; cs even).
// The columns' constants come from the lane's registers and the centroid table: formed anew for each
// sample (two FP64 and three float divisions, two polynomials) they were most of a slow row.  Adjacent
// samples nearly always share the integer walk, and then their loads: 16-byte units in place of 8-byte ones two
// columns apart.  A third of the rows slow (centroid 1039 Hz, PRF 2080 Hz, 5616 x 9973, n2 = 100): 684 -> 604
// us with the constants held, 593 with the loads shared (a lane per column and no table for any row: 607).
ASARF_HD ASARF_INLINE float2 rcmc_mf_sample(const AzRdArgs& a, const ColUse& c, float dc, int x, float bf,
                                            const float2* srow, int cs, unsigned int* err_flag) {
    const SampleWalk w = rcmc_decide(a, c, dc, x, bf, cs, err_flag);
    return mf_sample(a, c, bf, w, rcmc_taps(srow, w));
}
ASARF_HD ASARF_INLINE void rcmc_mf_samples(const AzRdArgs& a, const ColUse& ca, const ColUse& cb, float2 dc, int x,
                                           float bf, const float2* srow, int cs, unsigned int* err_flag, float2* va,
                                           float2* vb) {
    const SampleWalk wa = rcmc_decide(a, ca, dc.x, x, bf, cs, err_flag);
    SampleWalk wb{false, SampleWalk::kNoTaps, 0.0f};
    if (x + 1 < a.nk) wb = rcmc_decide(a, cb, dc.y, x + 1, bf, cs + 1, err_flag);
    float2 ua, ub;
    if (wa.first != SampleWalk::kNoTaps && wb.first == wa.first + 1) {
        if (wa.first & 1) rcmc_taps_pair<false>(srow, wa, wb, &ua, &ub);
        else rcmc_taps_pair<true>(srow, wa, wb, &ua, &ub);
    } else {
        ua = rcmc_taps(srow, wa);
        ub = rcmc_taps(srow, wb);
    }
    *va = mf_sample(a, ca, bf, wa, ua);
    *vb = mf_sample(a, cb, bf, wb, ub);
}

struct RowRec {
    float bf;   // Doppler bin frequency
    float num;  // uniform rows: lambda^2 fn^2
    int code;   // kRowSlow, kRowSkip or the packed decisions
};

// Record of the row at bin frequency bf.  Code of a uniform row: table node (from bit 12), wrap + 1
// (bits 8-9: the filter's frequency is bf - dc_off - wrap PRF), walk (bits 0-7).  All tests are
// written so that a NaN extreme takes the slow path.  (The device's extremes leave out the columns whose own
// constants are NaN: those columns come out NaN whichever path their rows take.)
ASARF_HD ASARF_INLINE RowRec rcmc_row(const AzRdArgs& a, const RowSpan& sp, float bf) {
    RowRec r{bf, 0.0f, kRowSlow};
    const float half = a.half_prf;
    float fn;
    if (!(sp.dc_min < 0.0f && bf > fadd_rn(half, sp.dc_min)) && !(sp.dc_max > 0.0f && bf < fadd_rn(-half, sp.dc_max)))
        fn = bf;
    else if (sp.dc_max < 0.0f && bf > fadd_rn(half, sp.dc_max)) fn = fsub_rn(bf, a.prf);
    else if (sp.dc_min > 0.0f && bf < fadd_rn(-half, sp.dc_min)) fn = fadd_rn(bf, a.prf);
    else return r;
    if (fn < sp.lo_min || fn > sp.hi_max) {
        r.code = kRowSkip;
        return r;
    }
    if (!(fn >= sp.lo_max && fn <= sp.hi_min)) return r;
    const float fc_max = fsub_rn(bf, sp.off_min), fc_min = fsub_rn(bf, sp.off_max);
    int wrap;
    if (fc_max <= half && fc_min >= -half) wrap = 0;
    else if (fc_min > half) wrap = 1;
    else if (fc_max < -half) wrap = -1;
    else return r;
    // the walk of every column lies in [lo, hi]
    r.num = rcmc_numerator(a, fn);
    const float lo = fmul_rn(r.num, sp.g_min), hi = fmul_rn(r.num, sp.g_max);
    const float mid = fmul_rn(fadd_rn(lo, hi), 0.5f), walk = floorf(fadd_rn(mid, 0.5f));
    if (!(walk >= 0.0f && walk < 256.0f && lo - walk >= -0.5f && hi - walk < 0.5f)) return r;
    int node = static_cast<int>(floorf((mid - walk + 0.5f) * kRcmcNodes + 0.5f));
    node = node < 0 ? 0 : (node > kRcmcNodes ? kRcmcNodes : node);
    const float d0 = fma_rn(static_cast<float>(node), 1.0f / kRcmcNodes, -0.5f);
    if (!(hi - walk - d0 <= kRcmcMaxStep && lo - walk - d0 >= -kRcmcMaxStep)) return r;
    const int w = static_cast<int>(walk);
    // every sample the two columns of a lane read, whole 16-byte units, inside the loaded row
    const int first = a.hl + w - kRcmcTaps / 2;
    if (first < 0 || first + a.xt + kRcmcTaps - 2 > a.wt) return r;
    r.code = node << 12 | (wrap + 1) << 8 | w;
    return r;
}

// Columns of the tile that the taps of its in-band samples reach: up to 6 right of the largest
// integer walk in the band.  The loaded halo holds the walk at |f| = PRF and a margin; the forward
// transform leaves out what no row of this tile reads (ERS: 80 of 82 columns, so that a radix-5 stage's
// 1000 butterfly pairs take 512 threads two rounds, not 1025 three).
ASARF_HD ASARF_INLINE int az_rd_used_columns(const AzRdArgs& a, const RowSpan& sp) {
    const float f = sp.hi_max > -sp.lo_min ? sp.hi_max : -sp.lo_min;  // largest |frequency| in a band
    const float walk = fmul_rn(rcmc_numerator(a, f), sp.g_max);
    const float n = static_cast<float>(a.hl + a.xt + kRcmcTaps / 2 - 2) + floorf(walk + 0.5f);
    if (!(n < static_cast<float>(a.wt))) return a.wt;
    return (static_cast<int>(n) + 1) & ~1;
}

// Shared-memory tables after the tile: the columns' constants (xt) and their extremes (two warps'),
// and in the same memory, once every lane holds its columns' constants, the 16 warps' weight buffers;
// the columns' centroids (xt); absolute-phase factors (xt, only when asked for); the rows' records (n2).
ASARF_HD ASARF_INLINE int az_rd_cols_bytes(int xt) {
    const int cols = static_cast<int>(sizeof(ColUse)) * xt + 2 * static_cast<int>(sizeof(RowSpan)) + 16;
    const int bufs = 16 * kRcmcBufFloats * static_cast<int>(sizeof(float));
    return cols > bufs ? cols : bufs;
}
struct AzRdTables {
    ColUse* cols;
    RowSpan* span;
    int* used;  // az_rd_used_columns
    float* weights;
    float* dc;  // the columns' centroids
    float2* phs;
    RowRec* rows;
    ASARF_HD ASARF_INLINE AzRdTables(const AzRdArgs& a, float2* tile) {
        // the tile is a multiple of 16 bytes (even tile width), and so are the parts before rows
        cols = reinterpret_cast<ColUse*>(tile + static_cast<size_t>(a.n2) * a.wt);
        span = reinterpret_cast<RowSpan*>(cols + a.xt);
        used = reinterpret_cast<int*>(span + 2);
        weights = reinterpret_cast<float*>(cols);
        dc = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(cols) + az_rd_cols_bytes(a.xt));
        phs = reinterpret_cast<float2*>(dc + a.xt);
        rows = reinterpret_cast<RowRec*>(phs + (a.absolute_phase ? a.xt : 0));
    }
};

// Per-block tables of the range-Doppler block, built while the tile is in flight: constants of
// the xt output columns (and their absolute-phase factors when asked for), and for each of the n2
// rows its Doppler bin frequency (bin k1 + n1 drev2(p)) and decisions.
ASARF_HD ASARF_INLINE void az_rd_tables(const AzRdArgs& a, int tile, int k1, int tid, int nthr, const AzRdTables& t) {
    const int x0 = tile * a.xt;
#if defined(__CUDA_ARCH__)
    if (tid < 64) {
        const int c = tid < a.xt ? tid : a.xt - 1;
        const ColParams cp = az_col_params(a, x0 + c);
        if (tid < a.xt) {
            t.cols[c].set(cp);
            t.dc[c] = cp.dc;
            if (a.absolute_phase) t.phs[c] = az_abs_phase(a, cp, x0 + c);
        }
        RowSpan sp;
        sp.set(cp);
        sp.join_warp();
        if ((tid & 31) == 0) t.span[tid >> 5] = sp;
    }
#else
    for (int c = 0; c < a.xt; ++c) {
        const ColParams cp = az_col_params(a, x0 + c);
        t.cols[c].set(cp);
        t.dc[c] = cp.dc;
        if (a.absolute_phase) t.phs[c] = az_abs_phase(a, cp, x0 + c);
        RowSpan o;
        o.set(cp);
        if (c == 0) t.span[0] = t.span[1] = o;
        t.span[0].join(o);
    }
#endif
    ASARF_SYNC();
    RowSpan sp = t.span[0];
    sp.join(t.span[1]);
    if (tid == 0) *t.used = az_rd_used_columns(a, sp);
    for (int p = tid; p < a.n2; p += nthr)
        t.rows[p] = rcmc_row(a, sp, bin_frequency(k1 + a.n1 * ASARF_LDG(a.drev2 + p), a.az_pad, a.bin_step));
}

// Shared-memory bytes of the range-Doppler block.
inline size_t az_rd_smem(int n2, int wt, int xt, bool absolute_phase) {
    return sizeof(float2) * static_cast<size_t>(n2) * wt + static_cast<size_t>(az_rd_cols_bytes(xt)) +
           sizeof(float) * static_cast<size_t>(xt) + sizeof(RowRec) * static_cast<size_t>(n2) +
           (absolute_phase ? sizeof(float2) * static_cast<size_t>(xt) : 0);
}

// Table row of a uniform row's weights.
ASARF_HD ASARF_INLINE const float* rcmc_weights(const AzRdArgs& a, int code) {
    return a.rcmc + static_cast<size_t>(code >> 12) * kRcmcRowFloats;
}

// Interpolated samples of two adjacent columns of a uniform row: q holds the 16-byte units from the
// even tile column at or below tap 1 of the first one (ODD: tap 1 is the unit's second sample), w
// its weights as (w, w', w, w') of taps (1, 2), (3, 4), ..., step the columns' dl - node.
template <bool ODD>
ASARF_HD ASARF_INLINE void rcmc_pair_taps(const float4* q, const float4* w, float2 step, float2* va, float2* vb) {
    float2 acc_a = make_float2(0.0f, 0.0f), acc_b = acc_a;
    float4 d = q[0];
    float2 lo = ODD ? make_float2(d.z, d.w) : make_float2(d.x, d.y);  // first column's next sample
#pragma unroll
    for (int i = 0; i < kRcmcTaps - 2; i += 2) {
        const float4 wv = w[i / 2];
        float2 mid, hi;
        if (ODD) {
            d = q[i / 2 + 1];
            mid = make_float2(d.x, d.y), hi = make_float2(d.z, d.w);
        } else {
            mid = make_float2(d.z, d.w);
            d = q[i / 2 + 1];
            hi = make_float2(d.x, d.y);
        }
        const float2 w0 = pfma2(step, make_float2(wv.y, wv.y), make_float2(wv.x, wv.x));
        const float2 w1 = pfma2(step, make_float2(wv.w, wv.w), make_float2(wv.z, wv.z));
        acc_a = pfma(lo, w0.x, acc_a);
        acc_b = pfma(mid, w0.y, acc_b);
        acc_a = pfma(mid, w1.x, acc_a);
        acc_b = pfma(hi, w1.y, acc_b);
        lo = hi;
    }
    *va = acc_a;
    *vb = acc_b;
}

// Fraction of the range walk past the row's integer walk, plus 8, with the reference's roundings.
ASARF_HD ASARF_INLINE float rcmc_offset(const ColUse& c, float num, float walk) {
    return fadd_rn(fsub_rn(rcmc_shift(c, num), walk), static_cast<float>(kRcmcTaps / 2));
}

// Two adjacent columns x, x + 1 of a uniform row, interpolated and filtered: srow the tile row, c the
// first one's column of the output tile (even).  edge: a column whose taps leave [0, nk) is zero.
ASARF_HD ASARF_INLINE void rcmc_mf_pair(const AzRdArgs& a, const RowRec& r, const float* weights, bool edge,
                                        const ColUse& ca, const ColUse& cb, int x, const float2* srow, int c,
                                        float2* va, float2* vb) {
    const int wk = r.code & 255;
    const float walk = static_cast<float>(wk);
    const float wrap = static_cast<float>(((r.code >> 8) & 3) - 1) * a.prf;
    const float node = fma_rn(static_cast<float>(r.code >> 12), 1.0f / kRcmcNodes, kRcmcTaps / 2 - 0.5f);  // exact
    const float2 step = make_float2(fsub_rn(rcmc_offset(ca, r.num, walk), node),
                                    fsub_rn(rcmc_offset(cb, r.num, walk), node));
    const int tap1 = a.hl + wk - kRcmcTaps / 2 + 1 + c;
    const float4* q = reinterpret_cast<const float4*>(srow + (tap1 & ~1));
    const float4* w = reinterpret_cast<const float4*>(weights);
    float2 v[2];
    if (tap1 & 1) rcmc_pair_taps<true>(q, w, step, &v[0], &v[1]);
    else rcmc_pair_taps<false>(q, w, step, &v[0], &v[1]);
    if (edge) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int cx = x + h + wk;
            if (cx - kRcmcTaps / 2 < 0 || cx + kRcmcTaps / 2 >= a.nk) v[h] = make_float2(0.0f, 0.0f);
        }
    }
    float2* out[2] = {va, vb};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const ColUse& k = h ? cb : ca;
        const float fc = fsub_rn(fsub_rn(r.bf, k.dc_off), wrap);
        const float mf_phase = div_by_recip_rn(fmul_rn(fmul_rn(3.14159265358979323846f, fc), fc), k.ka, k.rka);
        *out[h] = cmul(v[h], expj_neg_sum(mf_phase, fmul_rn(k.sh, r.bf)));
    }
}

// Right range halo of the range-Doppler block: the taps used (1 .. 14 of 16) reach 6 columns
// right of the integer walk, which is at most ceil of the largest walk (the left halo is the
// 8 columns of tap 0, kept whole so that the tile's TMA start stays 16-byte aligned).
inline int rcmc_right_halo(double max_walk) { return kRcmcTaps / 2 - 1 + static_cast<int>(std::ceil(max_walk)); }

// Range-tile width of the range-Doppler block: the widest even width <= 64 whose block leaves
// room for two resident blocks per SM (2 x 512 threads at 64 registers fill the register file;
// 228 KB of shared memory per SM, 1 KB reserved per block).  With one block per SM the
// block-wide barriers of the FFT stages leave the SM idle (measured 2.63 -> 1.92 ms at n2 = 168).
// Where the halo leaves no such width of at least 16, 16; 14 where only that fits a block at all (the row
// records and column tables take up to 3 KB more than the 16 columns they come with leave).
constexpr size_t kAzRdTwoBlockSmem = 228 * 1024 / 2 - 1024 - 128;
inline int az_rd_tile_width(int n2, int hl, int hr, bool absolute_phase, size_t limit) {
    int xt = 64;
    while (xt > 16 && az_rd_smem(n2, xt + hl + hr, xt, absolute_phase) > kAzRdTwoBlockSmem) xt -= 2;
    while (xt > 14 && az_rd_smem(n2, xt + hl + hr, xt, absolute_phase) > limit) xt -= 2;
    return xt;
}

// Blocks the B200 holds at a time (two on each of 148 SMs), and the fewest that a split other than the
// one at sqrt(N) may leave: below that a longer n2 would only idle SMs.
constexpr int kAzRdRound = 2 * 148;
constexpr int kAzRdMinBlocks = 3 * kAzRdRound / 2;

// Epilogue of the range-Doppler block: row r of the inverse transform, column pair cp.
struct AzRdOut {
    static constexpr bool kActive = true;
    float2* out;   // output row 0, column x0
    long long pitch;
    int cols;      // columns of the tile inside the line
    bool aligned;  // every row's pairs lie on 16-byte boundaries
    ASARF_HD ASARF_INLINE AzRdOut(const AzRdArgs& a, int x0, int k1)
        : out(a.out + static_cast<long long>(k1) * a.n2 * a.pitch + x0), pitch(a.pitch), cols(a.nk - x0),
          aligned((a.pitch & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {}
    ASARF_HD ASARF_INLINE void operator()(int r, int cp, float2 u, float2 v) const {
        float2* dst = out + r * pitch + 2 * cp;
        if (aligned && 2 * cp + 1 < cols) {
            *reinterpret_cast<float4*>(dst) = make_float4(u.x, u.y, v.x, v.y);
        } else {
            if (2 * cp < cols) dst[0] = u;
            if (2 * cp + 1 < cols) dst[1] = v;
        }
    }
};

// Packed twiddle products in the range-Doppler block's n2 transforms: for schedules of radices
// <= 5 only (ERS 5 x 5 x 5: 1.483 -> 1.460 ms; ASAR IM 8 x 7 x 3 measured slower with them,
// 1.604 -> 1.683 ms).  The compiled and run-time schedules apply the same rule, so they give
// identical results.
ASARF_HD ASARF_INLINE bool az_rd_packed_twiddles(const FftPlan& p) {
    bool small = true;
    for (int i = 0; i < p.nst; ++i) small = small && p.radix[i] <= 5;
    return small;
}

// FWD = false: the caller has already put the tile through the forward transform (the
// split-precision kernel's tensor-core DFT) and synchronised.  R0, R1, R2 > 0: the n2
// transforms' radix schedule as compile-time constants (it must be the plan's).
template <bool FWD = true, int R0 = 0, int R1 = 0, int R2 = 0>
ASARF_HD ASARF_INLINE void az_rd_body(const AzRdArgs& a, int tile, int k1, int tid, int nthr, float2* s,
                                      const AzRdTables& t, unsigned int* err_flag, bool preloaded) {
    const int x0 = tile * a.xt;
    const int n2 = a.n2, wt = a.wt;
    const int ncol = *t.used;
    const FastDiv dwt = make_fastdiv(static_cast<unsigned int>(wt));
    if (!preloaded) {
        for (int t = tid; t < n2 * wt; t += nthr) {
            const int r = static_cast<int>(fdiv_u(t, dwt)), c = t - r * wt;
            const int x = x0 - a.hl + c;
            float2 v = make_float2(0.0f, 0.0f);
            if (x >= 0 && x < a.nk) v = a.in[static_cast<long long>(k1 * n2 + r) * a.pitch + x];
            s[t] = v;
        }
    }
    if constexpr (FWD) {
        if (!preloaded) ASARF_SYNC();
        if constexpr (R0 > 0)
            fft_forward_pairs_cs3<R0, R1, R2, (R0 <= 5 && R1 <= 5 && R2 <= 5)>(s, ncol, wt, a.plan2.tw, tid, nthr);
        else if (az_rd_packed_twiddles(a.plan2))
            fft_forward_pairs<true>(a.plan2, s, ncol, wt, tid, nthr);
        else
            fft_forward_pairs<false>(a.plan2, s, ncol, wt, tid, nthr);
    }
    // RCMC + matched filter.  Every output (row p, column c) reads taps of row p only, so a
    // row is computed into registers by one warp (lane = two adjacent columns, xt <= 64), the warp
    // synchronises, and writes it back in place: no block-wide barrier per row.
    const bool edge = x0 < kRcmcTaps || x0 + a.wt + kRcmcTaps > a.nk;  // tiles where some taps may leave the line
#if defined(__CUDA_ARCH__)
    {
        const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
        // lanes past the tile repeat its last columns and store nothing
        const int c = 2 * lane < a.xt ? 2 * lane : a.xt - 2;
        const int x = x0 + c;
        // a lane's two column records stay in registers for all rows
        const ColUse ca = t.cols[c], cb = t.cols[c + 1];
        ASARF_SYNC();  // the records' memory becomes the warps' weight buffers
        // a row's weights reach the lanes while the row before it is processed, then the
        // warp's buffer (read straight from the table, their latency was exposed)
        float* wbuf = t.weights + warp * kRcmcBufFloats;
        auto fetch = [&](int p) -> float {
            const int code = p < n2 ? t.rows[p].code : kRowSkip;
            return code >= 0 && lane < kRcmcBufFloats ? ASARF_LDG(rcmc_weights(a, code) + lane) : 0.0f;
        };
        float wnext = fetch(warp);
        for (int p = warp; p < n2; p += nwarps) {
            const RowRec rec = t.rows[p];
            float2* srow = s + p * wt;
            float2 va = make_float2(0.0f, 0.0f), vb = va;
            if (lane < kRcmcBufFloats) wbuf[lane] = wnext;
            __syncwarp();
            wnext = fetch(p + nwarps);
            if (rec.code >= 0) {
                rcmc_mf_pair(a, rec, wbuf, edge, ca, cb, x, srow, c, &va, &vb);
            } else if (rec.code == kRowSlow) {
                if (x < a.nk) rcmc_mf_samples(a, ca, cb, *reinterpret_cast<const float2*>(t.dc + c), x, rec.bf, srow, a.hl + c, err_flag, &va, &vb);
            }
            if (a.absolute_phase) {
                va = cmul(va, t.phs[c]);
                vb = cmul(vb, t.phs[c + 1]);
            }
            __syncwarp();
            if (2 * lane < a.xt) *reinterpret_cast<float4*>(srow + a.hl + c) = make_float4(va.x, va.y, vb.x, vb.y);
            __syncwarp();
        }
    }
    ASARF_SYNC();
#else
    {
        float2 rowbuf[64];
        for (int p = 0; p < n2; ++p) {
            const RowRec rec = t.rows[p];
            float2* srow = s + p * wt;
            for (int c = 0; c < a.xt; ++c) {
                if (rec.code >= 0) {
                    if (!(c & 1))  // with the column after it
                        rcmc_mf_pair(a, rec, rcmc_weights(a, rec.code), edge, t.cols[c], t.cols[c + 1], x0 + c, srow,
                                     c, &rowbuf[c], &rowbuf[c + 1]);
                } else if (rec.code == kRowSlow && x0 + c < a.nk) {
                    rowbuf[c] = rcmc_mf_sample(a, t.cols[c], t.dc[c], x0 + c, rec.bf, srow, a.hl + c, err_flag);
                } else {
                    rowbuf[c] = make_float2(0.0f, 0.0f);
                }
            }
            for (int c = 0; c < a.xt; ++c)
                srow[a.hl + c] = a.absolute_phase ? cmul(rowbuf[c], t.phs[c]) : rowbuf[c];
        }
    }
#endif
    // the inverse transform's last stage stores the block's rows k1 * n2 + r directly
    if constexpr (R0 > 0)
        fft_inverse_pairs_cs3<R0, R1, R2, AzRdOut, (R0 <= 5 && R1 <= 5 && R2 <= 5)>(s + a.hl, a.xt, wt, a.plan2.tw, tid,
                                                                                   nthr, AzRdOut(a, x0, k1));
    else if (az_rd_packed_twiddles(a.plan2))
        fft_inverse_pairs<AzRdOut, true>(a.plan2, s + a.hl, a.xt, wt, tid, nthr, AzRdOut(a, x0, k1));
    else
        fft_inverse_pairs<AzRdOut, false>(a.plan2, s + a.hl, a.xt, wt, tid, nthr, AzRdOut(a, x0, k1));
}

// ----------------------------------------------------------------------------- level-0 packets
// The 16 bytes that start `sh` bytes (at most 15) into the 32 bytes (lo, hi).
ASARF_HD ASARF_INLINE uint4 shift_bytes(const uint4& lo, const uint4& hi, unsigned int sh) {
    const unsigned int bits = 8u * (sh & 3u);
    const bool two = (sh & 8u) != 0, one = (sh & 4u) != 0;
    unsigned int v0 = lo.x, v1 = lo.y, v2 = lo.z, v3 = lo.w, v4 = hi.x, v5 = hi.y, v6 = hi.z;
    const unsigned int v7 = hi.w;
    if (two) v0 = v2, v1 = v3, v2 = v4, v3 = v5, v4 = v6, v5 = v7;
    if (one) v0 = v1, v1 = v2, v2 = v3, v3 = v4, v4 = v5;
    return make_uint4(funnel_r(v0, v1, bits), funnel_r(v1, v2, bits), funnel_r(v2, v3, bits), funnel_r(v3, v4, bits));
}

// Whole 16-byte units that copy_units may write from n source bytes at src: a unit whose source
// is not 16-byte aligned is read as the two aligned 16-byte words it lies in, and both words
// must end inside the n bytes.
ASARF_HD ASARF_INLINE int copy_units_of(const uint8_t* src, int n) {
    const int sh = static_cast<int>(reinterpret_cast<uintptr_t>(src) & 15);
    const int usable = sh ? n - (16 - sh) : n;
    return usable > 0 ? usable / 16 : 0;
}

// units 16-byte units from src (any alignment) to dst (16-byte aligned), threads on
// consecutive units.  The aligned word below src is read too: the callers' sources start
// inside a packet, past its header.  kBatch units of a thread are loaded before any is stored.
template <int kBatch>
ASARF_HD ASARF_INLINE void copy_units(const uint8_t* src, uint8_t* dst, int units, int tid, int nthr) {
    const unsigned int sh = static_cast<unsigned int>(reinterpret_cast<uintptr_t>(src) & 15);
    const uint4* a = reinterpret_cast<const uint4*>(src - sh);
    uint4* d = reinterpret_cast<uint4*>(dst);
    for (int u0 = tid; u0 < units; u0 += kBatch * nthr) {
        uint4 lo[kBatch], hi[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = u0 + k * nthr;
            if (u < units) {
                lo[k] = ASARF_LDG(a + u);
                if (sh) hi[k] = ASARF_LDG(a + u + 1);
            }
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = u0 + k * nthr;
            if (u < units) d[u] = sh ? shift_bytes(lo[k], hi[k], sh) : lo[k];
        }
    }
}

// Line y of an ERS IM measurement data set: its packet's 11232 measurement bytes go to raw
// line y, its SWST and PRI codes (big-endian, ISP bytes 38-39 and 40-41 after the 32 bytes of
// sensing time and FEP annotation) to swst[y] / pri[y]; the FEP ISP length (11465) and the
// auxiliary section's 0xAA marker are checked as ParseErsLevel0ImPackets checks them
// (envisat_format/src/ers_im_parse.cc:423-453).  A warp takes the line.  Its 16-byte aligned interior moves by
// whole units, what lies before and after it (at most 15 and 31 bytes) by bytes: 28000 lines to a raw buffer
// 2 bytes off 16-byte alignment 113 us, as aligned; all by 2-byte words 400.
ASARF_HD ASARF_INLINE void ers_unpack_line(const ErsUnpackArgs& a, int y, int tid, int nthr) {
    const uint8_t* pk = a.mdsr + ASARF_LDG(a.offset + y);
    const uint8_t* src = pk + kErsMeasurementOffset;
    uint8_t* dst = a.raw + static_cast<long long>(y) * kErsMeasurementBytes;
    const int head = static_cast<int>((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15);
    const int units = copy_units_of(src + head, kErsMeasurementBytes - head);
    copy_units<4>(src + head, dst + head, units, tid, nthr);
    for (int i = tid; i < head; i += nthr) dst[i] = src[i];
    for (int i = head + 16 * units + tid; i < kErsMeasurementBytes; i += nthr) dst[i] = src[i];
    if (tid == 0) {
        const int isp_len = (pk[24] << 8) | pk[25];
        unsigned e = 0;
        if (isp_len != 11465) e |= kErrL0IspLength;
        if (pk[32 + 4 + 10] != 0xAA) e |= kErrL0AuxMarker;
        if (e) atomic_or_u32(a.errors, e);
        const uint8_t* aux = pk + 32 + 4 + 10;  // 0xAA, OBRC/orbit, 4-byte OBT, activity, flags, 4-byte IF counter
        if (a.swst) a.swst[y] = static_cast<uint16_t>((aux[12] << 8) | aux[13]);
        if (a.pri) a.pri[y] = static_cast<uint16_t>((aux[14] << 8) | aux[15]);
    }
}

// Line y of an ASAR IM level-0 list: the sample blocks of its source packet (an echo packet;
// a calibration line repeats the previous line's echo, as ParseEnvisatLevel0ImPackets copies
// the previous record, envisat_format/src/envisat_im_parse.cc:599-615) become FBAQ4 record y:
// the block-data length as a little-endian uint16 (the reference's memcpy of a uint16 on a
// little-endian host), the blocks, zeros up to record_bytes.  SWST and PRI codes are the source
// packet's.  The packet's data field header length (29) and mode ID (0x54) are checked as the
// reference checks them (:470-484); a block length beyond the record sets kErrL0Length and the
// record keeps only what fits.  A warp takes the record: its 16-byte aligned interior moves by whole
// units, what lies before and after it (records have any size and any alignment) by bytes.
ASARF_HD ASARF_INLINE void asar_unpack_line(const AsarUnpackArgs& a, int y, int tid, int nthr) {
    const uint8_t* pk = a.mdsr + ASARF_LDG(a.src + y);
    const int packet_length = (pk[36] << 8) | pk[37];
    int len = packet_length - 29;
    const int cap = a.record_bytes - 2;
    unsigned e = 0;
    if (((pk[38] << 8) | pk[39]) != 29) e |= kErrL0DataField;
    if (pk[41] != 0x54) e |= kErrL0Mode;
    if (len < 0 || len > cap) {
        e |= kErrL0Length;
        len = len < 0 ? 0 : cap;
    }
    uint8_t* rec = a.records + static_cast<long long>(y) * a.record_bytes;
    const uint8_t* blocks = pk + kAsarPacketHeader;
    // record bytes [head, head + 16 units) by units: head is the first aligned byte past the length
    const int head = 2 + static_cast<int>((16 - (reinterpret_cast<uintptr_t>(rec + 2) & 15)) & 15);
    const int units = copy_units_of(blocks + (head - 2), len - (head - 2));
    copy_units<4>(blocks + (head - 2), rec + head, units, tid, nthr);
    auto byte_at = [&](int i) -> uint8_t {
        if (i == 0) return static_cast<uint8_t>(len & 0xFF);
        if (i == 1) return static_cast<uint8_t>(len >> 8);
        return i - 2 < len ? blocks[i - 2] : static_cast<uint8_t>(0);
    };
    const int first = head < a.record_bytes ? head : a.record_bytes;
    for (int i = tid; i < first; i += nthr) rec[i] = byte_at(i);
    for (int i = head + 16 * units + tid; i < a.record_bytes; i += nthr) rec[i] = byte_at(i);
    if (tid == 0) {
        if (e) atomic_or_u32(a.errors, e);
        if (a.pri) a.pri[y] = static_cast<uint16_t>((pk[54] << 8) | pk[55]);
        if (a.swst) a.swst[y] = static_cast<uint16_t>((pk[56] << 8) | pk[57]);
    }
}

// ----------------------------------------------------------------------------- L1 product records
// Envisat MDS records of the level-1 products (ConditionResultsSLC / ConditionResultsDetected,
// envisat_format/src/envisat_format_kernels.cu:28-114): `hdr` zero bytes of record header, then
// the pixels.  IMS: I and Q of a complex pixel times the calibration constant, clamped to the
// int16 range and truncated toward zero (NaN gives 0), big-endian.  IMP: 10 log10 of the
// intensity times the constant, capped at 65535 and truncated to uint16 (negative, -inf and NaN
// give 0), least significant byte first as the reference kernel stores it.
ASARF_HD ASARF_INLINE int f2i_rz(float v) {
#if defined(__CUDA_ARCH__)
    return __float2int_rz(v);  // NaN -> 0
#else
    return v != v ? 0 : static_cast<int>(v);
#endif
}

ASARF_HD ASARF_INLINE unsigned int f2u_rz(float v) {
#if defined(__CUDA_ARCH__)
    return __float2uint_rz(v);  // negative, NaN -> 0
#else
    return (v != v || v <= 0.0f) ? 0u : static_cast<unsigned int>(v);
#endif
}

ASARF_HD ASARF_INLINE float log10_f32(float x) {
#if defined(__CUDA_ARCH__)
    return log10f(x);
#else
    return static_cast<float>(__builtin_log10(static_cast<double>(x)));
#endif
}

ASARF_HD ASARF_INLINE int ims_value(float v, float cal) {
    const float s = fmul_rn(v, cal);
    const float c = s > 32767.0f ? 32767.0f : (s < -32768.0f ? -32768.0f : s);
    return f2i_rz(c);
}

ASARF_HD ASARF_INLINE unsigned int imp_value(float v, float cal) {
    const float db = fmul_rn(10.0f, log10_f32(fmul_rn(v, cal)));
    return f2u_rz(65535.0f < db ? 65535.0f : db);
}

// IMP pixel x of a record payload.
ASARF_HD ASARF_INLINE void imp_store(uint8_t* payload, int x, float v, float cal) {
    const unsigned int u = imp_value(v, cal);
    payload[2 * x] = static_cast<uint8_t>(u & 0xff);
    payload[2 * x + 1] = static_cast<uint8_t>((u >> 8) & 0xff);
}

// ----------------------------------------------------------------------------- detected tail
// One output line per block: results-window subset (main_flow.cc:585-627), time-domain
// azimuth multilook (TimeDomainAzimuthLook, sar/az_multilook.cu:25-80), range spreading loss
// gain (sar/range_spreading_loss.cu:29-52) and slant-to-ground resampling with the
// reference's float Horner / IEEE division / truncation index (SrGrInterpolation,
// sar/srgr.cu:49-71).  ml holds one multilooked slant row (nx floats).
ASARF_HD ASARF_INLINE void tail_body(const TailArgs& a, int y, int tid, int nthr, float* ml, unsigned int* err_flag) {
    const FocusState& st = *a.state;
    const TailVariant& tv = a.tail[st.variant];
    if (y >= tv.out_az) return;
    const int in_y = st.n_lines;
    const float in_idx = fmul_rn(static_cast<float>(y), tv.ratio);
    const float mu = fsub_rn(in_idx, static_cast<float>(static_cast<int>(in_idx)));
    int s0 = static_cast<int>(fsub_rn(in_idx, 2.0f)), e0 = static_cast<int>(fadd_rn(in_idx, 2.0f));
    int s1 = static_cast<int>(fsub_rn(in_idx, 1.0f)), e1 = static_cast<int>(fadd_rn(in_idx, 3.0f));
    s0 = s0 > 0 ? s0 : 0;
    s1 = s1 > 0 ? s1 : 0;
    e0 = e0 < in_y ? e0 : in_y;
    e1 = e1 < in_y ? e1 : in_y;
    const int c0 = e0 > s0 ? e0 - s0 : 0;
    const int c1 = e1 > s1 ? e1 - s1 : 0;
    const float2* base = a.slc + static_cast<long long>(st.first_line) * a.pitch + a.col0;
    const float* ibase = a.intensity ? a.intensity + static_cast<long long>(st.first_line) * a.pitch + a.col0 : nullptr;
    const int r_lo = s0 < s1 ? s0 : s1;
    const int r_hi = e0 > e1 ? e0 : e1;
    // each input row is read once and added to whichever box mean(s) contain it, in row
    // order, so both sums accumulate exactly as the reference's two loops do
    // the window spans at most kTailRows rows (5, or 6 where x + 3 rounds up across a power
    // of two); all of a column's rows are loaded before any is summed, two columns at a time
    constexpr int kTailRows = 6;
    const int nr = r_hi - r_lo;
    // the box divisions and the resampling index divide by block constants: correctly rounded
    // quotients from their correctly rounded reciprocals (div_by_recip_rn)
    const float fc0 = c0 ? static_cast<float>(c0) : 1.0f, fc1 = c1 ? static_cast<float>(c1) : 1.0f;
    const float rc0 = fdiv_rn(1.0f, fc0), rc1 = fdiv_rn(1.0f, fc1);
    // |z|^2 of row r, column c: from the complex SLC, or read directly from the intensity rows
    // the inverse azimuth pass wrote for detected products (half the bytes, same rounding)
    auto power = [&](int r, int c) -> float {
        const long long o = static_cast<long long>(r) * a.pitch + c;
        if (ibase) return ibase[o];
        const float2 w = base[o];
        return fma_rn(w.x, w.x, fmul_rn(w.y, w.y));
    };
    // column c from its window rows v[0 .. kTailRows) (rows r_lo + k; later rows, when the window
    // is longer, read here): both box means, their interpolation and the range spreading loss
    auto finish = [&](int c, const float* v) {
        float sum0 = 0.0f, sum1 = 0.0f;
#pragma unroll
        for (int k = 0; k < kTailRows; ++k) {
            const int r = r_lo + k;
            if (k >= nr) break;
            if (r >= s0 && r < e0) sum0 = fadd_rn(sum0, v[k]);
            if (r >= s1 && r < e1) sum1 = fadd_rn(sum1, v[k]);
        }
        for (int r = r_lo + kTailRows; r < r_hi; ++r) {
            const float p2 = power(r, c);
            if (r >= s0 && r < e0) sum0 = fadd_rn(sum0, p2);
            if (r >= s1 && r < e1) sum1 = fadd_rn(sum1, p2);
        }
        if (c0) sum0 = div_by_recip_rn(sum0, fc0, rc0);
        if (c1) sum1 = div_by_recip_rn(sum1, fc1, rc1);
        float val = 0.0f;
        if (c0 && c1) val = fma_rn(fsub_rn(sum1, sum0), mu, sum0);
        ml[c] = fmul_rn(val, ASARF_LDG(tv.rsl + c));
    };
    // 16-byte aligned rows: four adjacent columns per thread, one 16-byte load per row of |z|^2
    // floats, or two of complex samples (|z|^2 formed with the same rounding as power())
    // (columns past the last whole group of four, when nx is not a multiple of 4, one per thread)
    const bool quad = (a.pitch & 3) == 0 && (ibase ? (reinterpret_cast<uintptr_t>(ibase) & 15) == 0
                                                   : (reinterpret_cast<uintptr_t>(base) & 15) == 0);
    if (quad) {
        for (int q = tid; q < a.nx / 4; q += nthr) {
            float4 w[kTailRows];
            if (ibase) {
#pragma unroll
                for (int k = 0; k < kTailRows; ++k) {
                    w[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (k < nr)
                        w[k] = *reinterpret_cast<const float4*>(ibase + static_cast<long long>(r_lo + k) * a.pitch + 4 * q);
                }
            } else {
#pragma unroll
                for (int k = 0; k < kTailRows; ++k) {
                    float4 z0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), z1 = z0;
                    if (k < nr) {
                        const float4* p =
                            reinterpret_cast<const float4*>(base + static_cast<long long>(r_lo + k) * a.pitch + 4 * q);
                        z0 = p[0];
                        z1 = p[1];
                    }
                    w[k] = make_float4(fma_rn(z0.x, z0.x, fmul_rn(z0.y, z0.y)), fma_rn(z0.z, z0.z, fmul_rn(z0.w, z0.w)),
                                       fma_rn(z1.x, z1.x, fmul_rn(z1.y, z1.y)), fma_rn(z1.z, z1.z, fmul_rn(z1.w, z1.w)));
                }
            }
            float v[kTailRows];
#pragma unroll
            for (int k = 0; k < kTailRows; ++k) v[k] = w[k].x;
            finish(4 * q, v);
#pragma unroll
            for (int k = 0; k < kTailRows; ++k) v[k] = w[k].y;
            finish(4 * q + 1, v);
#pragma unroll
            for (int k = 0; k < kTailRows; ++k) v[k] = w[k].z;
            finish(4 * q + 2, v);
#pragma unroll
            for (int k = 0; k < kTailRows; ++k) v[k] = w[k].w;
            finish(4 * q + 3, v);
        }
        for (int c = (a.nx & ~3) + tid; c < a.nx; c += nthr) {
            float v[kTailRows];
#pragma unroll
            for (int k = 0; k < kTailRows; ++k) v[k] = k < nr ? power(r_lo + k, c) : 0.0f;
            finish(c, v);
        }
    } else {
        for (int cb = tid; cb < a.nx; cb += 2 * nthr) {
            float v[2][kTailRows];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = cb + h * nthr;
#pragma unroll
                for (int k = 0; k < kTailRows; ++k) {
                    v[h][k] = 0.0f;
                    if (k < nr && c < a.nx) v[h][k] = power(r_lo + k, c);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = cb + h * nthr;
                if (c >= a.nx) break;
                finish(c, v[h]);
            }
        }
    }
    ASARF_SYNC();
    float* orow = a.mds ? nullptr : a.out + static_cast<long long>(y) * a.out_pitch;
    uint8_t* rec = a.mds ? a.mds + static_cast<long long>(y) * (a.mds_hdr + 2 * tv.ng) : nullptr;
    if (rec)
        for (int i = tid; i < a.mds_hdr; i += nthr) rec[i] = 0;
    const float rsp = fdiv_rn(1.0f, a.range_spacing);
    for (int xg = tid; xg < tv.ng; xg += nthr) {
        const float gd = fmul_rn(static_cast<float>(xg), a.ground_spacing);
        const float rd = polyval_f32(tv.grsr, gd);
        const float idx = div_by_recip_rn(rd, a.range_spacing, rsp);
        int i0 = static_cast<int>(idx);
        const float dx = fsub_rn(idx, static_cast<float>(i0));
        if (i0 < 0 || i0 + 1 >= a.nx) {
            atomic_or_u32(err_flag, kErrSrgrIndex);
            i0 = i0 < 0 ? 0 : a.nx - 2;
        }
        const float v0 = ml[i0], v1 = ml[i0 + 1];
        const float v = fma_rn(dx, fsub_rn(v1, v0), v0);
        if (rec)
            imp_store(rec + a.mds_hdr, xg, v, a.mds_cal);
        else
            orow[xg] = v;
        if (a.out2) a.out2[static_cast<long long>(y) * a.out_pitch + xg] = v;
    }
}

// One record of a level-1 product (row y of the input).  Records start at any byte, so the
// payload leaves in 16-byte aligned units: a thread forms the four 32-bit words (an IMS pixel, or
// two IMP ones, each) its unit starts in, takes the fifth from the next lane and funnels them into
// place.  kBatch units of a thread are loaded before any is converted.  The header, the bytes
// before the first aligned one and those past the last whole unit leave one by one.  Bound by
// HBM traffic: both records of a 5003 x 4896 SLC and a 1000 x 4896 image, calls included, 113 us
// with byte stores, 93 us so (132 us with the words staged in shared memory instead).
template <bool IMS>
ASARF_HD ASARF_INLINE void condition_row_of(const ConditionArgs& a, int y, int tid, int nthr) {
    constexpr int kBatch = 2;
    const float2* z = a.slc;
    int rows = a.y_size;
    if (IMS && a.state) {
        z += static_cast<long long>(a.state->first_line) * a.stride;
        rows = a.state->n_lines;
    }
    if (y >= rows) return;
    const int bytes = (IMS ? 4 : 2) * a.x_size;  // payload
    if (IMS) z += static_cast<long long>(y) * a.stride;
    const float* row = IMS ? nullptr : a.img + static_cast<long long>(y) * a.stride;
    uint8_t* rec = a.dest + static_cast<long long>(y) * (a.hdr + static_cast<long long>(bytes));
    uint8_t* payload = rec + a.hdr;
    // the pixels of payload word j (a complex one or two detected ones; zeros past the row)
    auto pixels = [&](int j) -> float2 {
        if (IMS) return j < a.x_size ? z[j] : make_float2(0.0f, 0.0f);
        return make_float2(2 * j < a.x_size ? row[2 * j] : 0.0f, 2 * j + 1 < a.x_size ? row[2 * j + 1] : 0.0f);
    };
    // payload word as it lies in memory, read little-endian
    auto word = [&](float2 v) -> unsigned int {
        if (IMS) {  // most significant byte of each value first
            const unsigned int i = static_cast<unsigned int>(ims_value(v.x, a.cal)) & 0xffffu;
            const unsigned int q = static_cast<unsigned int>(ims_value(v.y, a.cal)) & 0xffffu;
            return byte_perm(i, q, 0x4501u);
        }
        return (imp_value(v.x, a.cal) & 0xffffu) | (imp_value(v.y, a.cal) << 16);
    };
    auto byte_at = [&](int i) -> uint8_t { return static_cast<uint8_t>(word(pixels(i >> 2)) >> (8 * (i & 3))); };
    const int h = static_cast<int>((16 - (reinterpret_cast<uintptr_t>(payload) & 15)) & 15);
    const int units = bytes > h ? (bytes - h) / 16 : 0;
    const int w0 = h >> 2;
    const unsigned int sh = 8u * static_cast<unsigned int>(h & 3);
    uint4* dst = reinterpret_cast<uint4*>(payload + h);
    for (int u0 = 0; u0 < units; u0 += kBatch * nthr) {
        float2 px[kBatch][5];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = u0 + k * nthr + tid;
#pragma unroll
            for (int m = 0; m < 4; ++m) px[k][m] = u <= units ? pixels(w0 + 4 * u + m) : make_float2(0.0f, 0.0f);
#if defined(__CUDA_ARCH__)
            // the lane above holds the fifth word's pixels, except for the last lane
            px[k][4] = make_float2(0.0f, 0.0f);
            if ((tid & 31) == 31 && u < units) px[k][4] = pixels(w0 + 4 * u + 4);
#else
            px[k][4] = pixels(w0 + 4 * u + 4);
#endif
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = u0 + k * nthr + tid;
            const unsigned int v0 = word(px[k][0]), v1 = word(px[k][1]), v2 = word(px[k][2]), v3 = word(px[k][3]);
#if defined(__CUDA_ARCH__)
            unsigned int v4 = __shfl_down_sync(0xffffffffu, v0, 1);
            if ((tid & 31) == 31) v4 = word(px[k][4]);
#else
            const unsigned int v4 = word(px[k][4]);
#endif
            if (u < units)
                dst[u] = make_uint4(funnel_r(v0, v1, sh), funnel_r(v1, v2, sh), funnel_r(v2, v3, sh), funnel_r(v3, v4, sh));
        }
    }
    for (int i = tid; i < a.hdr; i += nthr) rec[i] = 0;
    const int head = h < bytes ? h : bytes;
    for (int i = tid; i < head; i += nthr) payload[i] = byte_at(i);
    for (int i = h + 16 * units + tid; i < bytes; i += nthr) payload[i] = byte_at(i);
}

ASARF_HD ASARF_INLINE void condition_row(const ConditionArgs& a, int y, int tid, int nthr) {
    if (a.product == 2) condition_row_of<true>(a, y, tid, nthr);
    else condition_row_of<false>(a, y, tid, nthr);
}

// ----------------------------------------------------------------------------- product statistics
// Pair p of the product statistics.  IMS form: SLC pixel p of the results window.  IMP form: the
// reference reuses the subset SLC's buffer for the ground-range floats and views it as a
// complex image of the ground-range size (main.cc:327-331), so pair p is floats 2p, 2p+1 of
// that buffer: ground-range pixels below N = ng * out_az, beyond it the SLC floats the
// resampling did not overwrite (SLC stored contiguously [lines][nx], as the subset copy leaves it).
ASARF_HD ASARF_INLINE float stats_float(const ProductStatsArgs& a, long long f, long long n_img, int ng) {
    if (f < n_img) {
        const long long r = f / ng;
        return a.img[r * a.img_pitch + (f - r * ng)];
    }
    const long long k = f >> 1;
    const long long r = k / a.nx;
    const float2 z = a.slc[(a.state->first_line + r) * a.slc_pitch + (k - r * a.nx)];
    return (f & 1) ? z.y : z.x;
}

ASARF_HD ASARF_INLINE long long stats_pairs(const ProductStatsArgs& a) {
    const FocusState& st = *a.state;
    return a.imaged ? static_cast<long long>(a.ng[st.variant]) * a.out_az[st.variant]
                    : static_cast<long long>(st.n_lines) * a.nx;
}

// Block `blk` of `a.blocks`: pairs blk * 256 + t, stepping by blocks * 256, into part[blk]
// (pairwise tree over the 256 lanes).
ASARF_HD ASARF_INLINE void product_stats_body(const ProductStatsArgs& a, int blk, int tid, int nthr, double* red) {
    const FocusState& st = *a.state;
    const long long n = stats_pairs(a);
    const int ng = a.ng[st.variant];
    const long long n_img = static_cast<long long>(ng) * a.out_az[st.variant];
    for (int t = tid; t < 256; t += nthr) {
        double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        for (long long p = static_cast<long long>(blk) * 256 + t; p < n; p += static_cast<long long>(a.blocks) * 256) {
            float x, y;
            if (a.imaged) {
                x = stats_float(a, 2 * p, n_img, ng);
                y = stats_float(a, 2 * p + 1, n_img, ng);
            } else {
                const long long r = p / a.nx;
                const float2 z = a.slc[(st.first_line + r) * a.slc_pitch + (p - r * a.nx)];
                x = z.x;
                y = z.y;
            }
            if (x != x || y != y) continue;
            v[0] += 1.0;
            v[1] += x;
            v[2] += y;
            v[3] += static_cast<double>(x) * x;
            v[4] += static_cast<double>(y) * y;
        }
        for (int k = 0; k < 5; ++k) red[k * 256 + t] = v[k];
    }
    ASARF_SYNC();
    for (int h = 128; h > 0; h >>= 1) {
        for (int t = tid; t < 5 * h; t += nthr) {
            const int k = t / h, i = t - k * h;
            red[k * 256 + i] += red[k * 256 + i + h];
        }
        ASARF_SYNC();
    }
    for (int k = tid; k < 5; k += nthr) a.part[static_cast<long long>(blk) * 5 + k] = red[k * 256];
}

// Fold of the block partials (pairwise tree over kStatsFoldLeaves leaves) and the statistics in
// the reference's arithmetic: mean = float(float(sum) / float(N)), deviation = sqrt(float(
// float(sum of squared differences) / float(N))) with N all pairs, as CalcMean / CalcStdDev
// divide by the image size; IMS: (mean I, mean Q, dev I, dev Q), IMP: ((mean I + mean Q) / 2, 0,
// (dev I + dev Q) / 2, 0); then scaled by the calibration constant as main.cc:336-342, 384-390.
constexpr int kStatsFoldLeaves = 1024;
ASARF_HD ASARF_INLINE void product_stats_fold(const ProductStatsArgs& a, int tid, int nthr, double* tree) {
    for (int t = tid; t < 5 * kStatsFoldLeaves; t += nthr) {
        const int k = t / kStatsFoldLeaves, i = t - k * kStatsFoldLeaves;
        tree[t] = i < a.blocks ? a.part[static_cast<long long>(i) * 5 + k] : 0.0;
    }
    ASARF_SYNC();
    for (int h = kStatsFoldLeaves / 2; h > 0; h >>= 1) {
        for (int t = tid; t < 5 * h; t += nthr) {
            const int k = t / h, i = t - k * h;
            tree[k * kStatsFoldLeaves + i] += tree[k * kStatsFoldLeaves + i + h];
        }
        ASARF_SYNC();
    }
    if (tid != 0) return;
    const double cnt = tree[0], sx = tree[kStatsFoldLeaves], sy = tree[2 * kStatsFoldLeaves];
    const double sxx = tree[3 * kStatsFoldLeaves], syy = tree[4 * kStatsFoldLeaves];
    const float nf = static_cast<float>(stats_pairs(a));
    const float mx = static_cast<float>(sx) / nf, my = static_cast<float>(sy) / nf;
    const double dx = sxx - 2.0 * mx * sx + cnt * static_cast<double>(mx) * mx;
    const double dy = syy - 2.0 * my * sy + cnt * static_cast<double>(my) * my;
    const float vx = static_cast<float>(dx) / nf, vy = static_cast<float>(dy) / nf;
    const float ex = sqrtf(vx), ey = sqrtf(vy);
    const double c = a.cal;
    if (a.imaged) {
        a.out[0] = static_cast<double>((mx + my) / 2) * c;
        a.out[1] = 0.0;
        a.out[2] = static_cast<double>((ex + ey) / 2) * c;
        a.out[3] = 0.0;
    } else {
        a.out[0] = mx * c;
        a.out[1] = my * c;
        a.out[2] = ex * c;
        a.out[3] = ey * c;
    }
}

// ============================================================================= per-stage bodies

// ConvertErsImSamplesToComplexKernel (envisat_format/src/envisat_format_kernels.cu:116-134)
// after the NaN pre-fill of ConvertRawSampleSetsToComplex (main_flow.cc:537-540): line y.
ASARF_HD ASARF_INLINE void decode_row(const DecodeArgs& a, int y, int tid, int nthr) {
    const int off = a.swst ? 4 * (static_cast<int>(a.swst[y]) - a.min_swst) : 0;
    const uint8_t* rec = a.raw + static_cast<long long>(y) * a.line_bytes;
    float2* row = a.img + static_cast<long long>(y) * a.stride;
    const bool even = (reinterpret_cast<uintptr_t>(rec) & 1) == 0;
#pragma unroll 4
    for (int x = tid; x < a.nr; x += nthr) {
        const int i = x - off;
        float2 v = make_float2(qnan_f(), qnan_f());
        if (i >= 0 && i < a.spl) {
            const unsigned int w = even ? ASARF_LDG(reinterpret_cast<const uint16_t*>(rec) + i)
                                        : static_cast<unsigned int>(rec[2 * i] | (rec[2 * i + 1] << 8));
            v = make_float2(static_cast<float>(w & 0xffu), static_cast<float>(w >> 8));
        }
        row[x] = v;
    }
}

// ConvertAsarImBlocksToComplexKernel (envisat_format/src/envisat_format_kernels.cu:160-209) as
// a gather over the pixels of line y: sample r = x - (swst[y] - min_swst) of record y through the
// instrument-file tables, NaN where the record holds no sample.
ASARF_HD ASARF_INLINE void decode_fbaq_row(const DecodeFbaqArgs& a, int y, int tid, int nthr) {
    const int off = a.swst ? static_cast<int>(a.swst[y]) - a.min_swst : 0;
    const uint8_t* rec = a.raw + static_cast<long long>(y) * a.line_bytes;
    const int len = fbaq_len(rec, a.line_bytes);
    float2* row = a.img + static_cast<long long>(y) * a.stride;
    for (int x = tid; x < a.nr; x += nthr) {
        const int r = x - off;
        float2 v = make_float2(qnan_f(), qnan_f());
        if (r >= 0) {
            const int b = r / 63;
            const int j = r + b + 1;
            if (j < len) {
                const int id = rec[2 + 64 * b];
                const int cw = rec[2 + j];
                v = make_float2(ASARF_LDG(a.lut_i + fbaq4_index(id, cw >> 4)),
                                ASARF_LDG(a.lut_q + fbaq4_index(id, cw & 15)));
            }
        }
        row[x] = v;
    }
}

ASARF_HD ASARF_INLINE bool is_nan_f(float v) { return v != v; }

// DevicePaddedImage::ZeroNaNs (cuda_util/device_padded_image.cu:322-329): only pixels that hold a NaN
// are written, so an image without any costs one read.
ASARF_HD ASARF_INLINE void zero_nan_item(float2* img, long long i) {
    float2 v = img[i];
    if (is_nan_f(v.x) || is_nan_f(v.y)) {
        if (is_nan_f(v.x)) v.x = 0.0f;
        if (is_nan_f(v.y)) v.y = 0.0f;
        img[i] = v;
    }
}

// Moment partials for RawDataCorrection / CalcMean / CalcStdDev
// (sar/iq_correction.cu:40-138, cuda_util/device_padded_image.cu:156-257): block `blk` sums
// rows [blk*rpb, ...) in double, NaN samples skipped; deterministic in-block tree.  ABOUT: the data
// columns' sums are taken about (about_i, about_q) in place of zero.
template <bool ABOUT>
ASARF_HD ASARF_INLINE void img_moments_add(const ImgMomentsArgs& a, double acc[6], float2 v) {
    if (is_nan_f(v.x) || is_nan_f(v.y)) return;
    double i = v.x, q = v.y;
    if (ABOUT) i -= a.about_i, q -= a.about_q;
    acc[0] += 1.0;
    acc[1] += i;
    acc[2] += q;
    acc[3] += i * i;
    acc[4] += q * q;
    acc[5] += i * q;
}
template <bool ABOUT>
ASARF_HD ASARF_INLINE void img_moments_body(const ImgMomentsArgs& a, int blk, int tid, int nthr, double* red) {
    double data[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, pad[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const int y0 = blk * a.rows_per_block;
    const int y1 = (y0 + a.rows_per_block < a.y_size) ? y0 + a.rows_per_block : a.y_size;
    for (int y = y0; y < y1; ++y) {
        const float2* row = a.img + static_cast<long long>(y) * a.x_stride;
        int x = tid;
        for (; x + 3 * nthr < a.x_size; x += 4 * nthr) {  // four loads in flight
            const float2 v0 = row[x], v1 = row[x + nthr], v2 = row[x + 2 * nthr], v3 = row[x + 3 * nthr];
            img_moments_add<ABOUT>(a, data, v0);
            img_moments_add<ABOUT>(a, data, v1);
            img_moments_add<ABOUT>(a, data, v2);
            img_moments_add<ABOUT>(a, data, v3);
        }
        for (; x < a.x_size; x += nthr) img_moments_add<ABOUT>(a, data, row[x]);
        for (; x < a.x_stride; x += nthr) img_moments_add<false>(a, pad, row[x]);
    }
    for (int k = 0; k < 6; ++k) red[k * nthr + tid] = data[k], red[(6 + k) * nthr + tid] = pad[k];
    ASARF_SYNC();
#if defined(__CUDA_ARCH__)
    for (int w = nthr / 2; w > 0; w >>= 1) {
        for (int t = tid; t < 12 * w; t += nthr) {
            const int k = t / w, i = t - k * w;
            red[k * nthr + i] += red[k * nthr + i + w];
        }
        ASARF_SYNC();
    }
#endif
    for (int k = tid; k < 12; k += nthr) a.partial[blk * 12 + k] = red[k * nthr];
}

// CorrectDCBias + ApplyGainCorrection + ApplyPhaseCorrection (sar/iq_correction.cu:140-178)
// over x < XStride, y < YSize; NaN stays NaN.
ASARF_HD ASARF_INLINE void iq_apply_item(const IqApplyArgs& a, long long idx) {
    float2 v = a.img[idx];
    const float i1 = fsub_rn(v.x, a.dc_i);
    const float q1 = fsub_rn(v.y, a.dc_q);
    const float i2 = fdiv_rn(i1, a.gain);
    const float q2 = fdiv_rn(fma_rn(-i2, a.sin_c, q1), a.cos_c);
    a.img[idx] = make_float2(i2, q2);
}

// PhaseDifference partials of CalculateDopplerCentroid (sar/fractional_doppler_centroid.cu:33-69):
// block (bx, by) takes kAcccCols columns (up to nblk*step, which may reach into the padding as the
// reference's last block does) of rows_per_block rows; a thread sums its column's pairs (y-1, y),
// y >= 1, of conj(z[y-1]) z[y] in FP64, reading each row once, and the columns of each Doppler
// block are added in order.  (One block per 256 rows, all columns in turn, left 28 blocks for a
// 7000-line image, 1346 us.)
ASARF_HD ASARF_INLINE void accc_body(const AcccArgs& a, int bx, int by, int grid_x, int tid, int nthr, double* cols) {
    const int y0 = by * a.rows_per_block;
    const int y1 = (y0 + a.rows_per_block < a.y_size) ? y0 + a.rows_per_block : a.y_size;
    const int x0 = bx * kAcccCols;
    constexpr int kBatch = 8;
    for (int t = tid; t < kAcccCols; t += nthr) {
        double re = 0.0, im = 0.0;
        if (x0 + t < a.xend) {
            const float2* col = a.img + x0 + t;
            float2 p = col[static_cast<long long>(y0 > 0 ? y0 - 1 : 0) * a.x_stride];
            for (int y = y0 > 0 ? y0 : 1; y < y1; y += kBatch) {
                float2 c[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                    c[u] = y + u < y1 ? col[static_cast<long long>(y + u) * a.x_stride] : make_float2(0.0f, 0.0f);
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    if (y + u >= y1) break;
                    re += static_cast<double>(p.x) * c[u].x + static_cast<double>(p.y) * c[u].y;
                    im += static_cast<double>(p.x) * c[u].y - static_cast<double>(p.y) * c[u].x;
                    p = c[u];
                }
            }
        }
        cols[2 * t] = re;
        cols[2 * t + 1] = im;
    }
    ASARF_SYNC();
    const int b0 = x0 / a.step;
    double* out = a.partial + (static_cast<long long>(by) * grid_x + bx) * a.span * 2;
    for (int t = tid; t < 2 * a.span; t += nthr) {
        const int lo = (b0 + t / 2) * a.step - x0, hi = lo + a.step;
        double acc = 0.0;
        for (int c = lo > 0 ? lo : 0; c < hi && c < kAcccCols; ++c) acc += cols[2 * c + (t & 1)];
        out[t] = acc;
    }
}

// RangeCompression on complex rows in place (sar/range_compression.cu:57-111): inputs
// x < nr, outputs x < nk scaled, [nk, x_zero_end) zeroed (FinishRangeCompression).
ASARF_HD ASARF_INLINE void rc_rows_body(const RcRowsArgs& a, int y, int tid, int nthr, float2* s) {
    const int L = a.plan.n;
    float2* row = a.img + static_cast<long long>(y) * a.stride;
    for (int l = tid; l < L; l += nthr) s[l] = l < a.nr ? row[l] : make_float2(0.0f, 0.0f);
    ASARF_SYNC();
    fft_forward(a.plan, s, 1, 1, tid, nthr);
    for (int l = tid; l < L; l += nthr) s[l] = cmul(s[l], ASARF_LDG(a.mf + l));
    ASARF_SYNC();
    fft_inverse(a.plan, s, 1, 1, tid, nthr);
    for (int l = tid; l < a.x_zero_end; l += nthr) row[l] = l < a.nk ? s[l] : make_float2(0.0f, 0.0f);
}

struct RowSource {
    static constexpr bool kActive = true;
    const float2* row;
    int nr;
    ASARF_HD ASARF_INLINE float2 operator()(int l) const { return l < nr ? row[l] : make_float2(0.0f, 0.0f); }
};

// The same with a compile-time schedule (lengths in kCtLengths), as the planned path's range
// compression: 7000 lines of 5616 samples 522 -> 242 us.
template <int L>
ASARF_HD ASARF_INLINE void rc_rows_ct_body(const RcRowsArgs& a, int y, int tid, float2* s) {
    constexpr int NTHR = CtSchedule<L>::nthr;
    float2* row = a.img + static_cast<long long>(y) * a.stride;
    ct_fft_mf_ifft<L>(s, a.ctw, a.mf, tid, RowSource{row, a.nr}, RcOut{row, a.nk});
    ct_phase<NTHR, false>([&](int t) {
        for (int x = a.nk + t; x < a.x_zero_end; x += NTHR) row[x] = make_float2(0.0f, 0.0f);
    }, tid);
}

// exp(2 pi i m / n) in FP64
ASARF_HD ASARF_INLINE void unit_root(long long m, int n, double* c, double* s) {
#if defined(__CUDA_ARCH__)
    sincospi(2.0 * static_cast<double>(m) / n, s, c);
#else
    const double a = 2.0 * 3.14159265358979323846 * static_cast<double>(m) / n;
    *c = cos(a);
    *s = sin(a);
#endif
}

// Part `part` of `parts` of the sum behind matched-filter position pos: the replica's samples of that
// stretch against exp(-2 pi i n k / L), stepped by a rotation in FP64 (L * nc terms: on one host
// thread 17 ms of every per-stage range compression and of every plan, here about 20 us).
ASARF_HD ASARF_INLINE void matched_filter_sum(const MatchedFilterArgs& a, int pos, int part, int parts, double* re,
                                              double* im) {
    const int L = a.plan.n;
    int rem = pos, k = 0, mult = 1;
    for (int i = 0; i < a.plan.nst; ++i) {
        const int q = rem / a.plan.span[i];
        rem -= q * a.plan.span[i];
        k += q * mult;
        mult *= a.plan.radix[i];
    }
    const int len = (a.nc + parts - 1) / parts, n0 = part * len, n1 = n0 + len < a.nc ? n0 + len : a.nc;
    double c, s, wc, ws, sr = 0.0, si = 0.0;
    unit_root(-(static_cast<long long>(n0) * k % L), L, &c, &s);
    unit_root(-static_cast<long long>(k), L, &wc, &ws);
    for (int n = n0; n < n1; ++n) {
        const float2 v = ASARF_LDG(a.chirp + n);
        sr += v.x * c - v.y * s;
        si += v.x * s + v.y * c;
        const double t = c * wc - s * ws;
        s = c * ws + s * wc;
        c = t;
    }
    *re = sr;
    *im = si;
}
ASARF_HD ASARF_INLINE void matched_filter_store(const MatchedFilterArgs& a, int pos, double re, double im) {
    const int R = a.last_radix;
    const int at = R > 0 ? (pos % R) * (a.plan.n / R) + pos / R : pos;
    a.mf[at] = make_float2(static_cast<float>(re * a.scale), static_cast<float>(-im * a.scale));
}

// Entry i of a twiddle table.
ASARF_HD ASARF_INLINE void twiddle_item(const TwiddleArgs& a, int i) {
    long long m = i;
    int n = a.n;
    if (a.r[0] > 0) {
        int at = i;
        for (int k = 0; k < 2; ++k) {  // pass k: (r_k - 1) * S entries exp(-2 pi i j q / M), q outer
            const int S = n / a.r[k];
            if (at < (a.r[k] - 1) * S) {
                m = static_cast<long long>(at / S + 1) * (at % S) % n;
                break;
            }
            at -= (a.r[k] - 1) * S;
            n = S;
        }
    }
    double c, s;
    unit_root(-m, n, &c, &s);
    a.out[i] = make_float2(static_cast<float>(c), static_cast<float>(s));
}
inline int twiddle_count(const TwiddleArgs& a) {
    return a.r[0] > 0 ? (a.r[0] - 1) * (a.n / a.r[0]) + (a.r[1] - 1) * (a.n / a.r[0] / a.r[1]) : a.n;
}

// TimeDomainAzimuthLook (sar/az_multilook.cu:25-80): one output line per block.  A column's window
// rows (at most 6) are loaded before any is summed.
ASARF_HD ASARF_INLINE void multilook_row_body(const MultilookArgs& a, int y, int tid, int nthr) {
    constexpr int kRows = 6;
    const float in_idx = fmul_rn(static_cast<float>(y), a.ratio);
    const float mu = fsub_rn(in_idx, static_cast<float>(static_cast<int>(in_idx)));
    int s0 = static_cast<int>(fsub_rn(in_idx, 2.0f)), e0 = static_cast<int>(fadd_rn(in_idx, 2.0f));
    int s1 = static_cast<int>(fsub_rn(in_idx, 1.0f)), e1 = static_cast<int>(fadd_rn(in_idx, 3.0f));
    s0 = s0 > 0 ? s0 : 0;
    s1 = s1 > 0 ? s1 : 0;
    e0 = e0 < a.in_y ? e0 : a.in_y;
    e1 = e1 < a.in_y ? e1 : a.in_y;
    const int c0 = e0 > s0 ? e0 - s0 : 0;
    const int c1 = e1 > s1 ? e1 - s1 : 0;
    const int r_lo = s0 < s1 ? s0 : s1;
    const int r_hi = e0 > e1 ? e0 : e1;
    const int nr = r_hi - r_lo;
    const float2* first = a.slc + static_cast<long long>(r_lo) * a.x_size;
    for (int c = tid; c < a.x_size; c += nthr) {
        float2 z[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k)
            z[k] = k < nr ? first[static_cast<long long>(k) * a.x_size + c] : make_float2(0.0f, 0.0f);
        float sum0 = 0.0f, sum1 = 0.0f;
        auto add = [&](int r, float2 v) {
            const float p2 = fma_rn(v.x, v.x, fmul_rn(v.y, v.y));
            if (r >= s0 && r < e0) sum0 = fadd_rn(sum0, p2);
            if (r >= s1 && r < e1) sum1 = fadd_rn(sum1, p2);
        };
#pragma unroll
        for (int k = 0; k < kRows; ++k)
            if (k < nr) add(r_lo + k, z[k]);
        for (int r = r_lo + kRows; r < r_hi; ++r) add(r, a.slc[static_cast<long long>(r) * a.x_size + c]);
        if (c0) sum0 = fdiv_rn(sum0, static_cast<float>(c0));
        if (c1) sum1 = fdiv_rn(sum1, static_cast<float>(c1));
        float val = 0.0f;
        if (c0 && c1) val = fma_rn(fsub_rn(sum1, sum0), mu, sum0);
        a.out[static_cast<long long>(y) * a.x_size + c] = val;
    }
}

// Rows a column's gain or resampling index serves in the two kernels below, which each form it once
// (an FP64 power, a polynomial and a division a pixel bound them before).
constexpr int kColumnRows = 32;

// CorrectionKernel of RangeSpreadingLossCorrection (sar/range_spreading_loss.cu:29-52): column x of rows
// [y0, y1).
ASARF_HD ASARF_INLINE void rsl_column(const RslArgs& a, int x, int y0, int y1) {
    const double r = a.slant_first + x * a.range_spacing;
    const double ratio = a.ref_range / r;
    const float g = static_cast<float>(1.0 / sqrt(pow(ratio, 3.0)));
    float* p = a.img + static_cast<long long>(y0) * a.range_size + x;
#pragma unroll 8
    for (int y = y0; y < y1; ++y, p += a.range_size) *p = fmul_rn(*p, g);
}

// SrGrInterpolation (sar/srgr.cu:49-71) with the float Horner / IEEE divide / truncation index: ground
// column xg of rows [y0, y1).
ASARF_HD ASARF_INLINE void srgr_column(const SrgrArgs& a, int xg, int y0, int y1) {
    const float gd = fmul_rn(static_cast<float>(xg), a.ground_spacing);
    const float rd = polyval_f32(a.grsr, gd);
    const float ridx = fdiv_rn(rd, a.range_spacing);
    int i0 = static_cast<int>(ridx);
    const float dx = fsub_rn(ridx, static_cast<float>(i0));
    if (a.start && y0 == 0) {
        a.start[xg] = i0;
        a.frac[xg] = dx;
    }
    if (!a.in) return;
    if (i0 < 0 || i0 + 1 >= a.in_x) {
        if (a.err) atomic_or_u32(a.err, kErrSrgrIndex);
        i0 = i0 < 0 ? 0 : a.in_x - 2;
    }
    const float* in = a.in + static_cast<long long>(y0) * a.in_x + i0;
    float* out = a.out + static_cast<long long>(y0) * a.out_x + xg;
#pragma unroll 8
    for (int y = y0; y < y1; ++y, in += a.in_x, out += a.out_x) {
        const float v0 = in[0], v1 = in[1];
        *out = fma_rn(dx, fsub_rn(v1, v0), v0);
    }
}

}  // namespace asarf
