// Compile-time-scheduled line FFTs for the range compression kernel.
//
// The range FFT length is a free choice (any L >= range size gives the same compressed
// samples), so the planner picks it from the lengths below and the whole transform is
// instantiated with constant radices, spans and per-thread item counts.
//
// Each length is three passes of composite radices (6, 8, 12, 16, 24 or 32), each pass one
// register-resident DFT per item: three shared-memory round trips per transform instead
// of one per radix-2..8 stage.  The last forward pass, the matched-filter multiply and the
// first inverse pass touch the same R contiguous positions, so one thread does all three in
// registers (no shared-memory traffic between them).  The tile is padded with one element
// after every Q = (last radix) elements: every pass's R inputs stay at a constant stride,
// and lanes reading blocks of Q contiguous elements fall into different banks.
//
// Twiddles: a per-pass table tw_I[q][j] = exp(-2 pi i j q / M_I) (q = 1..R_I-1, j < S_I,
// M_I = R_I S_I), adjacent j adjacent in memory so a warp's loads coalesce; the matched
// filter is stored transposed, mf[q][b] for position b*R_last + q, for the same reason.
// The output order of the forward transform (and so the matched filter's order) is the
// digit reversal of this radix sequence, which the host builds from ct_radices().
#pragma once

#include "fft.cuh"
#include "hd.cuh"

namespace asarf {

// ----------------------------------------------------------------------------- schedules
// Threads of a block, resident blocks an SM must hold (the register cap), radices.  A pass is L / R
// butterflies, so the thread counts are those that share every pass's butterflies evenly, or nearly,
// and the blocks are the most that registers (80 a thread, 64 at least for a radix of 24) and shared
// memory (the tile and the staged record) leave room for: what a barrier idles in one line's passes
// the others fill.  A last radix of 16 reads and writes the tile with fewer passes over its banks
// than 8 or 12 do.  Range compression of 12000 byte lines (FBAQ4 records), us, the schedules before
// (two blocks per SM asked for) and these:
//   768:  8 8 12 x 96 threads    53,       now  46      3072: 16 16 12 x 256  219 (265), now 169 (209)
//   1024: 8 8 16 x 128           66,       now  56      4096: 16 16 16 x 256  270 (352), now 235 (295)
//   1536: 24 8 8 x 192          158,       now  84      6144: 24 16 16 x 384  398 (508), now 379 (461)
//   2048: 16 16 8 x 128         135 (172), now 105 (130)
// Also timed: 1024 = 16 8 8 60, 4 16 16 58; 1536 = 24 8 8 x 64 91, 12 8 16 91; 2048 = 8 16 16 109
// (134); 3072 = 12 16 16 176 (222), 96 threads 205; 4096 x 128 267 (311); 6144 = 24 16 16 x 256 392
// (453), 16 16 24 397 (482), 24 16 16 x 128 424; 8192 = 32 16 16 545 (685), 16 32 16 602 (674),
// 32 16 16 x 512 751, against the 561 (664) of the one kept: its tile leaves room for two blocks.
template <int L>
struct CtSchedule {
    static constexpr int count = 0;
};
#define ASARF_CT_SCHEDULE(LEN, NT, BLK, R0, R1, R2) \
    template <>                                      \
    struct CtSchedule<LEN> {                         \
        static constexpr int r[] = {R0, R1, R2};     \
        static constexpr int count = 3;              \
        static constexpr int nthr = NT;              \
        static constexpr int blocks = BLK;           \
    }
ASARF_CT_SCHEDULE(768, 96, 6, 12, 8, 8);
ASARF_CT_SCHEDULE(1024, 64, 10, 8, 8, 16);
ASARF_CT_SCHEDULE(1536, 96, 8, 6, 16, 16);
ASARF_CT_SCHEDULE(2048, 128, 6, 16, 8, 16);
ASARF_CT_SCHEDULE(3072, 192, 4, 16, 12, 16);
ASARF_CT_SCHEDULE(4096, 256, 3, 16, 16, 16);
ASARF_CT_SCHEDULE(6144, 256, 3, 16, 24, 16);
ASARF_CT_SCHEDULE(8192, 256, 2, 16, 16, 32);
#undef ASARF_CT_SCHEDULE

#define ASARF_CT_LENGTHS(X) X(768) X(1024) X(1536) X(2048) X(3072) X(4096) X(6144) X(8192)
#define ASARF_LENGTH_ITEM(L) L,
constexpr int kCtLengths[] = {ASARF_CT_LENGTHS(ASARF_LENGTH_ITEM)};
#undef ASARF_LENGTH_ITEM

// Radix sequence of a compile-time length (host: digit reversal, matched filter, tables).
inline int ct_radices(int L, int* out) {
    auto put = [&](const int* r) {
        for (int i = 0; i < 3; ++i) out[i] = r[i];
        return 3;
    };
    switch (L) {
        case 768: return put(CtSchedule<768>::r);
        case 1024: return put(CtSchedule<1024>::r);
        case 1536: return put(CtSchedule<1536>::r);
        case 2048: return put(CtSchedule<2048>::r);
        case 3072: return put(CtSchedule<3072>::r);
        case 4096: return put(CtSchedule<4096>::r);
        case 6144: return put(CtSchedule<6144>::r);
        case 8192: return put(CtSchedule<8192>::r);
        default: return 0;
    }
}

template <int L, int I>
ASARF_HD constexpr int ct_span() {
    int m = L;
    for (int k = 0; k <= I; ++k) m /= CtSchedule<L>::r[k];
    return m;
}
// offset of pass I's twiddle table: sum over the earlier passes of (R - 1) * S
template <int L, int I>
ASARF_HD constexpr int ct_tw_offset() {
    int off = 0, m = L;
    for (int k = 0; k < I; ++k) {
        m /= CtSchedule<L>::r[k];
        off += (CtSchedule<L>::r[k] - 1) * m;
    }
    return off;
}
template <int L>
ASARF_HD constexpr int ct_padq() {
    return CtSchedule<L>::r[CtSchedule<L>::count - 1];
}
// padded shared-memory index of transform position e
template <int L>
ASARF_HD ASARF_INLINE int ct_pad(int e) {
    return e + e / ct_padq<L>();
}
// host: padded tile elements of a compile-time length
inline int ct_smem_elems_of(int L) {
    int r[3];
    return ct_radices(L, r) ? L + L / r[2] : 0;
}

// Run `phase(tid)` for this thread and barrier (device), or for every thread in turn (host
// emulation, where a phase must complete for all threads before the next one starts).
template <int NTHR, bool SYNC = true, class F>
ASARF_HD ASARF_INLINE void ct_phase(F&& phase, int tid) {
#if defined(__CUDA_ARCH__)
    phase(tid);
    if (SYNC) __syncthreads();
#else
    (void)tid;
    for (int t = 0; t < NTHR; ++t) phase(t);
#endif
}

// Inputs come from the tile.
struct NoSrc {
    static constexpr bool kActive = false;
};

// One pass I < count-1 (span S > 1, a multiple of Q): forward DIF (DFT, then twiddle output q
// by W_M^{jq}) or inverse DIT (conjugate twiddles on the inputs, then the inverse DFT).
// An active Epi receives each output (natural position, value) instead of the tile: the last
// inverse pass hands the line straight to its destination.  An active Src gives each input (natural
// position) instead of the tile: the first forward pass forms the line's samples as it reads them.
template <int L, int I, bool INV, class Epi = NoEpi, class Src = NoSrc>
ASARF_HD ASARF_INLINE void ct_pass(float2* s, const float2* __restrict__ ctw, int t, const Epi& epi = Epi{},
                                   const Src& src = Src{}) {
    constexpr int NTHR = CtSchedule<L>::nthr;
    constexpr int R = CtSchedule<L>::r[I];
    constexpr int S = ct_span<L, I>();
    constexpr int M = S * R;
    constexpr int Q = ct_padq<L>();
    constexpr int ITEMS = L / R;
    constexpr int PER = (ITEMS + NTHR - 1) / NTHR;
    constexpr int STRIDE = S + S / Q;  // padded distance between a butterfly's inputs
    constexpr int TWO = ct_tw_offset<L, I>();
    static_assert(S % Q == 0, "every pass but the last has a span divisible by the pad quotient");
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int it = t + k * NTHR;
        if (ITEMS % NTHR != 0 && it >= ITEMS) break;
        const int b = it / S;
        const int j = it - b * S;
        float2* p = s + ct_pad<L>(b * M + j);
        float2 v[R];
#pragma unroll
        for (int m = 0; m < R; ++m) {
            if constexpr (Src::kActive) v[m] = src(b * M + j + m * S);
            else v[m] = p[m * STRIDE];
        }
        if (INV) {
            if (j != 0) {
#pragma unroll
                for (int q = 1; q < R; ++q) v[q] = cmulc(v[q], ASARF_LDG(ctw + TWO + (q - 1) * S + j));
            }
            dft_any<R, true>(v);
        } else {
            dft_any<R, false>(v);
            if (j != 0) {
#pragma unroll
                for (int q = 1; q < R; ++q) v[q] = cmul(v[q], ASARF_LDG(ctw + TWO + (q - 1) * S + j));
            }
        }
        if constexpr (Epi::kActive) {
#pragma unroll
            for (int m = 0; m < R; ++m) epi(b * M + j + m * S, v[m]);
        } else {
#pragma unroll
            for (int m = 0; m < R; ++m) p[m * STRIDE] = v[m];
        }
    }
}

// Last forward pass, matched filter, first inverse pass: blocks of R contiguous positions
// (span 1, no twiddles), all in registers.  mf is transposed: position b*R + q at q*(L/R) + b.
template <int L>
ASARF_HD ASARF_INLINE void ct_middle(float2* s, const float2* __restrict__ mf, int t) {
    constexpr int NTHR = CtSchedule<L>::nthr;
    constexpr int R = ct_padq<L>();
    constexpr int ITEMS = L / R;
    constexpr int PER = (ITEMS + NTHR - 1) / NTHR;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int b = t + k * NTHR;
        if (ITEMS % NTHR != 0 && b >= ITEMS) break;
        float2* p = s + b * (R + 1);  // padded position of b * R
        float2 v[R];
#pragma unroll
        for (int m = 0; m < R; ++m) v[m] = p[m];
        dft_any<R, false>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = cmul(v[q], ASARF_LDG(mf + q * ITEMS + b));
        dft_any<R, true>(v);
#pragma unroll
        for (int m = 0; m < R; ++m) p[m] = v[m];
    }
}

// Forward transform, matched filter, inverse transform (unscaled) through the padded tile s: the
// first pass takes its inputs from src (natural position), the last hands its outputs to epi
// (natural position, value) and ends without a barrier, every other pass ends with one.
// The samples are formed where they are first used: decoding the line into the tile and reading it
// back took a fifth of the kernel's shared-memory passes and a barrier (5616 x 28000, L = 6144:
// 1000 -> 926 us).
template <int L, class Src, class Epi>
ASARF_HD ASARF_INLINE void ct_fft_mf_ifft(float2* s, const float2* __restrict__ ctw, const float2* __restrict__ mf,
                                          int tid, const Src& src, const Epi& epi) {
    constexpr int NTHR = CtSchedule<L>::nthr;
    static_assert(CtSchedule<L>::count == 3, "three-pass schedules");
    static_assert(Epi::kActive, "the last pass writes through its epilogue");
    static_assert(Src::kActive, "the first pass reads through its source");
    ct_phase<NTHR>([&](int t) { ct_pass<L, 0, false>(s, ctw, t, NoEpi{}, src); }, tid);
    ct_phase<NTHR>([&](int t) { ct_pass<L, 1, false>(s, ctw, t); }, tid);
    ct_phase<NTHR>([&](int t) { ct_middle<L>(s, mf, t); }, tid);
    ct_phase<NTHR>([&](int t) { ct_pass<L, 1, true>(s, ctw, t); }, tid);
    ct_phase<NTHR, false>([&](int t) { ct_pass<L, 0, true>(s, ctw, t, epi); }, tid);
}

}  // namespace asarf
