// CUDA kernels of the focusing path (sm_100a) and their launchers: statistics, finalisation, tail, records and the
// per-stage kernels.  The transform kernels are in range_compress.cu, az_strided.cu, az_rd.cu and az_rd_split.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "asarf.h"
#include "backend.h"
#include "bodies.cuh"
#include "context_cache.h"
#include "launch.cuh"
#include "tma.cuh"

namespace asarf {

namespace {

constexpr int kFinalizeThreads = 96;
static_assert(kFinalizeThreads >= kMaxDcBlocks, "one Doppler block per thread");

// Statistics lines through the ring of batches.  The warps take turns to issue one: lane u copies the bytes of
// line u under the block's columns, from the 16-byte boundary before its first to the one after its
// last; at the two ends of the raw buffer, where that would leave it, the odd bytes are moved by plain
// loads.  A batch is issued into its slots once every thread has read the one they held.
struct StatsRowsStaged {
    static constexpr bool kCollective = true;
    static constexpr int kMargin = 0;  // the words around a window stay inside its slot
    const RawStatsArgs& a;
    RawStatsSmem* sm;
    const StatsBatches& bt;
    unsigned char* ring;
    __device__ __forceinline__ void issue(int k) const {
        if (k >= bt.count) return;
        const int lane = threadIdx.x & 31, stage = k % kStatsStages, slot = stage * kStatsBatch + lane;
        int yg, ye;
        bt.lines(k, &yg, &ye);
        const int y = yg + lane;
        uint32_t bytes = 0;
        const uint8_t* src = nullptr;
        unsigned char* dst = nullptr;
        if (lane < kStatsBatch && y < ye) {
            const StatsSlotCopy c(a, y, sm->off[y - bt.ys], sm->x_lo, sm->x_hi);
            unsigned char* base = ring + slot * kStatsSlotBytes;
            c.plain(base);
            if (c.c0 < c.c1) {
                bytes = static_cast<uint32_t>(c.c1 - c.c0);
                src = c.c0;
                dst = base + c.lead + (c.c0 - c.b0);
            }
            sm->sample0[slot] = slot * kStatsSlotBytes + c.sample0;
        }
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) mbar_expect_tx(&sm->full[stage], total);
        __syncwarp();
        fence_async_smem();
        if (bytes) bulk_load(dst, src, bytes, &sm->full[stage]);
    }
    __device__ __forceinline__ void begin(int k) const {
        mbar_wait(&sm->full[k % kStatsStages], (k / kStatsStages) & 1, &a.acc->errors);
    }
    __device__ __forceinline__ void end(int k) const {
        __syncthreads();
        if (static_cast<int>(threadIdx.x >> 5) == k % (kStatsCols / 32)) issue(k + kStatsStages);
    }
    __device__ __forceinline__ const uint8_t* row(int k, int u, int) const {
        return ring + sm->sample0[k % kStatsStages * kStatsBatch + u];
    }
};

// Lines on 8-byte boundaries: every window is one 8-byte load, read in place.  Three blocks per SM (80
// registers): four blocks at 64 registers spilled 176 bytes per thread in the batched loads and
// measured slower, 0.156 against 0.143 ms.
__global__ void __launch_bounds__(kStatsCols, kStatsBlocksPerSm) k_raw_stats(RawStatsArgs a) {
    __shared__ RawStatsSmem sm;
    const StatsBatches bt = raw_stats_begin(a, blockIdx.y, threadIdx.x, kStatsCols, &sm);
    __syncthreads();
    raw_stats_body<true>(a, StatsRowsInPlace<true>{a}, bt, blockIdx.x, threadIdx.x, kStatsCols, &sm);
}

// Any other lines, through the ring (three blocks per SM by their rings, too).
__global__ void __launch_bounds__(kStatsCols, kStatsBlocksPerSm) k_raw_stats_ring(RawStatsArgs a) {
    extern __shared__ __align__(128) unsigned char smem_rs_raw[];
    __shared__ RawStatsSmem sm;
    const int tid = threadIdx.x;
    const StatsBatches bt = raw_stats_begin(a, blockIdx.y, tid, kStatsCols, &sm);
    if (tid == 0) {
        for (int i = 0; i < kStatsStages; ++i) mbar_init(&sm.full[i], 1);
        sm.x_lo = 0x3fffffff;  // no unit: past every record
        sm.x_hi = 0;
    }
    __syncthreads();
    const StatsUnit un(a, make_fastdiv(static_cast<unsigned int>(a.gpb)), blockIdx.x * kStatsCols + tid);
    if (un.colmask) {
        atomicMin(&sm.x_lo, un.x0);
        atomicMax(&sm.x_hi, un.x0 + 4);
    }
    __syncthreads();
    const StatsRowsStaged rows{a, &sm, bt, smem_rs_raw};
    if (tid < 32)
        for (int k = 0; k < kStatsStages; ++k) rows.issue(k);
    __syncthreads();
    raw_stats_body<false>(a, rows, bt, blockIdx.x, tid, kStatsCols, &sm);
}

// Which tile rows of the statistics have records of one shift and length (every column tile would
// otherwise read all its records' length fields, a 32-byte sector each).
__global__ void __launch_bounds__(1024) k_fbaq_uniform(RawStatsArgs a) {
    const int ys = fbaq_tile_start(blockIdx.x);
    const int y1 = min((static_cast<int>(blockIdx.x) + 1) * kFbaqStatsLines, a.na);
    const int off = a.swst ? static_cast<int>(a.swst[ys]) - a.min_swst : 0;
    const int len = fbaq_len(a.raw + static_cast<long long>(ys) * a.line_bytes, a.line_bytes);
    bool same = true;
    for (int y = ys + threadIdx.x; y < y1; y += 1024) same = same && fbaq_line_like(a, y, off, len);
    same = __syncthreads_and(same) != 0;
    if (threadIdx.x == 0) a.uniform[blockIdx.x] = same ? 1 : 0;
}

__global__ void __launch_bounds__(32 * kFbaqStatsWarps, 4) k_raw_stats_fbaq(RawStatsArgs a) {
    __shared__ FbaqStatsSmem sm;
    raw_stats_fbaq_body(a, blockIdx.x, blockIdx.y, threadIdx.x, blockDim.x, &sm);
}

__global__ void __launch_bounds__(1024) k_stats_fold(RawStatsArgs a, int tiles_y) {
    __shared__ double tree[6 * kFoldTree];
    stats_fold_body(a, tiles_y, threadIdx.x, blockDim.x, tree);
}

__global__ void __launch_bounds__(256) k_product_stats(ProductStatsArgs a) {
    __shared__ double red[5 * 256];
    product_stats_body(a, blockIdx.x, threadIdx.x, blockDim.x, red);
}

__global__ void __launch_bounds__(1024) k_product_stats_fold(ProductStatsArgs a) {
    __shared__ double tree[5 * kStatsFoldLeaves];
    product_stats_fold(a, threadIdx.x, blockDim.x, tree);
}

__global__ void __launch_bounds__(256) k_condition(ConditionArgs a) {
    condition_row(a, blockIdx.x, threadIdx.x, blockDim.x);
}

// Quadratic least-squares fit through nblk <= kMaxDcBlocks points by one warp: the Householder
// steps of polyfit_qr with row r on lane r % 32, every sum of a step reduced over the lanes at once
// (fixed order, the same on every lane).  Coefficients highest power first, on every lane.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ bool warp_fit_quadratic(const double* xs, const double* ys, int nblk, double out[3]) {
    constexpr int kRows = (kMaxDcBlocks + 31) / 32;
    const int lane = threadIdx.x & 31;
    if (nblk < 3) return false;
    double A[4][kRows];  // columns 1, x, x^2 and the right-hand side; rows past the last are zero
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int r = lane + 32 * i;
        const bool ok = r < nblk;
        const double x = ok ? xs[r] : 0.0;
        A[0][i] = ok ? 1.0 : 0.0;
        A[1][i] = x;
        A[2][i] = x * x;
        A[3][i] = ok ? ys[r] : 0.0;
    }
    double R[3][4];  // rows of the triangular system
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // sums over rows r > k of column k times each column from k on
        double dot[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < kRows; ++i)
            if (lane + 32 * i > k)
#pragma unroll
                for (int c = k; c < 4; ++c) dot[c] += A[k][i] * A[c][i];
#pragma unroll
        for (int c = k; c < 4; ++c) dot[c] = warp_sum(dot[c]);
        double head[4];
#pragma unroll
        for (int c = k; c < 4; ++c) head[c] = __shfl_sync(0xffffffffu, A[c][0], k);
        const double nrm = sqrt(head[k] * head[k] + dot[k]);
        if (nrm == 0.0) return false;
        const double alpha = head[k] > 0 ? -nrm : nrm;
        const double vk = head[k] - alpha;
        const double vn = vk * vk + dot[k];
        if (vn == 0.0) return false;
        R[k][k] = alpha;
#pragma unroll
        for (int c = k + 1; c < 4; ++c) {
            const double f = 2.0 * (vk * head[c] + dot[c]) / vn;
            R[k][c] = head[c] - f * vk;
#pragma unroll
            for (int i = 0; i < kRows; ++i)
                if (lane + 32 * i > k) A[c][i] -= f * A[k][i];
        }
    }
    const double c2 = R[2][3] / R[2][2];
    const double c1 = (R[1][3] - R[1][2] * c2) / R[1][1];
    const double c0 = (R[0][3] - R[0][1] * c1 - R[0][2] * c2) / R[0][0];
    out[0] = c2, out[1] = c1, out[2] = c0;
    return true;
}

// The Doppler blocks' angles (an FP64 atan2 each) one per thread, the statistics' own results on
// the last warp beside them, the fit over warp 0 (by one thread's serial QR the kernel took 16 us
// in every focus run, whatever the scene, and now 6; a chain of latencies, not work).  The accumulators are
// zeroed for the plan's next run once every thread has read them.
__global__ void __launch_bounds__(kFinalizeThreads) k_finalize(FinalizeArgs a) {
    __shared__ double xs[kMaxDcBlocks], ys[kMaxDcBlocks];
    if (blockIdx.x != 0) return;
    FocusState& st = *a.state;
    const int tid = threadIdx.x;
    const FinalizeMap m = finalize_stats(a, tid == kFinalizeThreads - 1 ? &st : nullptr);
    const int nblk = a.nblk < kMaxDcBlocks ? a.nblk : kMaxDcBlocks;
    if (tid < nblk) finalize_block(a, m, tid, xs, ys, st);
    __syncthreads();
    if (!a.facc) {
        unsigned long long* acc = &a.acc->mom[0];
        for (int i = tid; i < 6 + 9 * nblk; i += kFinalizeThreads) acc[i] = 0ull;
        if (tid == 0) a.acc->errors = 0u;
    }
    if (tid < 32) {
        double poly[3] = {0.0, 0.0, 0.0};
        if (!warp_fit_quadratic(xs, ys, nblk, poly)) poly[0] = poly[1] = poly[2] = 0.0;
        if (tid == 0) finalize_poly(a, st, poly, m.err);
    }
}

__global__ void __launch_bounds__(128) k_rcmc_table(float* table) {
    const int n = blockIdx.x * 128 + threadIdx.x;
    if (n <= kRcmcNodes) rcmc_weight_row(n, table + static_cast<size_t>(n) * kRcmcRowFloats);
}

__global__ void __launch_bounds__(512, 2) k_tail(TailArgs a, unsigned int* err) {
    extern __shared__ float smem_tail[];
    tail_body(a, blockIdx.x, threadIdx.x, blockDim.x, smem_tail, err);
}

template <class Args, void (*Item)(const Args&, long long)>
__global__ void __launch_bounds__(256) k_items(Args a, long long n) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        Item(a, i);
}

__global__ void __launch_bounds__(256) k_decode(DecodeArgs a) { decode_row(a, blockIdx.x, threadIdx.x, 256); }

__global__ void __launch_bounds__(256) k_decode_fbaq(DecodeFbaqArgs a) {
    decode_fbaq_row(a, blockIdx.x, threadIdx.x, 256);
}

__global__ void __launch_bounds__(256) k_zero_nans(float2* img, long long n) {
    const long long step = static_cast<long long>(gridDim.x) * 256;
#pragma unroll 4
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += step) zero_nan_item(img, i);
}

template <bool ABOUT>
__global__ void __launch_bounds__(256) k_img_moments(ImgMomentsArgs a) {
    __shared__ double red[12 * 256];
    img_moments_body<ABOUT>(a, blockIdx.x, threadIdx.x, 256, red);
}

__global__ void __launch_bounds__(kAcccCols) k_accc(AcccArgs a) {
    __shared__ double cols[2 * kAcccCols];
    accc_body(a, blockIdx.x, blockIdx.y, gridDim.x, threadIdx.x, kAcccCols, cols);
}

// Matched filter: eight threads share a position's sum.
__global__ void __launch_bounds__(256) k_matched_filter(MatchedFilterArgs a) {
    const int pos = blockIdx.x * 32 + (threadIdx.x >> 3);
    double re = 0.0, im = 0.0;
    if (pos < a.plan.n) matched_filter_sum(a, pos, threadIdx.x & 7, 8, &re, &im);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (pos < a.plan.n && (threadIdx.x & 7) == 0) matched_filter_store(a, pos, re, im);
}

__global__ void __launch_bounds__(128) k_twiddles(TwiddleArgs a, int count) {
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i < count) twiddle_item(a, i);
}

__global__ void __launch_bounds__(128) k_rsl(RslArgs a) {
    const int x = blockIdx.x * 128 + threadIdx.x;
    if (x >= a.range_size) return;
    for (long long y0 = blockIdx.y * kColumnRows; y0 < a.az_size; y0 += gridDim.y * kColumnRows)
        rsl_column(a, x, static_cast<int>(y0), static_cast<int>(min(y0 + kColumnRows, static_cast<long long>(a.az_size))));
}

__global__ void __launch_bounds__(128) k_srgr(SrgrArgs a) {
    const int x = blockIdx.x * 128 + threadIdx.x;
    if (x >= a.out_x) return;
    for (long long y0 = blockIdx.y * kColumnRows; y0 < a.y_size; y0 += gridDim.y * kColumnRows)
        srgr_column(a, x, static_cast<int>(y0), static_cast<int>(min(y0 + kColumnRows, static_cast<long long>(a.y_size))));
}

// Level-0 gathers: one warp per line, eight lines per block.  A line's own loads form a chain
// (its offset, its header, its data), so what matters is how many lines an SM has in flight: a block
// per line kept 8 of them, a warp per line keeps up to 32.  28000 ERS lines (630 MB moved): 2-byte
// words 297 us, 16-byte units with a block per line 131, with a warp per line 104 (6.0 TB/s);
// 30000 ASAR records of 5288 bytes (318 MB): single bytes 291 us, 114, 59 (5.4 TB/s).
constexpr int kUnpackLines = 8;
__global__ void __launch_bounds__(32 * kUnpackLines) k_ers_unpack(ErsUnpackArgs a) {
    const int y = blockIdx.x * kUnpackLines + (threadIdx.x >> 5);
    if (y < a.lines) ers_unpack_line(a, y, threadIdx.x & 31, 32);
}

__global__ void __launch_bounds__(32 * kUnpackLines) k_asar_unpack(AsarUnpackArgs a) {
    const int y = blockIdx.x * kUnpackLines + (threadIdx.x >> 5);
    if (y < a.lines) asar_unpack_line(a, y, threadIdx.x & 31, 32);
}

__global__ void __launch_bounds__(256) k_multilook(MultilookArgs a) {
    multilook_row_body(a, blockIdx.x, threadIdx.x, blockDim.x);
}

int grid_for(long long n) {
    long long g = (n + 255) / 256;
    return static_cast<int>(g < 148 * 32 ? (g > 0 ? g : 1) : 148 * 32);
}

// Grid height of the column kernels, whose blocks stride over the rows past it.
int column_blocks(int rows) { return static_cast<int>(std::min((rows + kColumnRows - 1ll) / kColumnRows, 1ll * kMaxGridY)); }

}  // namespace

int backend_raw_stats(const RawStatsArgs& a, int gx, int gy, void* stream) {
    // lines of 11232 bytes (28000): in place 113 us, through the ring 124; of 10386 (17011): 212 (three
    // loads a window instead of one, and the line's checks) and 118
    if (a.aligned) {
        k_raw_stats<<<dim3(gx, gy), kStatsCols, 0, S(stream)>>>(a);
    } else {
        int rc = ensure_smem(k_raw_stats_ring, kStatsRingBytes, "raw_stats");
        if (rc) return rc;
        k_raw_stats_ring<<<dim3(gx, gy), kStatsCols, kStatsRingBytes, S(stream)>>>(a);
    }
    return check_launch("raw_stats");
}

int backend_finalize(const FinalizeArgs& a, void* stream) {
    k_finalize<<<1, kFinalizeThreads, 0, S(stream)>>>(a);
    return check_launch("finalize");
}

int backend_raw_stats_fbaq(const RawStatsArgs& a, int gx, int gy, void* stream) {
    k_fbaq_uniform<<<gy, 1024, 0, S(stream)>>>(a);
    int rc = check_launch("fbaq_uniform");
    if (rc) return rc;
    k_raw_stats_fbaq<<<dim3(gx, gy), 32 * kFbaqStatsWarps, 0, S(stream)>>>(a);
    return check_launch("raw_stats_fbaq");
}

int backend_stats_fold(const RawStatsArgs& a, int tiles_y, void* stream) {
    k_stats_fold<<<1, 1024, 0, S(stream)>>>(a, tiles_y);
    return check_launch("stats_fold");
}

int backend_range_compress(const RangeCompressArgs& a, int lines, LaunchShape sh, void* stream) {
#define ASARF_CASE(L) \
    if (a.plan.n == L) return launch_range_compress<L>(a, lines, sh, stream);
    ASARF_CT_LENGTHS(ASARF_CASE)
#undef ASARF_CASE
    return launch_range_compress<0>(a, lines, sh, stream);
}

// The compiled schedules (strided_schedule_compiled) when the plan allows them.
int backend_az_strided(const AzStridedArgs& a, const void* tmap, int tiles, LaunchShape sh, void* stream) {
    if (a.compiled && a.nb == 1 && strided_schedule_compiled(a.plan1, a.xt)) {
#define ASARF_CASE(R0, R1, R2) \
    if (plan_is(a.plan1, R0, R1, R2)) return launch_az_strided<R0, R1, R2, 32, 1>(a, tmap, tiles, sh, stream);
        ASARF_STRIDED_SCHEDULES(ASARF_CASE)
#undef ASARF_CASE
    }
    if (a.xt == 16) return launch_az_strided<0, 0, 0, 16, 1>(a, tmap, tiles, sh, stream);
    if (a.nb == 2) return launch_az_strided<0, 0, 0, 32, 2>(a, tmap, tiles, sh, stream);
    if (a.nb == 4) return launch_az_strided<0, 0, 0, 32, 4>(a, tmap, tiles, sh, stream);
    if (a.nb == 8) return launch_az_strided<0, 0, 0, 32, 8>(a, tmap, tiles, sh, stream);
    return launch_az_strided<0, 0, 0, 32, 1>(a, tmap, tiles, sh, stream);
}

// The compiled schedules (block_schedule_compiled) when the plan allows them.
int backend_az_rd(const AzRdArgs& a, const void* tmap, int tiles, int nblocks, LaunchShape sh, unsigned int* err,
                  void* stream) {
    if (a.compiled && block_schedule_compiled(a.plan2)) {
#define ASARF_CASE(R0, R1, R2) \
    if (plan_is(a.plan2, R0, R1, R2)) return launch_az_rd<R0, R1, R2>(a, tmap, tiles, nblocks, sh, err, stream);
        ASARF_BLOCK_SCHEDULES(ASARF_CASE)
#undef ASARF_CASE
    }
    return launch_az_rd<0, 0, 0>(a, tmap, tiles, nblocks, sh, err, stream);
}

int backend_rcmc_table(float* table, void* stream) {
    k_rcmc_table<<<kRcmcNodes / 128 + 1, 128, 0, S(stream)>>>(table);
    return check_launch("rcmc_table");
}

int backend_make_tmap(void* out, int rank, void* base, const unsigned long long* dims,
                      const unsigned long long* strides, const unsigned int* box) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn) {
            cudaGetLastError();
            return set_error(ASARF_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        }
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    cuuint64_t gdim[5], gstr[4];
    cuuint32_t bdim[5], estr[5];
    for (int i = 0; i < rank; ++i) {
        gdim[i] = dims[i];
        bdim[i] = box[i];
        estr[i] = 1;
    }
    for (int i = 0; i + 1 < rank; ++i) gstr[i] = strides[i];
    CUresult r = encode(static_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, rank, base, gdim, gstr, bdim,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(ASARF_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
    return ASARF_OK;
}

int backend_tail(const TailArgs& a, int rows, LaunchShape sh, unsigned int* err, void* stream) {
    int rc = ensure_smem(k_tail, sh.smem, "tail");
    if (rc) return rc;
    k_tail<<<rows, sh.threads, sh.smem, S(stream)>>>(a, err);
    return check_launch("tail");
}

int backend_decode(const DecodeArgs& a, void* stream) {
    k_decode<<<a.lines, 256, 0, S(stream)>>>(a);
    return check_launch("decode");
}
int backend_product_stats(const ProductStatsArgs& a, void* stream) {
    k_product_stats<<<a.blocks, 256, 0, S(stream)>>>(a);
    int rc = check_launch("product_stats");
    if (rc) return rc;
    k_product_stats_fold<<<1, 1024, 0, S(stream)>>>(a);
    return check_launch("product_stats_fold");
}
int backend_condition(const ConditionArgs& a, int rows, void* stream) {
    if (rows <= 0) return ASARF_OK;
    k_condition<<<rows, 256, 0, S(stream)>>>(a);
    return check_launch("condition");
}
int backend_decode_fbaq(const DecodeFbaqArgs& a, void* stream) {
    k_decode_fbaq<<<a.lines, 256, 0, S(stream)>>>(a);
    return check_launch("decode_fbaq");
}
int backend_img_moments(const ImgMomentsArgs& a, int blocks, void* stream) {
    if (a.about) k_img_moments<true><<<blocks, 256, 0, S(stream)>>>(a);
    else k_img_moments<false><<<blocks, 256, 0, S(stream)>>>(a);
    return check_launch("img_moments");
}
int backend_iq_apply(const IqApplyArgs& a, long long n, void* stream) {
    k_items<IqApplyArgs, iq_apply_item><<<grid_for(n), 256, 0, S(stream)>>>(a, n);
    return check_launch("iq_apply");
}
int backend_zero_nans(float2* img, long long n, void* stream) {
    k_zero_nans<<<grid_for(n), 256, 0, S(stream)>>>(img, n);
    return check_launch("zero_nans");
}
int backend_accc(const AcccArgs& a, int grid_x, int grid_y, void* stream) {
    k_accc<<<dim3(grid_x, grid_y), kAcccCols, 0, S(stream)>>>(a);
    return check_launch("accc");
}

int backend_rc_rows(const RcRowsArgs& a, int rows, LaunchShape sh, void* stream) {
#define ASARF_CASE(L) \
    if (a.ctw && a.plan.n == L) return launch_rc_rows<L>(a, rows, sh, stream);
    ASARF_CT_LENGTHS(ASARF_CASE)
#undef ASARF_CASE
    return launch_rc_rows<0>(a, rows, sh, stream);
}

int backend_matched_filter(const MatchedFilterArgs& a, void* stream) {
    k_matched_filter<<<(a.plan.n + 31) / 32, 256, 0, S(stream)>>>(a);
    return check_launch("matched_filter");
}

int backend_twiddles(const TwiddleArgs& a, void* stream) {
    const int count = twiddle_count(a);
    k_twiddles<<<(count + 127) / 128, 128, 0, S(stream)>>>(a, count);
    return check_launch("twiddles");
}
int backend_ers_unpack(const ErsUnpackArgs& a, void* stream) {
    if (a.lines <= 0) return ASARF_OK;
    k_ers_unpack<<<(a.lines + kUnpackLines - 1) / kUnpackLines, 32 * kUnpackLines, 0, S(stream)>>>(a);
    return check_launch("ers_unpack");
}

int backend_asar_unpack(const AsarUnpackArgs& a, void* stream) {
    if (a.lines <= 0) return ASARF_OK;
    k_asar_unpack<<<(a.lines + kUnpackLines - 1) / kUnpackLines, 32 * kUnpackLines, 0, S(stream)>>>(a);
    return check_launch("asar_unpack");
}
int backend_multilook(const MultilookArgs& a, void* stream) {
    k_multilook<<<a.out_y, 256, 0, S(stream)>>>(a);
    return check_launch("multilook");
}
int backend_rsl(const RslArgs& a, void* stream) {
    k_rsl<<<dim3((a.range_size + 127) / 128, column_blocks(a.az_size)), 128, 0, S(stream)>>>(a);
    return check_launch("rsl");
}
int backend_srgr(const SrgrArgs& a, void* stream) {
    k_srgr<<<dim3((a.out_x + 127) / 128, column_blocks(a.y_size)), 128, 0, S(stream)>>>(a);
    return check_launch("srgr");
}

void* mem_alloc(size_t bytes) {
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void mem_free(void* p) {
    if (p) cudaFree(p);
}

// The library's scratch pool of the current context (keyed by the context's id, as a pool made before a
// device reset must not be used after it), or null.
static cudaMemPool_t scratch_pool() {
    static ContextAddressCache<64> pools;
    unsigned long long id = 0;
    if (current_context_id(&id) != ASARF_OK || id == 0) return nullptr;
    void* pool = nullptr;
    pools.get(id, [](void** out) {
        int dev = 0, supported = 0;
        cudaGetDevice(&dev);
        cudaMemPool_t made = nullptr;
        if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && supported) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            unsigned long long keep = kScratchKept;
            if (cudaMemPoolCreate(&made, &props) != cudaSuccess) made = nullptr;
            if (made && cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
                cudaMemPoolDestroy(made);
                made = nullptr;
            }
        }
        cudaGetLastError();
        *out = made;
        return 0;
    }, &pool);
    return static_cast<cudaMemPool_t>(pool);
}

void* scratch_alloc(size_t bytes, void* stream, bool* pooled) {
    void* p = nullptr;
    cudaMemPool_t pool = scratch_pool();
    *pooled = pool && cudaMallocFromPoolAsync(&p, bytes, pool, S(stream)) == cudaSuccess;
    if (*pooled) return p;
    cudaGetLastError();
    return mem_alloc(bytes);
}

void scratch_free(void* p, void* stream, bool pooled) {
    if (!p) return;
    if (pooled) cudaFreeAsync(p, S(stream));
    else cudaFree(p);
}

static int cuda_rc(cudaError_t e, const char* what) {
    if (e != cudaSuccess) return set_error(ASARF_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return ASARF_OK;
}

int mem_h2d(void* dst, const void* src, size_t n, void* stream) {
    return cuda_rc(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, S(stream)), "H2D copy");
}
int mem_d2h(void* dst, const void* src, size_t n, void* stream) {
    return cuda_rc(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, S(stream)), "D2H copy");
}
int mem_d2d(void* dst, const void* src, size_t n, void* stream) {
    return cuda_rc(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToDevice, S(stream)), "D2D copy");
}
int mem_d2d_2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t rows, void* stream) {
    return cuda_rc(cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows, cudaMemcpyDeviceToDevice, S(stream)),
                   "2D D2D copy");
}
int mem_zero(void* dst, size_t n, void* stream) {
    return cuda_rc(cudaMemsetAsync(dst, 0, n, S(stream)), "memset");
}
int mem_zero_2d(void* dst, size_t pitch, size_t width, size_t rows, void* stream) {
    if (width == 0 || rows == 0) return ASARF_OK;
    return cuda_rc(cudaMemset2DAsync(dst, pitch, 0, width, rows, S(stream)), "2D memset");
}
bool stream_capturing(void* stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(S(stream), &st) != cudaSuccess) {
        cudaGetLastError();  // the legacy stream beside another's capture: not capturing itself
        return false;
    }
    return st != cudaStreamCaptureStatusNone;
}
int stream_sync(void* stream) { return cuda_rc(cudaStreamSynchronize(S(stream)), "stream sync"); }

void* event_create() {
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return e;
}
void event_destroy(void* e) {
    if (e) cudaEventDestroy(static_cast<cudaEvent_t>(e));
}
int event_record(void* e, void* stream) {
    return cuda_rc(cudaEventRecord(static_cast<cudaEvent_t>(e), S(stream)), "event record");
}
int event_elapsed(void* a, void* b, float* ms) {
    cudaError_t e = cudaEventSynchronize(static_cast<cudaEvent_t>(b));
    if (e == cudaSuccess) e = cudaEventElapsedTime(ms, static_cast<cudaEvent_t>(a), static_cast<cudaEvent_t>(b));
    return cuda_rc(e, "event elapsed");
}

int event_sync(void* e) { return cuda_rc(cudaEventSynchronize(static_cast<cudaEvent_t>(e)), "event sync"); }

void* stream_create() {
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return s;
}
void stream_destroy(void* s) {
    if (s) cudaStreamDestroy(static_cast<cudaStream_t>(s));
}
int stream_wait_event(void* stream, void* event) {
    return cuda_rc(cudaStreamWaitEvent(S(stream), static_cast<cudaEvent_t>(event), 0), "stream wait");
}
bool graphs_supported() { return true; }
int graph_capture_begin(void* stream) {
    return cuda_rc(cudaStreamBeginCapture(S(stream), cudaStreamCaptureModeRelaxed), "begin capture");
}
int graph_capture_end(void* stream, void** exec) {
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(S(stream), &g);
    if (e != cudaSuccess) return cuda_rc(e, "end capture");
    cudaGraphExec_t x = nullptr;
    e = cudaGraphInstantiate(&x, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_rc(e, "graph instantiate");
    *exec = x;
    return ASARF_OK;
}
int graph_launch(void* exec, void* stream) {
    return cuda_rc(cudaGraphLaunch(static_cast<cudaGraphExec_t>(exec), S(stream)), "graph launch");
}
void graph_destroy(void* exec) {
    if (exec) cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(exec));
}

size_t smem_optin_limit() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 227 * 1024;
    }
    return static_cast<size_t>(v);
}

int backend_sm_count() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
        cudaGetLastError();
        return 148;
    }
    return v;
}

const char* backend_name() { return "cuda-sm100a"; }

}  // namespace asarf
