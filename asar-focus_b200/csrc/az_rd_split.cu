// Split-precision range-Doppler kernel: the forward contiguous transform on the tensor cores.
#include "bodies.cuh"
#include "launch.cuh"
#include "tc.cuh"
#include "tma.cuh"

namespace asarf {

namespace {

// ----------------------------------------------------------------------------- split precision
// Forward transform of the range-Doppler tile on the tensor cores.  Tile s[l][c], l < n2 =
// R * m, c < wt.  Operand row rho = r * wt + c holds the sub-sequence x[r + R mm] (mm < m) of
// column c as bf16 hi + lo parts (K = (mm, re / im)); it multiplies the m-point DFT matrix B
// (hi + lo, output slot s = frequency k1(s)) as Ahi Bhi + Ahi Blo + Alo Bhi with FP32
// accumulation, and the result times W_n2^(r k1(s)) goes back to row r + R s of column c (a
// row of the same sub-sequence, already consumed).  The operands live in tensor memory
// beside the accumulator (TMEM columns [0, 64) accumulator, [64, 96) A hi, [96, 128) A lo),
// so shared memory holds only B and the tile and two blocks stay resident per SM, as in the
// FP32 kernel.  Rounds of 128 operand rows: warp w writes TMEM lanes 32 (w % 4) .., K chunk
// w / 4 (8 inputs), one thread issues the products, every thread reads back its lane.  A
// radix-R FP32 pass over rows R s .. R s + R - 1 then leaves frequency k1(s) + m k2 at row
// R s + k2: the digit-reversed order of the FP32 forward transform (k1(s) from that
// transform's order table).  Returns false (error bit set, products drained) if a product did
// not complete in time.
constexpr uint32_t kSplitColAcc = 0, kSplitColAHi = 64, kSplitColALo = 96;

__device__ bool split_forward(const AzRdArgs& a, const AzRdSplit& sp, float2* s, const unsigned char* b_hi,
                              const unsigned char* b_lo, uint32_t tmem, uint64_t* mbar, unsigned int* err) {
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int wt = a.wt, R = sp.radix, m = sp.m;
    const int rows = R * wt;
    const int q = warp & 3, jb = warp >> 2;  // TMEM lane quarter, K chunk / accumulator column block
    const uint32_t lane_base = static_cast<uint32_t>(32 * q) << 16;
    const FastDiv dwt = make_fastdiv(static_cast<unsigned int>(wt));
    constexpr uint32_t kIdesc = umma_idesc_bf16(kSplitRows, kSplitN);
    constexpr uint32_t kSbo = kSplitK * 16;  // 8 rows x K bf16
    (void)nthr;
    uint32_t phase = 0;
    for (int g0 = 0; g0 < rows; g0 += kSplitRows) {
        const int rho = g0 + 32 * q + lane;
        const bool live = rho < rows;
        int r = 0, c = 0;
        if (live) {
            r = static_cast<int>(fdiv_u(static_cast<unsigned int>(rho), dwt));
            c = rho - r * wt;
        }
        {
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int mm = 8 * jb + i;
                const float2 v = (live && mm < m) ? s[(r + R * mm) * wt + c] : make_float2(0.0f, 0.0f);
                split_bf16x2(v.x, v.y, hi[i], lo[i]);
            }
            tmem_st8(tmem + lane_base + kSplitColAHi + 8u * jb, hi);
            tmem_st8(tmem + lane_base + kSplitColALo + 8u * jb, lo);
            tmem_wait_st();
        }
        tc_fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after_sync();
            const uint32_t bh = smem_u32(b_hi), bl = smem_u32(b_lo);
#pragma unroll
            for (int ks = 0; ks < kSplitK / 16; ++ks) {
                const uint32_t o = 256u * ks;  // B: two 128-byte core-matrix columns per k-step
                const uint64_t dbh = umma_smem_desc(bh + o, 128, kSbo), dbl = umma_smem_desc(bl + o, 128, kSbo);
                const uint32_t ah = tmem + kSplitColAHi + 8u * ks, al = tmem + kSplitColALo + 8u * ks;
                umma_bf16_ts(tmem + kSplitColAcc, ah, dbh, kIdesc, ks > 0);
                umma_bf16_ts(tmem + kSplitColAcc, ah, dbl, kIdesc, true);
                umma_bf16_ts(tmem + kSplitColAcc, al, dbh, kIdesc, true);
            }
            umma_commit(mbar);
        }
        const bool done = mbar_wait(mbar, phase, nullptr);
        if (__syncthreads_or(!done)) {
            if (tid == 0) atomicOr(err, kErrMmaTimeout);
            mbar_wait(mbar, phase, nullptr);  // one more bounded wait for the products in flight
            return false;
        }
        phase ^= 1u;
        tc_fence_after_sync();
        // accumulator: this warp's lanes, columns 16 jb .. (output slots 8 jb ..)
        if (8 * jb < m) {  // warp-uniform
            float v[16];
            tmem_ld16(tmem + lane_base + kSplitColAcc + 16u * jb, v);
            if (live) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int slot = 8 * jb + i;
                    if (slot < m)
                        s[(r + R * slot) * wt + c] = cmul(make_float2(v[2 * i], v[2 * i + 1]), __ldg(sp.tw + r * m + slot));
                }
            }
        }
        tc_fence_before_sync();
        __syncthreads();
    }
    // radix-R DFT over r of every (slot, column pair): rows R * slot + r, no twiddles
    const int npair = wt >> 1;
    fft_stage_pair_w_dispatch<false, false, NoEpi, false>(R, s, a.n2, 1, make_fastdiv(1u), PairTasks(npair), wt,
                                                          a.plan2.tw, tid, blockDim.x);
    __syncthreads();
    return true;
}

__global__ void __launch_bounds__(512, 2) k_az_rd_split(AzRdArgs a, AzRdSplit sp, unsigned int* err,
                                                        const __grid_constant__ CUtensorMap map) {
    extern __shared__ __align__(128) unsigned char smem_rds_raw[];
    unsigned char* b_hi = smem_rds_raw;
    unsigned char* b_lo = b_hi + kSplitMatrixBytes;
    float2* s = reinterpret_cast<float2*>(b_lo + kSplitMatrixBytes);
    const int wt = a.wt;
    const AzRdTables t(a, s);
    __shared__ uint64_t bar, mbar;
    __shared__ uint32_t tmem_base;
    if (threadIdx.x < 32) tmem_alloc(&tmem_base, kSplitTmemCols);
    if (threadIdx.x == 0) {
        mbar_init(&mbar, 1);
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, static_cast<uint32_t>(sizeof(float2) * a.n2 * wt));
        const int x = 2 * (static_cast<int>(blockIdx.x) * a.xt - a.hl);
        for (int r0 = 0; r0 < a.n2; r0 += a.n2_box)
            tma_load_2d(s + static_cast<size_t>(r0) * wt, &map, &bar, x, blockIdx.y * a.n2 + r0);
    }
    // the DFT matrix images and the column / row tables while the tile is in flight
    const uint4* bsrc = reinterpret_cast<const uint4*>(sp.bmat);
    for (int i = threadIdx.x; i < 2 * kSplitMatrixBytes / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(b_hi)[i] = __ldg(bsrc + i);
    az_rd_tables(a, blockIdx.x, blockIdx.y, threadIdx.x, blockDim.x, t);
    fence_async_smem();  // B is read by the tensor cores
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_base;
    mbar_wait(&bar, 0, err);
    if (split_forward(a, sp, s, b_hi, b_lo, tmem, &mbar, err))
        az_rd_body<false>(a, blockIdx.x, blockIdx.y, threadIdx.x, blockDim.x, s, t, err, true);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (threadIdx.x < 32) tmem_dealloc(tmem, kSplitTmemCols);
}

}  // namespace

int backend_az_rd_split(const AzRdArgs& a, const AzRdSplit& sp, const void* tmap, int tiles, int nblocks,
                        LaunchShape sh, unsigned int* err, void* stream) {
    if (!tmap) return set_error(ASARF_ERR_INVALID, "az_rd_split: needs the TMA tile loads");
    int rc = ensure_smem(k_az_rd_split, sh.smem, "az_rd_split");
    if (rc || tiles <= 0) return rc;
    k_az_rd_split<<<dim3(tiles, nblocks), sh.threads, sh.smem, S(stream)>>>(a, sp, err, tmap_or_zero(tmap));
    return check_launch("az_rd_split");
}

}  // namespace asarf
