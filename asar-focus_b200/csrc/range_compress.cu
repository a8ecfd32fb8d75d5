// Range compression kernels of one FFT length: ASARF_LENGTH (a compile-time-scheduled one of kCtLengths, or 0
// for the run-time schedules).
#include "bodies.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace asarf {

namespace {

// Raw record of n bytes into shared memory: its 16-byte aligned interior by one bulk copy of thread 0,
// the bytes before and after it (records start and end anywhere) by plain loads, so nothing outside
// the record is read.  The copy starts at buf + (address mod 16), buf 16-byte aligned, which keeps
// the interior aligned in shared memory as well.  (Lines off 16-byte alignment decoded from global
// memory sample by sample, FBAQ4 records moved by vector loads: 17011 lines of 10386 bytes 803 ->
// 626 us, 30000 FBAQ4 records 1287 -> 1238 us.)
__device__ __forceinline__ const uint8_t* stage_record(uint8_t* buf, const uint8_t* rec, int n, uint64_t* bar,
                                                       unsigned int* err) {
    const int lead = static_cast<int>(reinterpret_cast<uintptr_t>(rec) & 15);
    const int head = min(n, (16 - lead) & 15);
    const int body = (n - head) & ~15;
    uint8_t* dst = buf + lead;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, static_cast<uint32_t>(body));
        if (body) bulk_load(dst + head, rec + head, static_cast<uint32_t>(body), bar);
    }
    for (int i = threadIdx.x; i < head; i += blockDim.x) dst[i] = rec[i];
    for (int i = head + body + threadIdx.x; i < n; i += blockDim.x) dst[i] = rec[i];
    __syncthreads();
    mbar_wait(bar, 0, err);
    return dst;
}

// One raw line per block.
template <int FMT>
__device__ __forceinline__ const uint8_t* stage_line(const RangeCompressArgs& a, unsigned char* smem, uint64_t* bar) {
    const int n = FMT == kRawAsarFbaq4 ? static_cast<int>(a.line_bytes) : 2 * a.spl;
    return stage_record(smem + a.raw_smem_offset, a.raw + static_cast<long long>(blockIdx.x) * a.line_bytes, n, bar,
                        &const_cast<FocusState*>(a.state)->errors);
}

#if ASARF_LENGTH == 0
template <int FMT>
__global__ void __launch_bounds__(512) k_range_compress(RangeCompressArgs a) {
    extern __shared__ __align__(128) unsigned char smem_rc_raw[];
    __shared__ uint64_t bar;
    const uint8_t* line = stage_line<FMT>(a, smem_rc_raw, &bar);
    range_compress_body<FMT>(a, blockIdx.x, threadIdx.x, blockDim.x, reinterpret_cast<float2*>(smem_rc_raw), line);
}

__global__ void __launch_bounds__(512) k_rc_rows(RcRowsArgs a) {
    extern __shared__ float2 smem_rcr[];
    rc_rows_body(a, blockIdx.x, threadIdx.x, blockDim.x, smem_rcr);
}

template <int FMT>
int launch_format(const RangeCompressArgs& a, int lines, LaunchShape sh, void* stream) {
    int rc = ensure_smem(k_range_compress<FMT>, sh.smem, "range_compress");
    if (rc || lines <= 0) return rc;
    k_range_compress<FMT><<<lines, sh.threads, sh.smem, S(stream)>>>(a);
    return check_launch("range_compress");
}
#else
// Compile-time-scheduled variant (L in kCtLengths).
template <int L, int FMT>
__global__ void __launch_bounds__(CtSchedule<L>::nthr, CtSchedule<L>::blocks) k_range_compress_ct(RangeCompressArgs a) {
    extern __shared__ __align__(128) unsigned char smem_rcc_raw[];
    __shared__ uint64_t bar;
    const uint8_t* line = stage_line<FMT>(a, smem_rcc_raw, &bar);
    range_compress_ct_body<L, FMT>(a, blockIdx.x, threadIdx.x, reinterpret_cast<float2*>(smem_rcc_raw), line);
}

template <int L>
__global__ void __launch_bounds__(CtSchedule<L>::nthr, CtSchedule<L>::blocks) k_rc_rows_ct(RcRowsArgs a) {
    extern __shared__ float2 smem_rcrc[];
    rc_rows_ct_body<L>(a, blockIdx.x, threadIdx.x, smem_rcrc);
}

template <int FMT>
int launch_format(const RangeCompressArgs& a, int lines, LaunchShape sh, void* stream) {
    constexpr int L = ASARF_LENGTH;
    int rc = ensure_smem(k_range_compress_ct<L, FMT>, sh.smem, "range_compress");
    if (rc || lines <= 0) return rc;
    k_range_compress_ct<L, FMT><<<lines, CtSchedule<L>::nthr, sh.smem, S(stream)>>>(a);
    return check_launch("range_compress");
}
#endif

}  // namespace

template <>
int launch_range_compress<ASARF_LENGTH>(const RangeCompressArgs& a, int lines, LaunchShape sh, void* stream) {
    if (a.format == kRawAsarFbaq4) return launch_format<kRawAsarFbaq4>(a, lines, sh, stream);
    return launch_format<kRawErsBytes>(a, lines, sh, stream);
}

template <>
int launch_rc_rows<ASARF_LENGTH>(const RcRowsArgs& a, int rows, LaunchShape sh, void* stream) {
#if ASARF_LENGTH == 0
    int rc = ensure_smem(k_rc_rows, sh.smem, "rc_rows");
    if (rc) return rc;
    k_rc_rows<<<rows, sh.threads, sh.smem, S(stream)>>>(a);
#else
    constexpr int L = ASARF_LENGTH;
    int rc = ensure_smem(k_rc_rows_ct<L>, sh.smem, "rc_rows");
    if (rc) return rc;
    k_rc_rows_ct<L><<<rows, CtSchedule<L>::nthr, sh.smem, S(stream)>>>(a);
#endif
    return check_launch("rc_rows");
}

}  // namespace asarf
