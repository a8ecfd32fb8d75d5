// Strided azimuth kernel of one radix schedule ASARF_R0, ASARF_R1, ASARF_R2 (0, 0, 0: the run-time loops), tile width
// ASARF_XT and number of tiles ASARF_NB.
#include "bodies.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace asarf {

namespace {

// Strided azimuth pass: the [n1][NB][XT] tiles (rows r*n2 + b + k) arrive by 3-D TMA boxes.
// R0..R2 > 0: compile-time transform schedule (az_strided_body).
template <int R0, int R1, int R2, int XT, int NB>
__global__ void __launch_bounds__(256, 3) k_az_strided(AzStridedArgs a, const __grid_constant__ CUtensorMap map) {
    extern __shared__ __align__(128) unsigned char smem_as_raw[];
    float2* s = reinterpret_cast<float2*>(smem_as_raw);
    float2* tw = s + static_cast<size_t>(a.n1) * XT * NB;
    int* row = reinterpret_cast<int*>(tw + a.n1 * NB);
    __shared__ uint64_t bar;
    const int b = blockIdx.y * NB;
    if (a.use_tma && threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, static_cast<uint32_t>(sizeof(float2) * a.n1 * XT * NB));
        for (int r0 = 0; r0 < a.n1; r0 += a.n1_box)
            tma_load_3d(s + static_cast<size_t>(r0) * XT * NB, &map, &bar, 2 * blockIdx.x * XT, b, r0);
    }
    // twiddle and row tables are gathered while the tile is in flight
    az_strided_tables(a, b, threadIdx.x, blockDim.x, tw, row);
    __syncthreads();
    if (a.use_tma) mbar_wait(&bar, 0, a.state ? &const_cast<FocusState*>(a.state)->errors : nullptr);
    az_strided_body<R0, R1, R2, XT, NB>(a, blockIdx.x, b, threadIdx.x, blockDim.x, s, tw, row, a.use_tma != 0);
}

}  // namespace

template <int R0, int R1, int R2, int XT, int NB>
int launch_az_strided(const AzStridedArgs& a, const void* tmap, int tiles, LaunchShape sh, void* stream) {
    int rc = ensure_smem(k_az_strided<R0, R1, R2, XT, NB>, sh.smem, "az_strided");
    if (rc || tiles <= 0) return rc;
    k_az_strided<R0, R1, R2, XT, NB><<<dim3(tiles, (a.n2 + NB - 1) / NB), sh.threads, sh.smem, S(stream)>>>(
        a, tmap_or_zero(tmap));
    return check_launch("az_strided");
}

template int launch_az_strided<ASARF_R0, ASARF_R1, ASARF_R2, ASARF_XT, ASARF_NB>(const AzStridedArgs&, const void*, int,
                                                                                 LaunchShape, void*);

}  // namespace asarf
