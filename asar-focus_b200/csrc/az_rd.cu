// Range-Doppler kernel of one radix schedule ASARF_R0, ASARF_R1, ASARF_R2 (0, 0, 0: the run-time loops).
#include "bodies.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace asarf {

namespace {

// Range-Doppler block: the [n2][wt] tile (contiguous rows, range halo) arrives by 2-D TMA
// boxes; columns left of 0 and right of nk are filled with zeros by the TMA unit.
// R0..R2 > 0: compile-time radix schedule of the n2 transforms (az_rd_body).
template <int R0, int R1, int R2>
__global__ void __launch_bounds__(512, 2) k_az_rd(AzRdArgs a, unsigned int* err, const __grid_constant__ CUtensorMap map) {
    // (128-byte alignment: a larger one pads the static barrier below to as much, and two blocks
    // of kAzRdTwoBlockSmem bytes would no longer fit)
    extern __shared__ __align__(128) unsigned char smem_rd_raw[];
    const int wt = a.wt;
    float2* s = reinterpret_cast<float2*>(smem_rd_raw);
    const AzRdTables t(a, s);
    __shared__ uint64_t bar;
    if (a.use_tma && threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, static_cast<uint32_t>(sizeof(float2) * a.n2 * wt));
        const int x = 2 * (static_cast<int>(blockIdx.x) * a.xt - a.hl);
        for (int r0 = 0; r0 < a.n2; r0 += a.n2_box)
            tma_load_2d(s + static_cast<size_t>(r0) * wt, &map, &bar, x, blockIdx.y * a.n2 + r0);
    }
    // column constants and row frequencies are computed while the tile is in flight
    az_rd_tables(a, blockIdx.x, blockIdx.y, threadIdx.x, blockDim.x, t);
    __syncthreads();
    if (a.use_tma) mbar_wait(&bar, 0, err);
    az_rd_body<true, R0, R1, R2>(a, blockIdx.x, blockIdx.y, threadIdx.x, blockDim.x, s, t, err, a.use_tma != 0);
}

}  // namespace

template <int R0, int R1, int R2>
int launch_az_rd(const AzRdArgs& a, const void* tmap, int tiles, int nblocks, LaunchShape sh, unsigned int* err,
                 void* stream) {
    int rc = ensure_smem(k_az_rd<R0, R1, R2>, sh.smem, "az_rd");
    if (rc || tiles <= 0) return rc;
    k_az_rd<R0, R1, R2><<<dim3(tiles, nblocks), sh.threads, sh.smem, S(stream)>>>(a, err, tmap_or_zero(tmap));
    return check_launch("az_rd");
}

template int launch_az_rd<ASARF_R0, ASARF_R1, ASARF_R2>(const AzRdArgs&, const void*, int, int, LaunchShape,
                                                        unsigned int*, void*);

}  // namespace asarf
