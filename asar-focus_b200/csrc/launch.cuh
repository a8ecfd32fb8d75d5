// Launch helpers of the kernel translation units, and the launchers that live in units of their own.
//
// The runtime loads a unit's kernels as one module when the first of them is asked for. One unit
// for everything took 15 to 20 ms at a process's first kernel, most of it for schedules that its plans
// never run, so each compiled schedule and range length is a unit (build.py lists them); a plan loads
// its own ones when it is made. A launcher that is given nothing to run (no tiles or lines) only loads
// its kernel and sets its shared-memory size.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "asarf.h"
#include "backend.h"
#include "params.h"

namespace asarf {

inline int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(ASARF_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
    return ASARF_OK;
}

// Raise a kernel's dynamic shared-memory limit to `bytes` (once per kernel, device and size:
// the default limit of 48 KiB counts the kernel's static shared memory too, so any dynamic
// size is checked, not only those above 48 KiB).
template <class K>
int ensure_smem(K kernel, size_t bytes, const char* what) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
    auto it = done.find(key);
    if (it != done.end() && it->second >= bytes) return ASARF_OK;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return set_error(ASARF_ERR_CUDA, "%s smem %zu: %s", what, bytes, cudaGetErrorString(e));
    done[key] = bytes;
    return ASARF_OK;
}

inline cudaStream_t S(void* s) { return static_cast<cudaStream_t>(s); }

inline CUtensorMap tmap_or_zero(const void* tmap) {
    CUtensorMap m;
    if (tmap)
        std::memcpy(&m, tmap, sizeof(m));
    else
        std::memset(&m, 0, sizeof(m));
    return m;
}

// az_rd.cu: radix schedule of the contiguous transforms (0, 0, 0: run-time)
template <int R0, int R1, int R2>
int launch_az_rd(const AzRdArgs& a, const void* tmap, int tiles, int nblocks, LaunchShape sh, unsigned int* err,
                 void* stream);
// az_strided.cu: radix schedule of the strided transform (0, 0, 0: run-time), tile width, tiles a block
template <int R0, int R1, int R2, int XT, int NB>
int launch_az_strided(const AzStridedArgs& a, const void* tmap, int tiles, LaunchShape sh, void* stream);
// range_compress.cu: range FFT length (0: run-time)
template <int L>
int launch_range_compress(const RangeCompressArgs& a, int lines, LaunchShape sh, void* stream);
template <int L>
int launch_rc_rows(const RcRowsArgs& a, int rows, LaunchShape sh, void* stream);

}  // namespace asarf
