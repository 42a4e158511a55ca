// stream_impl.cuh -- body of one per-type translation unit of the stream kernel; the including
// file defines HPDEX_STREAM_T (suffix) and HPDEX_STREAM_V (value type).
#include "mwu_stream.cuh"
#include "rank_launch.h"

namespace hpdex {

#define HPDEX_CAT2(a, b) a##b
#define HPDEX_CAT(a, b) HPDEX_CAT2(a, b)

cudaError_t HPDEX_CAT(stream_launch_, HPDEX_STREAM_T)(const StreamArgs& a, int grid, size_t smem,
                                                      cudaStream_t s) {
    auto k = mwu_stream_kernel<HPDEX_STREAM_V, kStreamThreads>;
    cudaError_t e = allow_max_smem(k);
    if (e != cudaSuccess) return e;
    k<<<grid, kStreamThreads, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace hpdex
