// Per-(n, limbs) launch helper for walk_binary, instantiated in
// binary_walk_part*.cu (binary_dispatch.cu only declares it).
#pragma once

#include <mutex>

#include "binary_impl.cuh"

namespace spb {
namespace binary {

// With per_sm set, launches nothing and stores how many CTAs of `threads`
// threads and `smem` bytes fit on one SM.
template <int N, int L, bool X>
int launch_bin_nx(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s, int* per_sm)
{
    static std::once_flag once[64];
    static cudaError_t attr_err[64];
    int dev = 0;
    SPB_CUDA_TRY(cudaGetDevice(&dev));
    std::call_once(once[dev & 63], [&] {
        int optin = 0;
        cudaFuncAttributes fa{};
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        attr_err[dev & 63] = cudaFuncGetAttributes(&fa, walk_binary<N, L, X>);
        if (attr_err[dev & 63] == cudaSuccess)
            attr_err[dev & 63] = cudaFuncSetAttribute(walk_binary<N, L, X>,
                                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      optin - (int)fa.sharedSizeBytes);
    });
    SPB_CUDA_TRY(attr_err[dev & 63]);
    if (per_sm) {
        SPB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, walk_binary<N, L, X>, threads, smem));
        return SPB_OK;
    }
    walk_binary<N, L, X><<<blocks, threads, smem, s>>>(pb);
    SPB_CUDA_TRY(cudaGetLastError());
    return SPB_OK;
}

template <int N, int L>
int launch_bin_n(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s, int* per_sm)
{
    if constexpr (N >= kMinExpand)
        if (pb.m > 0) return launch_bin_nx<N, L, true>(pb, blocks, threads, smem, s, per_sm);
    return launch_bin_nx<N, L, false>(pb, blocks, threads, smem, s, per_sm);
}

}  // namespace binary
}  // namespace spb
