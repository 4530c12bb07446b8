// Host-side launch helpers.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace psb {

// Opt a kernel into the large dynamic shared-memory carve-out, once per
// (kernel, device).
template <class K>
void allow_big_smem(K kernel)
{
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, bool> done;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!done[key]) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        done[key] = true;
    }
}

// A kernel that may begin while the one before it in the stream ends (it waits
// for it itself: grid_wait).  Its fields come in through plain pointers, never
// const __restrict__ ones: that promises that nobody writes the data while the
// kernel lives, which the kernel before it still does, and lets the compiler
// load it through the non-coherent path or above the wait (whose memory clobber
// orders no load of data promised not to change).
template <class... P, class... A>
void launch_after(void (*k)(P...), int grid, int nt, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace psb
