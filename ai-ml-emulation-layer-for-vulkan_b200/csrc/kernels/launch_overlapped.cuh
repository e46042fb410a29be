// Programmatic dependent launch for the kernels between the tensor-core launches.
//
// A kernel launched this way is set up and its blocks are scheduled while the kernel before it in the stream drains; it
// calls dependencySync() before it touches memory that another kernel writes or will write.  Worth it between two
// tensor-core launches (the layer norms and the GELU of a BERT-shaped encoder: 2.495 -> 2.451 ms per dispatch of 168
// nodes); not in a chain of short element-wise kernels, where a replayed graph's ordinary edges are as quick (the twelve
// operators of a graph of small ones: 31 us with ordinary launches, 34 with these).
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "gemm_i8_tcgen05.hpp"

namespace mlel {

// Lets the next kernel of the stream be scheduled, then waits for the one before to complete with its writes visible.
// Both are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void dependencySync() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... Params, class... Args>
inline void launchOverlapped(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smemBytes, cudaStream_t stream,
                             Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = tensorCoreTuning().dependentLaunch.load(std::memory_order_relaxed) != 0 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

} // namespace mlel
