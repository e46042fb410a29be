// Programmatic dependent launch.  A kernel launched this way may start while the kernel before it in the stream is still
// running (on SMs that kernel has already left): everything up to dependencySync() - barrier and TMEM set-up, tables built
// from graph constants - overlaps the predecessor's tail.  The wait returns when the predecessor has completed and its
// writes are visible; nothing before it may touch memory that another kernel of the stream writes or reads for writing
// later.  The trigger lets the successor start as early as it finds room.  Both are no-ops in a kernel launched the
// ordinary way.
//
// Such a kernel reads activations by plain loads.  The read-only path (__ldg, or a const parameter with __restrict__) is for
// memory that nothing writes while the kernel runs, and this one runs beside the kernel that writes its input; for a pointer
// that is __restrict__ the compiler may also move an access across the wait.  __ldg is for graph constants.
//
// Beside the tensor-core kernels it is worth it between two of their launches (the layer norms and the GELU of a
// BERT-shaped encoder: 2.495 -> 2.451 ms per dispatch of 12 layers), and for the copies, transposes, windows and moves in
// front of and between them: an ordinary boundary between two kernels costs a whole number of 2.048 us on this machine, the
// remainder of the last one waited out (a padded copy and its product, enqueued one after the other: 8.2 us a pass as
// ordinary launches, 5.6-6.4 with these; one image of the ResNet-50 shape 214.4 -> 212.1).  Not for average pools (one image of
// the MobileNetV2 shape 2 us slower) and not in a chain of short element-wise kernels (the twelve operators of a graph of
// small ones: 31 us with ordinary launches, 34 with these, 18 on lanes of their own, see Session::capture).
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "gemm_i8_tcgen05.hpp"

namespace mlel {

__device__ __forceinline__ void dependencySync() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... Params, class... Args>
inline cudaError_t launchOverlapped(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smemBytes, cudaStream_t stream,
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
    cfg.numAttrs = dependentLaunches() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

} // namespace mlel
