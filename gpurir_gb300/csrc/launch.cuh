// launch.cuh -- kernels launched back to back in one stream (programmatic dependent launch).
//
// The next kernel's blocks come in as the last of this one's leave, and wait there for its
// results before they touch anything: launch latency and drain run under one another (a
// fused fitting step of 16 rooms, five kernels: 150 to 138 us).  Other work of the stream
// (copies, memsets, other libraries' kernels, graph nodes) is ordered as by a plain launch: the
// wait holds until everything before has completed and is visible.  No kernel asks for its
// successor earlier (griddepcontrol.launch_dependents): measured 2 us slower, and a foreign
// kernel launched this way might read before our results are there.
#pragma once

#include <cuda_runtime.h>

namespace gpurir {

// First statement of every kernel that is launched by launch_after.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A pointer whose read-only loads (__ldg, const __restrict__) must not be moved before the wait:
// the compiler may take such loads for free of any order, but not ahead of the pointer they use.
template <class T>
__device__ __forceinline__ T *after_wait(T *p) {
    asm volatile("" : "+l"(p));
    return p;
}

template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess) cudaGetLastError();   // (returned, not left behind)
    return e;
}

}  // namespace gpurir
