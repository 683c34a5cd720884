// arap_launch.cuh -- overlapped launches (programmatic dependent launch),
// shared by the single-request and the batched kernels.
#pragma once

#include <cuda_runtime.h>

namespace arapgpu {

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization may start once every CTA of the kernel before it has called
// pdl_trigger (or exited); pdl_wait then blocks until that kernel has
// finished and its memory is visible. Without the launch attribute pdl_wait
// returns at once.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A launch with programmatic stream serialization when `overlap` is set: the
// kernel may then start while the kernel before it in the stream still runs
// (see pdl_wait); otherwise an ordinary launch.
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), bool overlap, dim3 grid, int block, size_t smem, cudaStream_t st,
                       Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace arapgpu
