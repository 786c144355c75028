// Launches: dynamic shared memory beyond 48 KB, and programmatic dependent launch from both sides.
#pragma once
#include <cuda_runtime.h>

#include "once_per_device.h"

#include <utility>

namespace alpha {

// Lets launches of KERNEL on the current device ask for up to `bytes` of dynamic shared memory (always the same for a kernel).  The runtime
// keeps a function's attributes for each device apart.  A failure stays in cudaGetLastError, is met by the launch, and is tried again.
template <auto KERNEL>
inline cudaError_t allow_smem(int bytes = 227 * 1024)
{
    static OncePerDevice once;
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    return static_cast<cudaError_t>(once(device, [bytes] { return static_cast<int>(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)); }));
}

// A kernel launched with launch_after may start while its predecessor in the stream still runs.  Every thread calls
// grid_dependency_wait() before it touches global memory: it returns when the predecessor has completed and its writes are
// visible (at once in an ordinary launch).  grid_dependency_trigger() lets the successor start; a kernel calls it only after
// it holds its tensor memory, so that a waiting successor can never hold columns this one still needs.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// False while an SM budget leaves SMs to other streams' kernels: a waiting successor would take just those.
bool dependent_launches();

// Launches a kernel that waits for its predecessor itself (grid_dependency_wait), so that its launch and prologue overlap the
// predecessor's tail: 20 convolutions of the ResNet-18 stack with their gradients, some 180 launches, at batch 64 1636 -> 1351 us, at
// batch 512 4.39 -> 4.07 ms.  Only for kernels whose every thread does; an ordinary launch while the stream is being captured, where
// the captured dependencies say it all, and under an SM budget (ten 56 x 56 x 64 layers on 100 SMs beside 100 small GEMMs of another
// stream: the GEMMs end after 1.2 ms, after 2.1 ms with the successors resident on the other 48 SMs).
template <class... Params, class... Args>
inline void launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    bool plain = true;
    if (!dependent_launches()) {
        plain = true;
    } else if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
        cudaGetLastError();   // (a legacy stream beside another one's capture)
    } else {
        plain = cap != cudaStreamCaptureStatusNone;
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = &attr; cfg.numAttrs = plain ? 0 : 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);   // the caller looks at cudaGetLastError()
}

// The same for a kernel with more than 48 KB of dynamic shared memory.
template <auto KERNEL, class... Args>
inline void launch_large(dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args)
{
    allow_smem<KERNEL>();
    launch_after(KERNEL, grid, block, smem, stream, std::forward<Args>(args)...);
}

}  // namespace alpha
