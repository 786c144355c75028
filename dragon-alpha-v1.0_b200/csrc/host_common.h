// Declarations shared by the host translation units of the library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                    const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*PFN_encodeIm2col)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                     const cuuint64_t*, const cuuint64_t*, const int*, const int*,
                                     cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion,
                                     CUtensorMapFloatOOBfill);

namespace alpha {

// Records a printf-style message as the calling thread's last error and returns `code`.
int fail(int code, const char* fmt, ...);
// Counts one kernel launch and remembers the kernel family for alpha_conv_last_algo().
void note_launch(const char* algo);

// Launches a kernel that waits for its predecessor itself (grid_dependency_wait), so that its launch and prologue overlap the
// predecessor's tail: 20 convolutions of the ResNet-18 stack with their gradients, 190 launches, at batch 64 1636 -> 1351 us, at
// batch 512 4.39 -> 4.07 ms.  Only for kernels whose every thread does; an ordinary launch while the stream is being captured, where
// the captured dependencies say it all.
template <class... Params, class... Args>
inline void launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    bool plain = true;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
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

}  // namespace alpha
