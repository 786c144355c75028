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
// What alpha_conv_last_plan() reports (printf style).
void note_plan(const char* fmt, ...);
// SMs of the current device that kernels may spread over (option SM_BUDGET).
int device_sms(int* sms);
// Where kernels report a wait that ran out.
int device_status_word(int** status);
// CTAs of one launch of the bf16-plane kernel, 0 = no limit.
int planes_launch_slice(int* ctas);
// Option F32_PLANES.
int option_f32_planes();

}  // namespace alpha
