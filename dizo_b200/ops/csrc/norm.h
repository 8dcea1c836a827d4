// Host interface of the LayerNorm / RMSNorm kernels inside the library.  `dependent`: programmatic dependent launch.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dz {

int layernorm_launch(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, const __nv_bfloat16* b,
                     __nv_bfloat16* y, long long ldy, long long rows, int d, float eps, bool dependent,
                     cudaStream_t stream);
int rmsnorm_launch(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, __nv_bfloat16* y, long long ldy,
                   long long rows, int d, float eps, bool dependent, cudaStream_t stream);

}  // namespace dz
