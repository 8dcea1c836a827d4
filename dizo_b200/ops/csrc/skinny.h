// Host interface of the skinny GEMM (skinny_sm100.cu) inside the library: what the decode step prepares once (tensor
// maps) and launches per token.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace dz {

constexpr int SK_MAX_ROWS = 64;      // sequences of a decoding step

struct SkinnyArgs {
  int M, N, K;                       // N: columns written (half the rows of W for act 3)
  int splits, kb_per_cta, num_kb, num_n;
  void* out;                         // bf16 or fp32 [M, ldo]
  long long ldo;
  const __nv_bfloat16* bias;         // [N] or null
  const __nv_bfloat16* residual;     // [M, ldr] or null; may be `out` itself
  long long ldr;
  int act;                           // 0 none, 1 relu, 2 gelu, 3 silu(gate) * up over W = gate rows | up rows
  int out_fp32;
  int w_static;                      // W was complete before the predecessor kernel started: load it before waiting
  float out_scale;
  uint32_t* err;
};

// Tensor maps of the operands; the width of the activation box follows from M.
int skinny_map_w(CUtensorMap* map, const void* W, long long ldw, int rows, int K, bool swiglu);
int skinny_map_x(CUtensorMap* map, const void* A, long long lda, int M, int K);
// `splits` 0: chosen from the shape and, with `in_step`, so that the next launch of a decoding step fits beside this one.
// `dependent`: programmatic dependent launch.
int skinny_launch(const CUtensorMap& tmW, const CUtensorMap& tmX, SkinnyArgs a, int splits, bool in_step, bool dependent,
                  cudaStream_t stream);

// One to four rows without tensor cores (gemv.cu), where gemv_takes(); worth it where gemv_pays().
bool gemv_takes(int M, int K);
bool gemv_pays(int M, int N, int K);
int gemv_launch(const void* W, long long ldw, const void* A, long long lda, const SkinnyArgs& a, bool dependent,
                cudaStream_t stream);

}  // namespace dz
