// LoRA merge for forward-only training:  out[n, k] = W[n, k] + s * sum_r B[n, r] * A[r, k].
//
// Zeroth-order training never back-propagates, so the low-rank update can be folded into
// the projection weight before the (single, full-speed) QKV GEMM instead of running the two
// skinny GEMMs x A^T B^T of the reference (large_models/lora.py:89-98).  The merge is one
// bandwidth-bound pass over the d x d weight (read W, write the staged W_eff), r <= 16.
#include "common.cuh"
#include "host_util.h"

namespace dz {

constexpr int LORA_MAX_R = 16;

// Small matrices: one row of W per thread, so that every load of the launch is independent of the others.  Us, this kernel /
// the one below: 768 x 768, rank 2 1.8 / 2.1, rank 8 2.3 / 2.7; 1536 x 1536, rank 8 4.2 / 4.7; 2048 x 2048, rank 1 3.1 / 3.5,
// rank 4 3.9 / 4.3, rank 8 5.5 / 5.3; 2560 x 2560, rank 1 4.3 / 4.3, rank 4 5.9 / 5.3.
template <int R>
__global__ void __launch_bounds__(256)
lora_merge_row_kernel(const __nv_bfloat16* __restrict__ W, long long ldw,
                  const __nv_bfloat16* __restrict__ A, long long lda,   // [R, K]
                  const __nv_bfloat16* __restrict__ B, long long ldb,   // [N, R]
                  __nv_bfloat16* __restrict__ out, long long ldo, int N, int K, float s) {
  // grid: (ceil(K / 2048), N); each thread owns 8 consecutive k of one row n
  const int n = blockIdx.y;
  const int k0 = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (k0 >= K) return;
  float b[R];
#pragma unroll
  for (int r = 0; r < R; ++r) b[r] = s * __bfloat162float(B[(long long)n * ldb + r]);
  uint4 w = *reinterpret_cast<const uint4*>(W + (long long)n * ldw + k0);
  float v[8] = {bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y),
                bf16_lo(w.z), bf16_hi(w.z), bf16_lo(w.w), bf16_hi(w.w)};
#pragma unroll
  for (int r = 0; r < R; ++r) {
    uint4 a = __ldg(reinterpret_cast<const uint4*>(A + (long long)r * lda + k0));
    v[0] = fmaf(b[r], bf16_lo(a.x), v[0]); v[1] = fmaf(b[r], bf16_hi(a.x), v[1]);
    v[2] = fmaf(b[r], bf16_lo(a.y), v[2]); v[3] = fmaf(b[r], bf16_hi(a.y), v[3]);
    v[4] = fmaf(b[r], bf16_lo(a.z), v[4]); v[5] = fmaf(b[r], bf16_hi(a.z), v[5]);
    v[6] = fmaf(b[r], bf16_lo(a.w), v[6]); v[7] = fmaf(b[r], bf16_hi(a.w), v[7]);
  }
  uint4 o;
  o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
  o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
  if (DZ_STORE_OK(out + (long long)n * ldo + k0, 16)) *reinterpret_cast<uint4*>(out + (long long)n * ldo + k0) = o;
}

constexpr int LM_THREADS = 128;  // 8 columns each
constexpr int LM_ROWS = 32;      // most rows of W per CTA
constexpr int LM_UNROLL = 8;     // rows in flight per thread

// grid (ceil(K / 1024), ceil(N / LM_ROWS)).  A thread keeps its 8 columns of A in registers (as floats up to rank 8) and
// walks down up to LM_ROWS rows of W, LM_UNROLL loads ahead; the CTA's rows of s * B sit in shared memory.  With one row per
// thread every 16 bytes of W needed 144 bytes through L1: 5120 x 5120, rank 8 29.8 -> 24.6 us (40 -> 28.5 us within a
// training step); eight rows in flight measured 24.6, four 28.4.
template <int R>
__global__ void __launch_bounds__(LM_THREADS)
lora_merge_kernel(const __nv_bfloat16* __restrict__ W, long long ldw,
                  const __nv_bfloat16* __restrict__ A, long long lda,   // [R, K]
                  const __nv_bfloat16* __restrict__ B, long long ldb,   // [N, R]
                  __nv_bfloat16* __restrict__ out, long long ldo, int N, int K, float s, int cta_rows) {
  __shared__ float s_b[LM_ROWS * R];
  const int n0 = blockIdx.y * cta_rows;
  const int rows = min(cta_rows, N - n0);
  const int k0 = (blockIdx.x * LM_THREADS + threadIdx.x) * 8;
  const bool col_ok = k0 < K;
  // A and the first rows of W are on their way while s * B is staged: on a small matrix the launch is one such round trip
  uint4 ap[R], w[LM_UNROLL];
  auto load_w = [&](int n) {
#pragma unroll
    for (int u = 0; u < LM_UNROLL; ++u)
      if (n + u < rows) w[u] = *reinterpret_cast<const uint4*>(W + (long long)(n0 + n + u) * ldw + k0);
  };
  if (col_ok) {
#pragma unroll
    for (int r = 0; r < R; ++r) ap[r] = __ldg(reinterpret_cast<const uint4*>(A + (long long)r * lda + k0));
    load_w(0);
  }
  for (int i = threadIdx.x; i < rows * R; i += LM_THREADS)
    s_b[i] = s * __bfloat162float(B[(long long)(n0 + i / R) * ldb + i % R]);
  __syncthreads();
  if (!col_ok) return;
  constexpr bool FLOATS = R <= 8;
  float af[FLOATS ? R : 1][8];
  if constexpr (FLOATS) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      af[r][0] = bf16_lo(ap[r].x); af[r][1] = bf16_hi(ap[r].x); af[r][2] = bf16_lo(ap[r].y); af[r][3] = bf16_hi(ap[r].y);
      af[r][4] = bf16_lo(ap[r].z); af[r][5] = bf16_hi(ap[r].z); af[r][6] = bf16_lo(ap[r].w); af[r][7] = bf16_hi(ap[r].w);
    }
  }
  for (int n = 0; n < rows; n += LM_UNROLL) {
    if (n) load_w(n);
#pragma unroll
    for (int u = 0; u < LM_UNROLL; ++u) {
      if (n + u >= rows) break;
      float v[8] = {bf16_lo(w[u].x), bf16_hi(w[u].x), bf16_lo(w[u].y), bf16_hi(w[u].y),
                    bf16_lo(w[u].z), bf16_hi(w[u].z), bf16_lo(w[u].w), bf16_hi(w[u].w)};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float b = s_b[(n + u) * R + r];
        if (FLOATS) {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = fmaf(b, af[r][j], v[j]);
        } else {
          const uint4 a = ap[r];
          v[0] = fmaf(b, bf16_lo(a.x), v[0]); v[1] = fmaf(b, bf16_hi(a.x), v[1]);
          v[2] = fmaf(b, bf16_lo(a.y), v[2]); v[3] = fmaf(b, bf16_hi(a.y), v[3]);
          v[4] = fmaf(b, bf16_lo(a.z), v[4]); v[5] = fmaf(b, bf16_hi(a.z), v[5]);
          v[6] = fmaf(b, bf16_lo(a.w), v[6]); v[7] = fmaf(b, bf16_hi(a.w), v[7]);
        }
      }
      uint4 o;
      o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
      o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
      uint4* op = reinterpret_cast<uint4*>(out + (long long)(n0 + n + u) * ldo + k0);
      if (DZ_STORE_OK(op, 16)) *op = o;
    }
  }
}

}  // namespace dz

using namespace dz;
DZ_DEBUG_TU(peft)

extern "C" int dz_lora_merge(const void* W, long long ldw, const void* A, long long lda,
                             const void* B, long long ldb, void* out, long long ldo, int N, int K,
                             int r, float scaling, cudaStream_t stream) {
  if (!W || !A || !B || !out || N <= 0 || K <= 0 || r <= 0) return DZ_ERR_ARG;
  if (r > LORA_MAX_R) return DZ_ERR_TOO_LARGE;
  if ((K & 7) || (ldw & 7) || (lda & 7) || (ldo & 7) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
    return DZ_ERR_ALIGN;
  const bool small = (long long)N * K <= (r <= 4 ? 8LL << 19 : 5LL << 19) && N <= 65535;      // 2048^2; between 1536^2 and that
  // 32 rows share a CTA's columns of A while that leaves a few CTAs per SM; smaller matrices are cut finer
  const int cols = (K + LM_THREADS * 8 - 1) / (LM_THREADS * 8);
  int rows = LM_ROWS;
  while (rows > 4 && (long long)cols * ((N + rows - 1) / rows) < 4LL * sm_count()) rows /= 2;
  if (!small && (N + rows - 1) / rows > 65535) return DZ_ERR_TOO_LARGE;
  const dim3 grid = small ? dim3((K + 2047) / 2048, N) : dim3(cols, (N + rows - 1) / rows);
  auto w = (const __nv_bfloat16*)W; auto a = (const __nv_bfloat16*)A;
  auto b = (const __nv_bfloat16*)B; auto o = (__nv_bfloat16*)out;
  switch (r) {
#define DZ_R(RR)                                                                                                       \
    case RR:                                                                                                           \
      if (small) lora_merge_row_kernel<RR><<<grid, 256, 0, stream>>>(w, ldw, a, lda, b, ldb, o, ldo, N, K, scaling);   \
      else lora_merge_kernel<RR><<<grid, LM_THREADS, 0, stream>>>(w, ldw, a, lda, b, ldb, o, ldo, N, K, scaling, rows); \
      break;
    DZ_R(1) DZ_R(2) DZ_R(3) DZ_R(4) DZ_R(5) DZ_R(6) DZ_R(7) DZ_R(8)
    DZ_R(9) DZ_R(10) DZ_R(11) DZ_R(12) DZ_R(13) DZ_R(14) DZ_R(15) DZ_R(16)
#undef DZ_R
  }
  return cuda_rc(cudaGetLastError());
}
