// out[M,N] = epilogue( A[M,K] * W[N,K]^T ) for one to four activation rows: plain FMA, W straight into registers.
//
// With so few rows a product is a read of W, and in a decoding step the kernels form a chain, so what counts beside the
// bytes is how long a kernel takes from the moment its input is there.  The tensor-core kernel (skinny_sm100.cu) then still
// has to fetch A by TMA, multiply, drain TMEM and reduce over a cluster.  Here a warp holds 2 rows x 2048 columns of W in
// registers (16 loads of 16 bytes per lane, issued before the input is waited for where W is static), and after the wait
// only A passes through shared memory, 128 to 512 FMAs per lane run, and a shuffle tree ends the sum.  K beyond 2048 is
// split over the warps of the CTA, which meet in shared memory in a fixed order.  N 2048 K 2048, one row: 5.1 us there, 3.6
// here; a block of OPT-1.3b in a decoding step 45.7 and 41.1 us.
#include "common.cuh"
#include "host_util.h"
#include "pdl.cuh"
#include "skinny.h"

namespace dz {

constexpr int GV_CHUNKS = 8;                     // 16-byte loads per lane and row
constexpr int GV_K = GV_CHUNKS * 32 * 8;         // columns of W per warp
constexpr int GV_WARPS = 10;                     // most warps of a CTA (K up to 20480)
constexpr int GV_SMEM = 96 * 1024;               // A of a CTA

// Coherent: outside a decoding step the sweep that stages W may have been launched just ahead (pdl.cuh).
__device__ __forceinline__ uint4 ld_weight(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// ks: warps that share a row pair; groups: row pairs per CTA.
template <int M>
__global__ void __launch_bounds__(GV_WARPS * 32)
gemv_kernel(const __nv_bfloat16* W, long long ldw, const __nv_bfloat16* A, long long lda, const SkinnyArgs p,
            int ks, int groups) {
  extern __shared__ __align__(16) uint8_t gv_smem[];          // A as [M][K] bf16
  __shared__ float s_part[GV_WARPS][2 * M];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slice = warp % ks, pair = (int)blockIdx.x * groups + warp / ks;
  // the two rows of W: neighbours, or (SwiGLU) the gate and the up row of one output column
  const int row0 = p.act == 3 ? pair : 2 * pair;
  const int row1 = p.act == 3 ? p.N + pair : row0 + 1;
  const bool ok0 = row0 < p.N, ok1 = p.act == 3 ? ok0 : row1 < p.N;
  const int k0 = slice * GV_K + lane * 8;
  uint4 w[2][GV_CHUNKS];
  auto load_w = [&]() {
#pragma unroll
    for (int c = 0; c < GV_CHUNKS; ++c) {
      const int k = k0 + c * 256;
      w[0][c] = w[1][c] = make_uint4(0u, 0u, 0u, 0u);
      if (k < p.K) {
        if (ok0) w[0][c] = ld_weight(W + row0 * ldw + k);
        if (ok1) w[1][c] = ld_weight(W + row1 * ldw + k);
      }
    }
  };
  if (p.w_static) load_w();
  pdl_wait();
  // only now: the next kernel of the chain never runs beside a predecessor of this one, whose lines its L1 could hold
  pdl_trigger();
  if (!p.w_static) load_w();
  const int kvec = p.K >> 3;
  for (int i = threadIdx.x; i < M * kvec; i += blockDim.x) {
    const int m = i / kvec, j = i - m * kvec;
    reinterpret_cast<uint4*>(gv_smem)[i] = __ldcg(reinterpret_cast<const uint4*>(A + m * lda) + j);
  }
  __syncthreads();
  float acc[2][M];
#pragma unroll
  for (int m = 0; m < M; ++m) acc[0][m] = acc[1][m] = 0.f;
#pragma unroll
  for (int c = 0; c < GV_CHUNKS; ++c) {
    const int k = k0 + c * 256;
    if (k >= p.K) break;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const uint4 x = reinterpret_cast<const uint4*>(gv_smem)[m * kvec + (k >> 3)];
      const uint32_t xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t wv[4] = {w[r][c].x, w[r][c].y, w[r][c].z, w[r][c].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[r][m] = fmaf(bf16_lo(xv[j]), bf16_lo(wv[j]), acc[r][m]);
          acc[r][m] = fmaf(bf16_hi(xv[j]), bf16_hi(wv[j]), acc[r][m]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc[r][m] += __shfl_xor_sync(0xffffffffu, acc[r][m], off);
    }
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) s_part[warp][r * M + m] = acc[r][m];
  }
  __syncthreads();
  if (slice != 0 || lane >= (p.act == 3 ? M : 2 * M)) return;
  // ---- one output element per lane
  const int m = lane % M, r = lane / M;
  const int col = p.act == 3 ? pair : row0 + r;
  if (col >= p.N) return;
  float v = 0.f, up = 0.f;
  for (int s = 0; s < ks; ++s) {
    v += s_part[warp + s][r * M + m];
    if (p.act == 3) up += s_part[warp + s][M + m];
  }
  if (p.act == 3) {
    v = v / (1.f + __expf(-v)) * up;
  } else {
    if (p.bias) v += __bfloat162float(p.bias[col]);
    v *= p.out_scale;
    if (p.act == 1) v = fmaxf(v, 0.f);
    else if (p.act == 2) v = gelu_erf(v);
  }
  if (p.residual) {
    const unsigned short b = __ldcg(reinterpret_cast<const unsigned short*>(p.residual + m * p.ldr + col));
    v += __uint_as_float(static_cast<uint32_t>(b) << 16);
  }
  if (p.out_fp32) {
    float* op = reinterpret_cast<float*>(p.out) + m * p.ldo + col;
    if (DZ_STORE_OK(op, 4)) *op = v;
  } else {
    __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(p.out) + m * p.ldo + col;
    if (DZ_STORE_OK(op, 2)) *op = __float2bfloat16(v);
  }
}

bool gemv_takes(int M, int K) {
  return M >= 1 && M <= 4 && K <= GV_K * GV_WARPS && (long long)M * K * 2 <= GV_SMEM;
}

// Small matrices only: the larger ones are read faster through the TMA ring.  One row, us, skinny_sm100.cu / here: N 2304 K
// 768 4.2 / 2.4, N 768 K 3072 4.9 / 3.3, N 2048 K 2048 5.1 / 3.6 (four rows 5.3 / 4.6); N 6144 K 2048 7.5 / 8.1, N 4096 K
// 4096 8.7 / 9.6, N 4096 K 11008 17.8 / 27.9.
bool gemv_pays(int M, int N, int K) { return gemv_takes(M, K) && (long long)N * K <= 6LL << 20; }

template <int M>
static int launch_m(const void* W, long long ldw, const void* A, long long lda, const SkinnyArgs& a, bool dependent,
                    cudaStream_t stream) {
  const int ks = (a.K + GV_K - 1) / GV_K;
  const int groups = ks >= 8 ? 1 : 8 / ks;
  const int pairs = a.act == 3 ? a.N : (a.N + 1) / 2;
  auto kern = gemv_kernel<M>;
  static PerDeviceFlag configured;
  if (int rc = ensure_dyn_smem(configured, kern, GV_SMEM)) return rc;
  return cuda_rc(pdl_launch(kern, dim3((unsigned)((pairs + groups - 1) / groups)), ks * groups * 32, (size_t)M * a.K * 2,
                            stream, 1, dependent, reinterpret_cast<const __nv_bfloat16*>(W), ldw,
                            reinterpret_cast<const __nv_bfloat16*>(A), lda, a, ks, groups));
}

int gemv_launch(const void* W, long long ldw, const void* A, long long lda, const SkinnyArgs& a, bool dependent,
                cudaStream_t stream) {
  switch (a.M) {
    case 1: return launch_m<1>(W, ldw, A, lda, a, dependent, stream);
    case 2: return launch_m<2>(W, ldw, A, lda, a, dependent, stream);
    case 3: return launch_m<3>(W, ldw, A, lda, a, dependent, stream);
    default: return launch_m<4>(W, ldw, A, lda, a, dependent, stream);
  }
}

}  // namespace dz

using namespace dz;
DZ_DEBUG_TU(gemv)

// Same contract as dz_gemm_skinny for M <= 4 and M * K <= 48 Ki.
extern "C" int dz_gemv(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo,
                       const void* bias, const void* residual, long long ldr, int M, int N, int K, int act, int out_fp32,
                       float out_scale, uint32_t* err, cudaStream_t stream) {
  if (!A || !W || !out || M <= 0 || N <= 0 || K <= 0 || act < 0 || act > 3) return DZ_ERR_ARG;
  if (!gemv_takes(M, K) || (long long)N * 2 > 0x7fffffffLL) return DZ_ERR_TOO_LARGE;
  if ((K & 7) || (lda & 7) || (ldw & 7)) return DZ_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) return DZ_ERR_ALIGN;
  if (act == 3 && (bias || residual || out_fp32 || out_scale != 1.0f)) return DZ_ERR_ARG;
  SkinnyArgs a{};
  a.M = M; a.N = N; a.K = K; a.out = out; a.ldo = ldo;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  a.ldr = ldr; a.act = act; a.out_fp32 = out_fp32; a.out_scale = out_scale; a.err = err;
  return gemv_launch(W, ldw, A, lda, a, true, stream);
}
