// A whole OPT decoder block launched by one call, and the choice of the GEMM kernel for a shape.
//
// The seven kernels of a block run for 2 to 15 us each on the small models, but issued one by one from Python each costs
// about 35 us of host time (tensor views, allocations, argument conversion).  A training step of OPT-125m, 16 prompts of 64
// tokens, has 2.0 ms of kernels: 7.05 ms from Python, 2.98 ms with whole blocks; scoring 32 prompts of 120 tokens with
// OPT-1.3b 8.9 ms of kernels: 12.7 and 10.7 ms.
// The caller keeps one set of workspaces per forward and passes pointers; nothing is kept here between calls.
#include "host_util.h"
#include "linear.h"

extern "C" {
int dz_layernorm(const void* x, long long ldx, const void* w, const void* b, void* y, long long ldy, long long rows, int d,
                 float eps, cudaStream_t stream);
int dz_gemm_skinny(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo, const void* bias,
                   const void* residual, long long ldr, int M, int N, int K, int act, int out_fp32, float out_scale,
                   int splits, uint32_t* err, cudaStream_t stream);
int dz_gemm2_bf16_tn(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo, const void* bias,
                     const void* residual, long long ldr, int M, int N, int K, int act, int out_fp32, float out_scale,
                     uint32_t* err, cudaStream_t stream);
int dz_gemm_bf16_tn(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo, const void* bias,
                    const void* residual, long long ldr, int M, int N, int K, int act, int out_fp32, float out_scale,
                    int tile_n, uint32_t* err, cudaStream_t stream);
int dz_attn_fwd(const void* qkv, long long ld_qkv, int q_col0, int k_col0, int v_col0, void* out, long long ld_out,
                const int* pad_left, const void* prefix_k, const void* prefix_v, long long ld_prefix, int n_prefix, int B,
                int L, int H, int hd, float scale, uint32_t* err, cudaStream_t stream);
}

using namespace dz;

// Whether the swapped-operand, K-split kernel (skinny_sm100.cu) takes a product.  Up to 16 rows it always wins (one row,
// us, 128-row tiles / skinny: N 2048 K 8192 32.9 / 10.3, N 50272 K 2048 57.6 / 36.1).  With more rows its wider activation
// operand costs L2 traffic per tile of W, which only K splitting makes up for: at 32 rows N 32000 K 4096 50.2 / 48.1 but
// N 50272 K 2048 40.6 / 42.8; at 64 rows N 2048 K 8192 31.9 / 13.7, N 8192 K 2048 12.4 / 11.9, but N 16384 K 4096 29.2 /
// 29.6 and N 50272 K 2048 40.4 / 49.5.
static bool skinny_pays(int M, int N) {
  const int tiles = (N + 127) / 128;
  return M <= 16 || (M <= 32 && tiles <= 296) || (M <= 64 && tiles <= 74);
}

// CTAs per 128 x 128 tile where the K-split kernel pays for more rows than that, else 0: few tiles, and enough K blocks
// that the halved loop is worth the reduction over the cluster.  Launches beyond about 128 CTAs of split tiles, or clusters
// of 8, do not pack and run in two rounds.  Measured, us, 128-row tiles / split (CTAs a tile): M 360 N 1024 K 4096 17.9 /
// 11.6 (4), M 512 N 1024 K 4096 17.7 / 12.1 (4), M 128 N 2048 K 8192 32.3 / 13.8 (6), M 100 N 4096 K 16384 62.1 / 32.4 (4),
// M 300 N 2048 K 8192 31.5 / 23.9 (2), M 1000 N 1024 K 4096 17.8 / 16.7 (2); but M 360 N 1024 K 1024 7.2 / 8.4 (4), M 1024
// N 768 K 768 7.4 / 10.3 (3), M 300 N 2048 K 2048 11.5 / 13.1 (2).
static int split_pays(int M, int N, int K) {
  const long long tiles = (long long)((M + 127) / 128) * ((N + 127) / 128);
  const int num_kb = (K + 63) / 64;
  if (tiles <= 32 && num_kb >= 32) return tiles <= 21 ? 6 : 4;
  return tiles <= 64 && num_kb >= 64 ? 2 : 0;
}

extern "C" int dz_linear(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo,
                         const void* bias, const void* residual, long long ldr, int M, int N, int K, int act,
                         int out_fp32, float out_scale, uint32_t* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return DZ_ERR_ARG;
  const bool skinny = skinny_pays(M, N);
  const int splits = skinny || M <= 64 ? 0 : split_pays(M, N, K);
  if (skinny || splits)
    return dz_gemm_skinny(A, lda, W, ldw, out, ldo, bias, residual, ldr, M, N, K, act, out_fp32, out_scale, splits, err,
                          stream);
  // pairs of SMs (256-row tiles) once there is work for most of them
  if (M >= 256 && (long long)((M + 255) / 256) * ((N + 255) / 256) >= 48)
    return dz_gemm2_bf16_tn(A, lda, W, ldw, out, ldo, bias, residual, ldr, M, N, K, act, out_fp32, out_scale, err, stream);
  return dz_gemm_bf16_tn(A, lda, W, ldw, out, ldo, bias, residual, ldr, M, N, K, act, out_fp32, out_scale, 0, err, stream);
}

// Mirrored by ops/block.py (ctypes).  h_out may be h_in; no other two buffers coincide.
extern "C" struct DzOptBlock {
  int B, L, d, F, H, pre_norm, act, pad_;
  float eps, scale;
  const void *ln1_w, *ln1_b, *qkv_w, *qkv_b, *out_w, *out_b, *ln2_w, *ln2_b, *fc1_w, *fc1_b, *fc2_w, *fc2_b;
  const void* h_in;                        // [B * L, d]
  void *h_out, *h_mid, *xn, *qkv, *ctx, *f;
  const int* pad_left;
  uint32_t* err;
};

extern "C" int dz_opt_block(const DzOptBlock* blk, cudaStream_t stream) {
  if (!blk || blk->B <= 0 || blk->L <= 0 || blk->H <= 0 || blk->d % blk->H || !blk->h_in || !blk->h_out || !blk->h_mid ||
      !blk->xn || !blk->qkv || !blk->ctx || !blk->f)
    return DZ_ERR_ARG;
  const DzOptBlock& b = *blk;
  if ((long long)b.B * b.L > 0x7fffffffLL) return DZ_ERR_TOO_LARGE;
  const int M = b.B * b.L, d = b.d, F = b.F;
  auto norm = [&](const void* x, const void* w, const void* bias, void* y) {
    return dz_layernorm(x, d, w, bias, y, d, M, d, b.eps, stream);
  };
  auto linear = [&](const void* x, const void* w, const void* bias, void* y, int N, int K, const void* res, int act) {
    return dz_linear(x, K, w, K, y, N, bias, res, N, M, N, K, act, 0, 1.0f, b.err, stream);
  };
  const void* x = b.h_in;
  int rc = DZ_OK;
  if (b.pre_norm) {
    rc = norm(b.h_in, b.ln1_w, b.ln1_b, b.xn);
    x = b.xn;
  }
  if (!rc) rc = linear(x, b.qkv_w, b.qkv_b, b.qkv, 3 * d, d, nullptr, 0);
  if (!rc) rc = dz_attn_fwd(b.qkv, 3 * d, 0, d, 2 * d, b.ctx, d, b.pad_left, nullptr, nullptr, 0, 0, b.B, b.L, b.H, d / b.H,
                            b.scale, b.err, stream);
  if (!rc) rc = linear(b.ctx, b.out_w, b.out_b, b.h_mid, d, d, b.h_in, 0);
  if (b.pre_norm) {
    if (!rc) rc = norm(b.h_mid, b.ln2_w, b.ln2_b, b.xn);
    if (!rc) rc = linear(b.xn, b.fc1_w, b.fc1_b, b.f, F, d, nullptr, b.act);
    if (!rc) rc = linear(b.f, b.fc2_w, b.fc2_b, b.h_out, d, F, b.h_mid, 0);
  } else {
    if (!rc) rc = norm(b.h_mid, b.ln1_w, b.ln1_b, b.xn);
    if (!rc) rc = linear(b.xn, b.fc1_w, b.fc1_b, b.f, F, d, nullptr, b.act);
    if (!rc) rc = linear(b.f, b.fc2_w, b.fc2_b, b.h_mid, d, F, b.xn, 0);
    if (!rc) rc = norm(b.h_mid, b.ln2_w, b.ln2_b, b.h_out);
  }
  return rc;
}
