// A whole OPT or LLaMA decoder block launched by one call, and the choice of the GEMM kernel for a shape.
//
// The seven kernels of a block run for 2 to 15 us each on the small models, but issued one by one from Python each costs
// about 35 us of host time (tensor views, allocations, argument conversion).  A training step of OPT-125m, 16 prompts of 64
// tokens, has 2.0 ms of kernels: 7.05 ms from Python, 2.98 ms with whole blocks; scoring 32 prompts of 120 tokens with
// OPT-1.3b 8.9 ms of kernels: 12.7 and 10.7 ms.
// The caller keeps one set of workspaces per forward and passes pointers; nothing is kept here between calls.
#include "host_util.h"
#include "linear.h"
#include "skinny.h"

extern "C" {
int dz_layernorm(const void* x, long long ldx, const void* w, const void* b, void* y, long long ldy, long long rows, int d,
                 float eps, cudaStream_t stream);
int dz_gemm_skinny(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo, const void* bias,
                   const void* residual, long long ldr, int M, int N, int K, int act, int out_fp32, float out_scale,
                   int splits, uint32_t* err, cudaStream_t stream);
int dz_gemv(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo, const void* bias,
            const void* residual, long long ldr, int M, int N, int K, int act, int out_fp32, float out_scale, uint32_t* err,
            cudaStream_t stream);
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

// Whether the swapped-operand, K-split kernel (skinny_sm100.cu) takes a product.  Up to 16 rows it, or gemv.cu ahead of it, won
// on each of the 36 weight shapes measured (N 768 to 50272, K 768 to 20480): 1.22 to 4.0 times as fast as 128-row tiles with
// 1 to 8 rows, 1.10 to 3.3 with 16 (one row, us: N 2048 K 8192 32.9 / 10.3, N 50272 K 2048 57.6 / 36.1).  With more rows its
// wider activation operand costs L2 traffic per tile of W, which only K splitting makes up for: at 32 rows N 32000 K 4096
// 50.2 / 48.1 but N 50272 K 2048 40.6 / 42.8; at 64 rows N 2048 K 8192 31.9 / 13.7, N 8192 K 2048 12.4 / 11.9, but N 16384
// K 4096 29.2 / 29.6 and N 50272 K 2048 40.4 / 49.5.
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
  // the vector kernel has no alignment rule for the output rows, the others do: what they refuse stays refused
  const int esz = out_fp32 ? 4 : 2;
  const bool rows_ok = !(reinterpret_cast<uintptr_t>(out) & 15) && !((ldo * esz) & 15) &&
                       !(reinterpret_cast<uintptr_t>(bias) & 15) &&
                       (!residual || (!(reinterpret_cast<uintptr_t>(residual) & 15) && !(ldr & 7)));
  if (rows_ok && gemv_pays(M, N, K))
    return dz_gemv(A, lda, W, ldw, out, ldo, bias, residual, ldr, M, N, K, act, out_fp32, out_scale, err, stream);
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

// Mirrored by ops/block.py.  A LLaMA-family block: RMSNorm, q | k | v with the rotary embedding, attention, output
// projection, RMSNorm, SwiGLU, down projection.  The forms with the rotary embedding and SwiGLU in the GEMM's epilogue run
// under the rules of ops/gemm.py (linear_qkv_rope, linear_swiglu); otherwise `raw` holds the plain projection in between.
extern "C" struct DzLlamaBlock {
  int B, L, d, F, H, Hkv, pos0, n_pos;
  float eps, scale;
  const void *ln1_w, *qkv_w, *out_w, *ln2_w, *gu_w, *down_w;
  const void* h_in;                        // [B * L, d]
  void *h_out, *h_mid, *xn, *qkv, *ctx, *f, *raw;   // raw: [B * L, max((H + 2 Hkv) hd, 2 F)], needed without the fused forms
  const void* rope_cs;
  const int* pad_left;
  uint32_t* err;
  int fused_rope, fused_swiglu;            // the options that switch the fused epilogues
};

extern "C" {
int dz_rmsnorm(const void* x, long long ldx, const void* w, void* y, long long ldy, long long rows, int d, float eps,
               cudaStream_t stream);
int dz_rope_qkv(const void* in, long long ld_in, void* out, long long ld_out, const void* cs, long long rows, int L, int pos0,
                int n_pos, int H, int Hkv, int hd, cudaStream_t stream);
int dz_silu_mul(const void* gu, long long ld, void* out, long long ldo, long long rows, int F, cudaStream_t stream);
int dz_gemm2_qkv_rope(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo, const float* cs,
                      int M, int K, int L, int pos0, int n_pos, int H, int Hkv, uint32_t* err, cudaStream_t stream);
}

static bool pairs_pay(int M, int N) { return M >= 256 && (long long)((M + 255) / 256) * (N / 256) >= 48; }

// Bit 0: the projection with the rotary embedding is one kernel; bit 1: SwiGLU is.
extern "C" int dz_llama_block_fused(int M, int H, int Hkv, int hd, int F, int fused_rope, int fused_swiglu) {
  int r = 0;
  if (fused_rope && hd == 128 && H % 2 == 0 && Hkv % 2 == 0 && pairs_pay(M, (H + 2 * Hkv) * hd)) r |= 1;
  if (fused_swiglu && (M <= 64 || ((2 * F) % 256 == 0 && pairs_pay(M, 2 * F)))) r |= 2;
  return r;
}

extern "C" int dz_llama_block(const DzLlamaBlock* blk, cudaStream_t stream) {
  if (!blk || blk->B <= 0 || blk->L <= 0 || blk->H <= 0 || blk->Hkv <= 0 || blk->H % blk->Hkv || blk->d % blk->H ||
      !blk->h_in || !blk->h_out || !blk->h_mid || !blk->xn || !blk->qkv || !blk->ctx || !blk->f || !blk->rope_cs)
    return DZ_ERR_ARG;
  const DzLlamaBlock& b = *blk;
  if ((long long)b.B * b.L > 0x7fffffffLL) return DZ_ERR_TOO_LARGE;
  const int M = b.B * b.L, d = b.d, F = b.F, hd = d / b.H, n_qkv = (b.H + 2 * b.Hkv) * hd;
  const int fused = dz_llama_block_fused(M, b.H, b.Hkv, hd, F, b.fused_rope, b.fused_swiglu);
  if (fused != 3 && !b.raw) return DZ_ERR_ARG;
  auto linear = [&](const void* x, const void* w, void* y, int N, int K, const void* res) {
    return dz_linear(x, K, w, K, y, N, nullptr, res, N, M, N, K, 0, 0, 1.0f, b.err, stream);
  };
  int rc = dz_rmsnorm(b.h_in, d, b.ln1_w, b.xn, d, M, d, b.eps, stream);
  if (fused & 1) {
    if (!rc) rc = dz_gemm2_qkv_rope(b.xn, d, b.qkv_w, d, b.qkv, 3 * d, static_cast<const float*>(b.rope_cs), M, d, b.L,
                                    b.pos0, b.n_pos, b.H, b.Hkv, b.err, stream);
  } else {
    if (!rc) rc = linear(b.xn, b.qkv_w, b.raw, n_qkv, d, nullptr);
    if (!rc) rc = dz_rope_qkv(b.raw, n_qkv, b.qkv, 3 * d, b.rope_cs, M, b.L, b.pos0, b.n_pos, b.H, b.Hkv, hd, stream);
  }
  if (!rc) rc = dz_attn_fwd(b.qkv, 3 * d, 0, d, 2 * d, b.ctx, d, b.pad_left, nullptr, nullptr, 0, 0, b.B, b.L, b.H, hd,
                            b.scale, b.err, stream);
  if (!rc) rc = linear(b.ctx, b.out_w, b.h_mid, d, d, b.h_in);
  if (!rc) rc = dz_rmsnorm(b.h_mid, d, b.ln2_w, b.xn, d, M, d, b.eps, stream);
  if (fused & 2) {
    if (!rc && M <= 64)
      rc = dz_gemm_skinny(b.xn, d, b.gu_w, d, b.f, F, nullptr, nullptr, 0, M, F, d, 3, 0, 1.0f, 0, b.err, stream);
    else if (!rc)
      rc = dz_gemm2_bf16_tn(b.xn, d, b.gu_w, d, b.f, F, nullptr, nullptr, 0, M, 2 * F, d, 3, 0, 1.0f, b.err, stream);
  } else {
    if (!rc) rc = linear(b.xn, b.gu_w, b.raw, 2 * F, d, nullptr);
    if (!rc) rc = dz_silu_mul(b.raw, 2 * F, b.f, F, M, F, stream);
  }
  if (!rc) rc = linear(b.f, b.down_w, b.h_out, d, F, b.h_mid);
  return rc;
}
