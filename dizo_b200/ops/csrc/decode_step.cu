// One decoding step through every block of a decoder, launched by one call.
//
// A token's pass through an OPT or LLaMA block is seven kernels of a few microseconds each (norm, q|k|v, attention with
// cache append, output projection, norm, FFN up, FFN down).  Issued one by one from Python they cost about 15 us of host
// time per kernel, several times what they run for.  Here the tensor maps of the weights and workspaces are built once
// for a run of tokens and a step is a plain loop of launches, each a programmatic dependent of the one before: while a
// GEMM drains, the next one already streams its first weight tiles.  The first kernel of a step is launched the ordinary
// way, so everything before the step (the weights included) is complete before any kernel of the step starts.
//
// Measured, per token: OPT-1.3b, one sequence of 300 tokens: 6.5 ms launched from Python, 1.44 ms from here without and
// 1.10 ms with programmatic launches, 0.99 with its products through gemv.cu (the weights at the copy rate: 0.42 ms); LLaMA-2-7b, 16 sequences of 150: 3.80 and
// 3.34 ms (2.0 ms).  What is left is the chain of seven dependent kernels, about 3 us each beyond its bytes.
#include <new>
#include <vector>
#include "common.cuh"
#include "decode.h"
#include "host_util.h"
#include "norm.h"
#include "skinny.h"

// Mirrored by ops/decode.py (ctypes).
extern "C" struct DzDecodeLayer {
  const void *ln1_w, *ln1_b, *qkv_w, *qkv_b, *out_w, *out_b, *ln2_w, *ln2_b, *up_w, *up_b, *down_w, *down_b;
  const void *prefix_k, *prefix_v;
};
extern "C" struct DzDecodeConfig {
  int layers, B, d, F, H, Hkv, hd, n_prefix;
  int rms;             // RMSNorm (no bias) instead of LayerNorm
  int pre_norm;        // norms in front of the sub-layers (else behind the residual sums)
  int act;             // of the FFN: 1 relu, 2 gelu, 3 SwiGLU (up_w = gate rows | up rows)
  int rope_n_pos;      // 0: no rotary embedding
  int cache_rows;      // rows of a sequence in the caches: a step at or past it is refused
  float eps, scale;
  long long ld_prefix, ld_seq, ld_row;
  const void* rope_cs; // fp32 [rope_n_pos][hd / 2][2]
  void *h, *h2, *xn, *qkv, *ctx, *f;   // bf16 workspaces: [B, d] x 3, [B, (H + 2 Hkv) hd], [B, H hd], [B, F]
  uint32_t* err;
};

namespace {

using namespace dz;

struct LayerPlan {
  DzDecodeLayer w;
  CUtensorMap qkv, out, up, down;
};

struct DecodePlan {
  DzDecodeConfig c;
  bool vector;                         // gemv.cu for every product of a block
  CUtensorMap x_h, x_h2, x_xn, x_ctx, x_f;
  std::vector<LayerPlan> layers;
};

bool al16(const void* p) { return p && !(reinterpret_cast<uintptr_t>(p) & 15); }
bool al16_or_null(const void* p) { return !(reinterpret_cast<uintptr_t>(p) & 15); }

int check(const DzDecodeConfig& c, const DzDecodeLayer* L) {
  if (c.layers <= 0 || c.B <= 0 || c.d <= 0 || c.F <= 0 || c.H <= 0 || c.Hkv <= 0 || c.H % c.Hkv || c.hd <= 0 ||
      c.hd > 128 || c.hd * c.H != c.d || c.n_prefix < 0 || c.cache_rows <= 0 || c.act < 0 || c.act > 3 || (c.rms && !c.pre_norm))
    return DZ_ERR_ARG;
  if (c.B > SK_MAX_ROWS || (c.d >> 3) > 2048) return DZ_ERR_TOO_LARGE;
  if ((c.d & 7) || (c.F & 7) || (c.hd & 7) || (c.ld_seq & 7) || (c.ld_row & 7) || (c.n_prefix && (c.ld_prefix & 7)))
    return DZ_ERR_ALIGN;
  if (c.rope_n_pos && !al16(c.rope_cs)) return DZ_ERR_ALIGN;
  for (void* p : {c.h, c.h2, c.xn, c.qkv, c.ctx, c.f}) if (!al16(p)) return DZ_ERR_ALIGN;
  for (int i = 0; i < c.layers; ++i) {
    const DzDecodeLayer& w = L[i];
    for (const void* p : {w.ln1_w, w.ln2_w, w.qkv_w, w.out_w, w.up_w, w.down_w}) if (!al16(p)) return DZ_ERR_ALIGN;
    if (!c.rms && (!al16(w.ln1_b) || !al16(w.ln2_b))) return DZ_ERR_ALIGN;
    for (const void* p : {w.qkv_b, w.out_b, w.up_b, w.down_b}) if (!al16_or_null(p)) return DZ_ERR_ALIGN;
    if (c.n_prefix && (!al16(w.prefix_k) || !al16(w.prefix_v))) return DZ_ERR_ALIGN;
    if (c.act == 3 && w.up_b) return DZ_ERR_ARG;
  }
  return DZ_OK;
}

// Whether a block's products go through gemv.cu.  All or none: it lets its successor start only once its own input is there
// (its reads need that), so a ring kernel behind it would lose its head start.  OPT-1.3b, one sequence, per token: 1.10 ms
// through the ring kernel, 0.99 ms with all four products here, 1.09 with the two small ones.  Beyond about 20 Mi weights a
// matrix, or with more rows beyond 6 Mi, the ring kernel reads W faster by more than the chain gains (gemv_pays).
bool vector_pays(const DzDecodeConfig& c) {
  const long long most = c.B == 1 ? 20LL << 20 : 6LL << 20;
  const long long up = (long long)(c.act == 3 ? 2 : 1) * c.F * c.d;
  const long long qkv = (long long)(c.H + 2 * c.Hkv) * c.hd * c.d;
  return gemv_takes(c.B, c.d) && gemv_takes(c.B, c.F) && up <= most && qkv <= most && (long long)c.d * c.d <= most &&
         (long long)c.d * c.F <= most;
}

int build(DecodePlan& p, const DzDecodeLayer* L) {
  const DzDecodeConfig& c = p.c;
  const int n_qkv = (c.H + 2 * c.Hkv) * c.hd;
  p.vector = vector_pays(c);
  int rc = skinny_map_x(&p.x_h, c.h, c.d, c.B, c.d);
  if (!rc) rc = skinny_map_x(&p.x_h2, c.h2, c.d, c.B, c.d);
  if (!rc) rc = skinny_map_x(&p.x_xn, c.xn, c.d, c.B, c.d);
  if (!rc) rc = skinny_map_x(&p.x_ctx, c.ctx, c.d, c.B, c.d);
  if (!rc) rc = skinny_map_x(&p.x_f, c.f, c.F, c.B, c.F);
  for (int i = 0; i < c.layers && !rc; ++i) {
    LayerPlan l;
    l.w = L[i];
    rc = skinny_map_w(&l.qkv, l.w.qkv_w, c.d, n_qkv, c.d, false);
    if (!rc) rc = skinny_map_w(&l.out, l.w.out_w, c.d, c.d, c.d, false);
    if (!rc) rc = skinny_map_w(&l.up, l.w.up_w, c.d, c.act == 3 ? 2 * c.F : c.F, c.d, c.act == 3);
    if (!rc) rc = skinny_map_w(&l.down, l.w.down_w, c.F, c.d, c.F, false);
    if (!rc) p.layers.push_back(l);
  }
  return rc;
}

}  // namespace

// *plan receives a handle for dz_decode_step; the caller keeps every tensor named here alive until dz_decode_plan_free.
extern "C" int dz_decode_plan_create(const DzDecodeConfig* cfg, const DzDecodeLayer* layers, void** plan) {
  if (!cfg || !layers || !plan) return DZ_ERR_ARG;
  *plan = nullptr;
  if (int rc = check(*cfg, layers)) return rc;
  DecodePlan* p = nullptr;
  int rc;
  try {
    p = new DecodePlan();
    p->c = *cfg;
    p->layers.reserve(cfg->layers);
    rc = build(*p, layers);
  } catch (const std::bad_alloc&) {
    rc = DZ_ERR_TOO_LARGE;
  }
  if (rc) {
    delete p;
    return rc;
  }
  *plan = p;
  return DZ_OK;
}

extern "C" void dz_decode_plan_free(void* plan) { delete static_cast<DecodePlan*>(plan); }

// cfg.h [B, d] (the embedded tokens) -> the last block's output, in cfg.h.  k_cache / v_cache: one pointer per layer;
// row t of every sequence is written, columns [pad_left, t] are attended to.  Asynchronous on `stream`.
extern "C" int dz_decode_step(const void* plan, const void* const* k_cache, const void* const* v_cache, int t,
                              const int* pad_left, cudaStream_t stream) {
  if (!plan || !k_cache || !v_cache) return DZ_ERR_ARG;
  const DecodePlan& p = *static_cast<const DecodePlan*>(plan);
  const DzDecodeConfig& c = p.c;
  if (t < 0 || t >= c.cache_rows) return DZ_ERR_ARG;            // row t of every sequence is written
  if ((long long)c.n_prefix + t + 1 > DA_MAX_KEYS) return DZ_ERR_TOO_LARGE;
  if (c.rope_n_pos && c.n_prefix + t >= c.rope_n_pos) return DZ_ERR_ARG;
  for (int i = 0; i < c.layers; ++i) {
    if (!k_cache[i] || !v_cache[i]) return DZ_ERR_ARG;
    if (!al16(k_cache[i]) || !al16(v_cache[i])) return DZ_ERR_ALIGN;
  }
  const int n_qkv = (c.H + 2 * c.Hkv) * c.hd;
  auto B16 = [](const void* q) { return static_cast<const __nv_bfloat16*>(q); };
  bool first = true;
  auto norm = [&](const void* x, const void* w, const void* b, void* y) {
    const bool dep = !first;
    first = false;
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(y);
    return c.rms ? rmsnorm_launch(B16(x), c.d, B16(w), o, c.d, c.B, c.d, c.eps, dep, stream)
                 : layernorm_launch(B16(x), c.d, B16(w), B16(b), o, c.d, c.B, c.d, c.eps, dep, stream);
  };
  auto gemm = [&](const CUtensorMap& w, const CUtensorMap& x, const void* W, const void* X, void* out, int N, int K,
                  const void* bias, const void* residual, int act) {
    SkinnyArgs a{};
    a.M = c.B; a.N = N; a.K = K; a.out = out; a.ldo = N; a.bias = B16(bias); a.residual = B16(residual);
    a.ldr = N; a.act = act; a.out_scale = 1.0f; a.err = c.err;
    a.w_static = first ? 0 : 1;
    const bool dep = !first;
    first = false;
    if (p.vector) return gemv_launch(W, K, X, K, a, dep, stream);
    return skinny_launch(w, x, a, 0, true, dep, stream);
  };
  for (int i = 0; i < c.layers; ++i) {
    const LayerPlan& l = p.layers[i];
    int rc = DZ_OK;
    if (c.pre_norm) rc = norm(c.h, l.w.ln1_w, l.w.ln1_b, c.xn);
    if (!rc) rc = gemm(l.qkv, c.pre_norm ? p.x_xn : p.x_h, l.w.qkv_w, c.pre_norm ? c.xn : c.h, c.qkv, n_qkv, c.d, l.w.qkv_b, nullptr, 0);
    if (rc) return rc;
    DecodeAttnArgs a{};
    a.q = B16(c.qkv); a.ldq = n_qkv;
    a.k_new = a.q + c.H * c.hd;
    a.v_new = a.k_new + c.Hkv * c.hd;
    a.rep = c.H / c.Hkv;
    a.rope = c.rope_n_pos ? static_cast<const float2*>(c.rope_cs) : nullptr;
    a.rope_pos = c.n_prefix + t;
    a.kc = static_cast<__nv_bfloat16*>(const_cast<void*>(k_cache[i]));
    a.vc = static_cast<__nv_bfloat16*>(const_cast<void*>(v_cache[i]));
    a.ld_seq = c.ld_seq; a.ld_row = c.ld_row;
    a.pk = B16(l.w.prefix_k); a.pv = B16(l.w.prefix_v); a.ldp = c.ld_prefix; a.n_prefix = c.n_prefix;
    a.pad_left = pad_left; a.kv_len = t + 1; a.hd = c.hd; a.scale = c.scale;
    a.out = static_cast<__nv_bfloat16*>(c.ctx); a.ldo = c.d;
    rc = decode_attn_launch(a, c.B, c.H, true, stream);
    if (rc) return rc;
    if (c.pre_norm) {
      rc = gemm(l.out, p.x_ctx, l.w.out_w, c.ctx, c.h, c.d, c.d, l.w.out_b, c.h, 0);
      if (!rc) rc = norm(c.h, l.w.ln2_w, l.w.ln2_b, c.xn);
      if (!rc) rc = gemm(l.up, p.x_xn, l.w.up_w, c.xn, c.f, c.F, c.d, l.w.up_b, nullptr, c.act);
      if (!rc) rc = gemm(l.down, p.x_f, l.w.down_w, c.f, c.h, c.d, c.F, l.w.down_b, c.h, 0);
    } else {
      rc = gemm(l.out, p.x_ctx, l.w.out_w, c.ctx, c.h2, c.d, c.d, l.w.out_b, c.h, 0);
      if (!rc) rc = norm(c.h2, l.w.ln1_w, l.w.ln1_b, c.h);
      if (!rc) rc = gemm(l.up, p.x_h, l.w.up_w, c.h, c.f, c.F, c.d, l.w.up_b, nullptr, c.act);
      if (!rc) rc = gemm(l.down, p.x_f, l.w.down_w, c.f, c.h2, c.d, c.F, l.w.down_b, c.h, 0);
      if (!rc) rc = norm(c.h2, l.w.ln2_w, l.w.ln2_b, c.h);
    }
    if (rc) return rc;
  }
  return DZ_OK;
}
