// Generation-time kernels: single-token attention over a KV cache and token sampling.
//
// decode_attn: one new query per sequence against the cached keys / values (plus optional
// prefix rows).  One pass: a group of 8 (head dim <= 64) or 16 lanes owns a key, reads its K and V
// rows with one 16-byte load each and keeps a running (max, sum, weighted V) of its own; the
// groups meet at the end, across the warps through shared memory and across a cluster of CTAs that
// share the keys of one (sequence, head) through distributed shared memory.  In a decoding step the
// kernel also takes the raw q | k | v row of the new token: it rotates q and k (rotary models),
// appends k and v to the cache and attends to the new key from registers, which replaces the rotary
// kernel and two strided copies per layer.  OPT-1.3b, one sequence of 300 tokens, per layer: 20 us before (32 CTAs, two
// passes over the keys) and 5.8 us now; LLaMA-2-7b, 16 sequences of 180: 16.7 + 7.7 us with the rotary kernel, 14 us now.
//
// sample_topk_topp: temperature -> top-k -> nucleus (top-p) filtering and one draw per row,
// (the row's probabilities stay in shared memory: 677 us -> 63 us for 16 rows of 32000)
// without sorting the vocabulary: the k-th largest logit and the nucleus threshold are found
// by bisection on the value (each step is one block-wide count / mass reduction), the draw
// walks the kept probability mass with a uniform from Philox(seed, row).  Semantics follow
// Hugging Face's logits warpers (temperature, TopK, TopP in that order), which is what the
// reference's model.generate applies (large_models/run.py:280-287).
#include "common.cuh"
#include "cluster2sm.cuh"
#include "decode.h"
#include "host_util.h"
#include "pdl.cuh"
#include "philox.cuh"

namespace dz {

constexpr int DA_WARPS = 8;
constexpr int DA_FEW_KEYS = 64;
constexpr int DA_UNROLL = 4;      // keys in flight per lane group

__device__ __forceinline__ void unpack8(const uint4& r, float (&f)[8]) {
  f[0] = bf16_lo(r.x); f[1] = bf16_hi(r.x); f[2] = bf16_lo(r.y); f[3] = bf16_hi(r.y);
  f[4] = bf16_lo(r.z); f[5] = bf16_hi(r.z); f[6] = bf16_lo(r.w); f[7] = bf16_hi(r.w);
}

// LPK: lanes per key (8 columns each); WARPS of a CTA.  grid (H * splits, B), cluster (splits, 1, 1).
template <int LPK, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
decode_attn_kernel(const DecodeAttnArgs p) {
  constexpr int KPW = 32 / LPK;               // keys a warp reads at a time
  __shared__ float s_q[128];
  __shared__ float s_kv[2][128];              // the new key and value (append mode)
  __shared__ float s_m[WARPS], s_l[WARPS];
  __shared__ float s_acc[WARPS][128];
  __shared__ float s_cta[2 + 128];            // this CTA's (max, sum, weighted V)
  const int rank = (int)blockIdx.x % p.splits, h = (int)blockIdx.x / p.splits, b = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hd = p.hd;
  pdl_trigger();
  pdl_wait();
  const int pad = p.pad_left ? p.pad_left[b] : 0;
  const long long seq = (long long)b * p.ld_seq + h * hd;
  const bool append = p.k_new != nullptr;
  const int cached = append ? p.kv_len - 1 : p.kv_len;       // columns read from the cache
  // ---- q (and the new k, v) into shared memory; rotary pairs (j, j + hd/2)
  if (tid < hd) {
    const int half = hd >> 1;
    const int j = tid < half ? tid : tid - half;
    float2 cs = make_float2(1.f, 0.f);
    if (p.rope) cs = ld_table(p.rope + (long long)p.rope_pos * half + j);
    // the new token's row is the predecessor's output: read past L1
    auto fresh = [](const __nv_bfloat16* e) {
      return __uint_as_float(static_cast<uint32_t>(__ldcg(reinterpret_cast<const unsigned short*>(e))) << 16);
    };
    auto rotated = [&](const __nv_bfloat16* row) {
      const float a = fresh(row + j), c = fresh(row + j + half);
      const float r = tid < half ? a * cs.x - c * cs.y : c * cs.x + a * cs.y;
      return __bfloat162float(__float2bfloat16(r));           // q and k are held in bf16
    };
    const __nv_bfloat16* qr = p.q + (long long)b * p.ldq + h * hd;
    s_q[tid] = (p.rope ? rotated(qr) : fresh(qr + tid)) * p.scale;
    if (append) {
      const int hk = h / p.rep;
      const __nv_bfloat16* kr = p.k_new + (long long)b * p.ldq + hk * hd;
      const __nv_bfloat16* vr = p.v_new + (long long)b * p.ldq + hk * hd;
      const float k = p.rope ? rotated(kr) : fresh(kr + tid);
      const float v = fresh(vr + tid);
      s_kv[0][tid] = k;
      s_kv[1][tid] = v;
      if (rank == 0) {
        const long long at = seq + (long long)cached * p.ld_row + tid;
        if (DZ_STORE_OK(p.kc + at, 2)) p.kc[at] = __float2bfloat16(k);
        if (DZ_STORE_OK(p.vc + at, 2)) p.vc[at] = __float2bfloat16(v);
      }
    }
  }
  __syncthreads();
  const int grp = lane / LPK, lg = lane % LPK;
  const bool col_ok = lg * 8 < hd;
  float q[8], acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    q[c] = col_ok ? s_q[lg * 8 + c] : 0.f;
    acc[c] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  auto group_sum = [&](float s) {
#pragma unroll
    for (int off = LPK / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
  };
  if (append && rank == 0 && warp == 0) {     // the new key, kept by the first group
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) s = fmaf(q[c], col_ok ? s_kv[0][lg * 8 + c] : 0.f, s);
    s = group_sum(s);
    if (grp == 0 && p.kv_len - 1 >= pad) {
      m = s;
      l = 1.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = col_ok ? s_kv[1][lg * 8 + c] : 0.f;
    }
  }
  // ---- prefix rows, then the cached columns right of the padding
  const int first = min(pad, cached);
  const int n = p.n_prefix + cached - first;
  const __nv_bfloat16* kbase = p.kc + seq + (long long)(first - p.n_prefix) * p.ld_row;
  const __nv_bfloat16* vbase = p.vc + seq + (long long)(first - p.n_prefix) * p.ld_row;
  const int stride = p.splits * WARPS * KPW;
  // the trip count is the same for every lane of a warp (the shuffles need all of them)
  for (int jb = (rank * WARPS + warp) * KPW; jb < n; jb += stride * DA_UNROLL) {
    uint4 kr[DA_UNROLL], vr[DA_UNROLL];
#pragma unroll
    for (int u = 0; u < DA_UNROLL; ++u) {
      const int j = jb + u * stride + grp;
      kr[u] = make_uint4(0u, 0u, 0u, 0u);
      vr[u] = kr[u];
      if (j < n && col_ok) {
        const bool pre = j < p.n_prefix;
        const __nv_bfloat16* ks = pre ? p.pk + (long long)j * p.ldp + h * hd : kbase + (long long)j * p.ld_row;
        const __nv_bfloat16* vs = pre ? p.pv + (long long)j * p.ldp + h * hd : vbase + (long long)j * p.ld_row;
        kr[u] = *reinterpret_cast<const uint4*>(ks + lg * 8);
        vr[u] = *reinterpret_cast<const uint4*>(vs + lg * 8);
      }
    }
    float s[DA_UNROLL], m_new = m;
#pragma unroll
    for (int u = 0; u < DA_UNROLL; ++u) {
      float k[8], t = 0.f;
      unpack8(kr[u], k);
#pragma unroll
      for (int c = 0; c < 8; ++c) t = fmaf(q[c], k[c], t);
      t = group_sum(t);
      s[u] = jb + u * stride + grp < n ? t : -INFINITY;
      m_new = fmaxf(m_new, s[u]);
    }
    const float m_ref = m_new == -INFINITY ? 0.f : m_new;     // a group without a key so far
    const float keep = __expf(m - m_ref);
    l *= keep;
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] *= keep;
#pragma unroll
    for (int u = 0; u < DA_UNROLL; ++u) {
      const float e = __expf(s[u] - m_ref);
      float v[8];
      unpack8(vr[u], v);
      l += e;
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = fmaf(e, v[c], acc[c]);
    }
    m = m_new;
  }
  // ---- groups of the warp, warps of the CTA, CTAs of the cluster
#pragma unroll
  for (int off = LPK; off < 32; off <<= 1) {
    const float mo = __shfl_xor_sync(0xffffffffu, m, off), lo = __shfl_xor_sync(0xffffffffu, l, off);
    const float mn = fmaxf(m, mo), ref = mn == -INFINITY ? 0.f : mn;
    const float fa = __expf(m - ref), fb = __expf(mo - ref);
    l = l * fa + lo * fb;
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = acc[c] * fa + __shfl_xor_sync(0xffffffffu, acc[c], off) * fb;
    m = mn;
  }
  if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
  if (grp == 0 && col_ok) {
#pragma unroll
    for (int c = 0; c < 8; ++c) s_acc[warp][lg * 8 + c] = acc[c];
  }
  __syncthreads();
  if (tid < hd) {
    float mm = s_m[0];
    for (int w = 1; w < WARPS; ++w) mm = fmaxf(mm, s_m[w]);
    const float ref = mm == -INFINITY ? 0.f : mm;
    float o = 0.f, ll = 0.f;
    for (int w = 0; w < WARPS; ++w) {
      const float f = __expf(s_m[w] - ref);
      o = fmaf(s_acc[w][tid], f, o);
      ll = fmaf(s_l[w], f, ll);
    }
    if (p.splits == 1) {
      __nv_bfloat16* op = p.out + (long long)b * p.ldo + h * hd + tid;
      if (DZ_STORE_OK(op, 2)) *op = __float2bfloat16(o / ll);
    } else {
      s_cta[2 + tid] = o;
      if (tid == 0) { s_cta[0] = mm; s_cta[1] = ll; }
    }
  }
  if (p.splits > 1) {
    __syncthreads();
    cluster_sync_all();
    if (rank == 0 && tid < hd) {
      const uint32_t base = smem_u32(s_cta);
      float mm = -INFINITY, ms[8], ls[8], os[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {             // every load in flight before the first use
        ms[r] = r < p.splits ? ld_dsmem_f32(map_to_cta(base, r)) : -INFINITY;
        ls[r] = r < p.splits ? ld_dsmem_f32(map_to_cta(base + 4, r)) : 0.f;
        os[r] = r < p.splits ? ld_dsmem_f32(map_to_cta(base + 8 + tid * 4, r)) : 0.f;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) mm = fmaxf(mm, ms[r]);
      const float ref = mm == -INFINITY ? 0.f : mm;
      float o = 0.f, ll = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float f = __expf(ms[r] - ref);
        o = fmaf(os[r], f, o);
        ll = fmaf(ls[r], f, ll);
      }
      __nv_bfloat16* op = p.out + (long long)b * p.ldo + h * hd + tid;
      if (DZ_STORE_OK(op, 2)) *op = __float2bfloat16(o / ll);
    }
    __syncwarp();
    cluster_sync_all();                       // nobody leaves while rank 0 may still read its partial result
  }
}

int decode_attn_launch(DecodeAttnArgs a, int B, int H, bool dependent, cudaStream_t stream) {
  // CTAs that share one (sequence, head): up to two CTAs per SM over the launch, at least 64 keys each
  int s = 2 * sm_count() / (B * H > 0 ? B * H : 1);
  const int by_keys = (a.n_prefix + a.kv_len) / 64;
  if (s > by_keys) s = by_keys;
  a.splits = s < 1 ? 1 : s > 8 ? 8 : s;
  const dim3 grid((unsigned)(H * a.splits), (unsigned)B);
  auto launch = [&](auto kern, int threads) {
    return cuda_rc(pdl_launch(kern, grid, threads, 0, stream, a.splits, dependent, a));
  };
  // Few keys and more CTAs than run at once (74 registers: three CTAs of 256 threads an SM): CTAs of four warps, of which
  // twice as many fit.  Us, 8 / 4 warps: 16 sequences of 32 heads of 128, 16 keys 5.1 / 3.5, 64 keys 5.6 / 4.7; 64 sequences
  // of 12 heads of 64, one key 4.7 / 3.2.  With more keys it depends: 32 sequences of 40 heads of 128, 301 keys 35.9 / 39.9.
  const bool few = a.n_prefix + a.kv_len <= DA_FEW_KEYS && (long long)B * H > 2LL * sm_count();
  if (a.hd <= 64) return few ? launch(decode_attn_kernel<8, 4>, 128) : launch(decode_attn_kernel<8, DA_WARPS>, DA_WARPS * 32);
  return few ? launch(decode_attn_kernel<16, 4>, 128) : launch(decode_attn_kernel<16, DA_WARPS>, DA_WARPS * 32);
}

constexpr int SP_THREADS = 512;

__device__ __forceinline__ float block_sum(float v, float* s_red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < SP_THREADS / 32; ++w) t += s_red[w];
  __syncthreads();
  return t;
}
__device__ __forceinline__ float block_max(float v, float* s_red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = -INFINITY;
  for (int w = 0; w < SP_THREADS / 32; ++w) t = fmaxf(t, s_red[w]);
  __syncthreads();
  return t;
}

constexpr int SP_CACHE = 50 * 1024;    // vocabulary entries whose probabilities fit in shared memory
constexpr int SP_LIST = 2048;          // kept tokens collected per pass of the draw

// One CTA per row.  do_sample == 0: argmax.  CACHED: the row's probabilities are computed once into shared memory;
// the bisection of the nucleus threshold (32 passes over the row) and the draw read them there.
template <bool CACHED>
__global__ void __launch_bounds__(SP_THREADS)
sample_topk_topp_kernel(const float* __restrict__ logits, long long ld, int V, float temperature,
                        int top_k, float top_p, int do_sample, unsigned long long seed,
                        unsigned long long offset, int* __restrict__ done, const int* __restrict__ eos, int n_eos,
                        int pad_id, int* __restrict__ out) {
  extern __shared__ float s_prob[];            // [V] when CACHED
  __shared__ float s_red[SP_THREADS / 32];
  __shared__ int s_idx[SP_THREADS / 32];
  __shared__ __align__(16) float s_list[SP_LIST];
  __shared__ int s_list_i[SP_LIST];
  __shared__ int s_cnt[SP_THREADS / 32];
  __shared__ float s_run;
  __shared__ int s_found;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* lg = logits + (long long)row * ld;
  // the row's token: padding once the sequence has ended, which it does with an end-of-sequence id
  auto emit = [&](int tok) {
    if (done) {
      if (done[row]) {
        tok = pad_id;
      } else {
        for (int e = 0; e < n_eos; ++e)
          if (tok == eos[e] && DZ_STORE_OK(done + row, 4)) done[row] = 1;
      }
    }
    if (DZ_STORE_OK(out + row, 4)) out[row] = tok;
  };
  const float inv_t = (do_sample && temperature > 0.f) ? 1.0f / temperature : 1.0f;
  // ---- maximum (and argmax with the lowest index on ties)
  float best = -INFINITY;
  int best_i = V;
  auto larger = [&](float x, int i) {
    x *= inv_t;
    if (x > best) { best = x; best_i = i; }
  };
  const int wide = (reinterpret_cast<uintptr_t>(lg) & 15) ? 0 : V & ~3;     // rows on a 16-byte boundary: four at a time
#pragma unroll 4
  for (int i = tid * 4; i < wide; i += SP_THREADS * 4) {
    const float4 x = *reinterpret_cast<const float4*>(lg + i);
    larger(x.x, i); larger(x.y, i + 1); larger(x.z, i + 2); larger(x.w, i + 3);
  }
  for (int i = wide + tid; i < V; i += SP_THREADS) larger(lg[i], i);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    float ob = __shfl_xor_sync(0xffffffffu, best, off);
    int oi = __shfl_xor_sync(0xffffffffu, best_i, off);
    if (ob > best || (ob == best && oi < best_i)) { best = ob; best_i = oi; }
  }
  if (lane == 0) { s_red[warp] = best; s_idx[warp] = best_i; }
  __syncthreads();
  float m = s_red[0];
  int mi = s_idx[0];
  for (int w = 1; w < SP_THREADS / 32; ++w)
    if (s_red[w] > m || (s_red[w] == m && s_idx[w] < mi)) { m = s_red[w]; mi = s_idx[w]; }
  __syncthreads();
  if (!do_sample) {
    if (tid == 0) emit(mi);
    return;
  }
  // ---- top-k: smallest logit that is still kept = k-th largest, by bisection on the value
  float lo_keep = -INFINITY;
  if (top_k > 0 && top_k < V) {
    float lo = m - 60.f, hi = m;                     // logits more than 60 below the max carry no mass
    for (int it = 0; it < 32; ++it) {
      float mid = 0.5f * (lo + hi);
      float c = 0.f;
#pragma unroll 8
      for (int i = tid; i < V; i += SP_THREADS) c += (lg[i] * inv_t >= mid) ? 1.f : 0.f;
      c = block_sum(c, s_red);
      if (c >= (float)top_k) lo = mid; else hi = mid;  // keep at least k tokens at threshold lo
    }
    lo_keep = lo;
  }
  // ---- normaliser of the top-k set
  float z = 0.f;
#pragma unroll 8
  for (int i = tid; i < V; i += SP_THREADS) {
    float x = lg[i] * inv_t;
    float e = 0.f;
    if (x >= lo_keep) {
      e = __expf(x - m);
      z += e;
    }
    if (CACHED) s_prob[i] = e;
  }
  z = block_sum(z, s_red);
  if (CACHED) {
    // each thread rescales (and, in the bisection, reads) the entries it wrote; a token outside the top-k set keeps 0,
    // which no threshold below keeps: its mass is 0 either way
    for (int i = tid; i < V; i += SP_THREADS) s_prob[i] = s_prob[i] / z;
  }
  auto prob = [&](int i) -> float {                  // 0 outside the top-k set
    if (CACHED) return s_prob[i];
    const float x = lg[i] * inv_t;
    return x >= lo_keep ? __expf(x - m) / z : 0.f;
  };
  // ---- nucleus: largest threshold whose kept mass still reaches top_p
  float p_keep = 0.f;                                // keep probabilities >= p_keep
  if (top_p > 0.f && top_p < 1.f) {
    float lo = 0.f, hi = 1.0f;
    for (int it = 0; it < 32; ++it) {
      float mid = 0.5f * (lo + hi);
      float mass = 0.f;
#pragma unroll 8
      for (int i = tid; i < V; i += SP_THREADS) {
        const float pr = prob(i);
        if (pr >= mid) mass += pr;
      }
      mass = block_sum(mass, s_red);
      if (mass >= top_p) lo = mid; else hi = mid;
    }
    p_keep = lo;
  }
  // ---- kept mass, then walk it with one uniform
  float kept = 0.f;
#pragma unroll 8
  for (int i = tid; i < V; i += SP_THREADS) {
    const float pr = prob(i);
    if (pr >= p_keep) kept += pr;
  }
  kept = block_sum(kept, s_red);                     // its barriers also publish s_prob to the whole block
  Philox4 r = philox4x32<10>((uint32_t)row, (uint32_t)offset, (uint32_t)(offset >> 32), 3u,
                             (uint32_t)seed, (uint32_t)(seed >> 32));
  const float u = ((r.x >> 8) + 0.5f) * (1.0f / 16777216.0f) * kept;
  // The running mass is a sum in index order, one addition after the other: the tokens that are kept with a positive
  // probability are collected in order (SP_LIST indices at a time, four per thread), then one thread adds them up.  A
  // zero never changes the sum, so only kept tokens cost a serial addition, not the vocabulary.
  if (tid == 0) { s_run = 0.f; s_found = -1; }
  for (int base = 0; base < V; base += SP_LIST) {
    __syncthreads();
    if (s_found >= 0) break;
    constexpr int PER = SP_LIST / SP_THREADS;
    float pr[PER];
    int cnt = 0;
#pragma unroll
    for (int c = 0; c < PER; ++c) {
      const int i = base + tid * PER + c;
      pr[c] = 0.f;
      if (i < V) {
        const float q = prob(i);
        if (q >= p_keep) pr[c] = q;
      }
      cnt += pr[c] > 0.f ? 1 : 0;
    }
    int before = cnt;                                // inclusive scan over the warp
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, before, off);
      if (lane >= off) before += t;
    }
    if (lane == 31) s_cnt[warp] = before;
    __syncthreads();
    int at = before - cnt, n = 0;
    for (int w = 0; w < SP_THREADS / 32; ++w) {
      if (w < warp) at += s_cnt[w];
      n += s_cnt[w];
    }
#pragma unroll
    for (int c = 0; c < PER; ++c) {
      if (pr[c] > 0.f) {
        s_list[at] = pr[c];
        s_list_i[at] = base + tid * PER + c;
        ++at;
      }
    }
    __syncthreads();
    if (tid == 0) {
      // 16 at a time, the next ones loaded ahead: a running sum of positive terms never falls, so it is compared with u once
      // per 16 and only the 16 that reach it are walked again.  One row of 32000 tokens without top-k and top-p: 898 us with
      // a comparison after each addition, behind which every load waited, and 166 us.
      float run = s_run;
      int t = 0;
      const float4* l4 = reinterpret_cast<const float4*>(s_list);
      float4 nx[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) nx[j] = l4[j];
      for (; t + 16 <= n; t += 16) {
        float p[16], r = run;
#pragma unroll
        for (int j = 0; j < 4; ++j) { p[4 * j] = nx[j].x; p[4 * j + 1] = nx[j].y; p[4 * j + 2] = nx[j].z; p[4 * j + 3] = nx[j].w; }
        if (t + 32 <= n) {
#pragma unroll
          for (int j = 0; j < 4; ++j) nx[j] = l4[(t >> 2) + 4 + j];
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) r += p[j];
        if (r >= u) break;
        run = r;
      }
      for (; t < n; ++t) {
        run += s_list[t];
        if (run >= u) { s_found = s_list_i[t]; break; }
      }
      s_run = run;
    }
  }
  __syncthreads();
  if (tid == 0) emit(s_found >= 0 ? s_found : mi);
}

}  // namespace dz

using namespace dz;
DZ_DEBUG_TU(decode)

extern "C" int dz_decode_attn(const void* q, long long ldq, const void* kc, const void* vc,
                              long long ld_seq, long long ld_row, const void* pk, const void* pv,
                              long long ldp, int n_prefix, const int* pad_left, int kv_len, int B,
                              int H, int hd, float scale, void* out, long long ldo,
                              cudaStream_t stream) {
  if (!q || !kc || !vc || !out || B <= 0 || H <= 0 || kv_len <= 0) return DZ_ERR_ARG;
  if (hd > 128 || (hd & 7) || (ld_row & 7) || (ld_seq & 7) || (n_prefix > 0 && (!pk || !pv || (ldp & 7))))
    return DZ_ERR_ARG;
  for (const void* rows : {kc, vc, pk, pv})                       // read in 16-byte vectors
    if (reinterpret_cast<uintptr_t>(rows) & 15) return DZ_ERR_ALIGN;
  if ((long long)n_prefix + kv_len > DA_MAX_KEYS) return DZ_ERR_TOO_LARGE;
  DecodeAttnArgs a{};
  a.q = (const __nv_bfloat16*)q; a.ldq = ldq;
  // without a new key the cache is only read
  a.kc = const_cast<__nv_bfloat16*>((const __nv_bfloat16*)kc);
  a.vc = const_cast<__nv_bfloat16*>((const __nv_bfloat16*)vc);
  a.ld_seq = ld_seq; a.ld_row = ld_row;
  a.pk = (const __nv_bfloat16*)pk; a.pv = (const __nv_bfloat16*)pv; a.ldp = ldp; a.n_prefix = n_prefix;
  a.pad_left = pad_left; a.kv_len = kv_len; a.hd = hd; a.rep = 1; a.scale = scale;
  a.out = (__nv_bfloat16*)out; a.ldo = ldo;
  return decode_attn_launch(a, B, H, false, stream);
}

// One token per row.  done [rows] (optional): rows whose entry is set give pad_id, and a row that draws one of the n_eos
// ids of `eos` sets its entry.
extern "C" int dz_sample_step(const float* logits, long long ld, int rows, int V, float temperature, int top_k,
                              float top_p, int do_sample, unsigned long long seed, unsigned long long offset,
                              int* done, const int* eos, int n_eos, int pad_id, int* out, cudaStream_t stream) {
  if (!logits || !out || rows <= 0 || V <= 0 || n_eos < 0 || (n_eos > 0 && (!eos || !done))) return DZ_ERR_ARG;
  // the probabilities of the row stay in shared memory while they fit beside the static arrays
  if (do_sample && V <= SP_CACHE) {
    auto kern = sample_topk_topp_kernel<true>;
    static PerDeviceFlag configured;
    if (int rc_cfg = ensure_dyn_smem(configured, kern, SP_CACHE * 4)) return rc_cfg;
    kern<<<rows, SP_THREADS, sizeof(float) * (size_t)V, stream>>>(logits, ld, V, temperature, top_k, top_p, do_sample,
                                                                 seed, offset, done, eos, n_eos, pad_id, out);
  } else {
    sample_topk_topp_kernel<false><<<rows, SP_THREADS, 0, stream>>>(logits, ld, V, temperature, top_k, top_p, do_sample,
                                                                    seed, offset, done, eos, n_eos, pad_id, out);
  }
  return cuda_rc(cudaGetLastError());
}
