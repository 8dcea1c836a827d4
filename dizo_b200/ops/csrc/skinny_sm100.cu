// GEMM for few output tiles on sm_100a:  out[M,N] = epilogue( A[M,K] * W[N,K]^T ), K split over a cluster of CTAs.
//
// Decoding, the option rows of a loss and the last block's tail multiply a few rows with whole weight matrices: the
// bytes of W bound the time and the only question is how to keep enough of them in flight on every SM.  The 128-row
// tile kernel (gemm_sm100.cu) spends half of its shared memory and TMA traffic on zero rows of A and runs one CTA per
// 128 or 256 columns - 16 CTAs for N = 2048 - so it read W at 0.5 to 2 TB/s.  Here
//   * the operands are swapped: the tcgen05 "A" operand is a tile of 128 rows of W, the activations are the "B" operand
//     padded to NB = 16 / 32 / 64 columns, D[128 features x NB rows] accumulates in TMEM; a stage is 16 KB of W and 2 to
//     8 KB of activations;
//   * K is split over a cluster of up to 8 CTAs where N gives too few tiles to fill the chip; the partial tiles meet
//     through distributed shared memory in a fixed order (deterministic, no workspace, no second launch);
//   * two CTAs fit on an SM (about 108 KB each), so the next launch of a decoding step can fill its ring while this one
//     drains (programmatic dependent launch; `w_static` says that W may be read before the predecessor has finished).
//
// The same kernel with 128-row activation tiles (NB = 128, one CTA per SM) takes the products of small models whose tiles
// leave most SMs idle: 360 x 1024 outputs are 24 tiles of 128 x 128.
//
// Warp 0: TMA producer; warp 1: TMEM, MMA issue; warps 2-5: accumulator -> shared memory; all warps: reduction over
// the cluster and epilogue.  Every wait is bounded (common.cuh).
#include "common.cuh"
#include "cluster2sm.cuh"
#include "host_util.h"
#include "pdl.cuh"
#include "skinny.h"

namespace dz {

constexpr int SK_BM = 128;           // rows of W per tile
constexpr int SK_BK = 64;
constexpr int SK_THREADS = 192;

template <int NB>
struct SkinnySmem {
  static constexpr int W_BYTES = SK_BM * SK_BK * 2;
  static constexpr int X_BYTES = NB * SK_BK * 2;
  static constexpr int STAGE = W_BYTES + X_BYTES;
  static constexpr int STAGES = NB <= 16 ? 6 : NB <= 32 ? 5 : NB <= 64 ? 4 : 6;
  static constexpr int TOTAL = STAGES * STAGE + 1024;
  static_assert(STAGES * STAGE >= NB * SK_BM * 4, "the partial tile reuses the ring");
  static_assert(TOTAL <= 226 * 1024 && (NB > 64 || 2 * (TOTAL + 1024) <= 227 * 1024), "two CTAs per SM up to 64 rows");
};

template <int NB>
__global__ void __launch_bounds__(SK_THREADS, NB > 64 ? 1 : 2)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   const SkinnyArgs p) {
  using S = SkinnySmem<NB>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[S::STAGES], bar_empty[S::STAGES], bar_acc;
  __shared__ uint32_t s_tmem_base;
  __shared__ volatile int s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  constexpr uint32_t TMEM_COLS = NB < 32 ? 32 : NB;
  const int rank = (int)blockIdx.x % p.splits;
  const int tile = (int)blockIdx.x / p.splits % p.num_n;       // of W
  const int m0 = (int)blockIdx.x / p.splits / p.num_n * NB;    // first activation row
  const int rows = min(NB, p.M - m0);
  const int kb0 = rank * p.kb_per_cta;
  const int n_kb = min(p.kb_per_cta, p.num_kb - kb0);      // >= 1: the host leaves no CTA of a cluster without work

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_acc), 1);
    fence_mbar_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&s_tmem_base), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;
  pdl_trigger();

  if (warp == 0) {
    if (elect_one()) {
      // ---------------------------------------------------------- TMA producer
      auto load_w = [&](int i, int stage) {
        const uint32_t full = smem_u32(&bar_full[stage]);
        const uint32_t dst = smem_base + stage * S::STAGE;
        mbar_arrive_expect_tx(full, S::STAGE);
        const int k = (kb0 + i) * SK_BK;
        if (p.act == 3) {
          // 64 gate rows above the 64 up rows of the same columns (the box is 64 rows high)
          tma_load_2d(dst, &tmW, full, k, tile * (SK_BM / 2));
          tma_load_2d(dst + S::W_BYTES / 2, &tmW, full, k, p.N + tile * (SK_BM / 2));
        } else {
          tma_load_2d(dst, &tmW, full, k, tile * SK_BM);
        }
      };
      auto load_x = [&](int i, int stage) {
        tma_load_2d(smem_base + stage * S::STAGE + S::W_BYTES, &tmX, smem_u32(&bar_full[stage]), (kb0 + i) * SK_BK, m0);
      };
      const int head = p.w_static ? min(n_kb, S::STAGES) : 0;
      for (int i = 0; i < head; ++i) load_w(i, i);           // the ring's first turn: every stage is free
      pdl_wait();
      for (int i = 0; i < head; ++i) load_x(i, i);
      for (int i = head; i < n_kb; ++i) {
        const int stage = i % S::STAGES;
        if (!mbar_wait(smem_u32(&bar_empty[stage]), ((i / S::STAGES) & 1) ^ 1, &s_abort, p.err, ERR_WAIT_EMPTY)) break;
        load_w(i, stage);
        load_x(i, stage);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // ---------------------------------------------------------- MMA issuer
      constexpr uint32_t idesc = umma_idesc_bf16(SK_BM, NB);
      pdl_wait();                     // the time limits below count from here, not from an early start beside predecessors
      bool ok = true;
      for (int i = 0; i < n_kb; ++i) {
        const int stage = i % S::STAGES;
        ok = mbar_wait(smem_u32(&bar_full[stage]), (i / S::STAGES) & 1, &s_abort, p.err, ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w_src = smem_base + stage * S::STAGE;
        const uint64_t w_desc = umma_desc_k_sw128(w_src), x_desc = umma_desc_k_sw128(w_src + S::W_BYTES);
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k)
          umma_bf16_ss(tmem_base, w_desc + 2 * k, x_desc + 2 * k, idesc, (i | k) != 0);
        umma_commit(smem_u32(&bar_empty[stage]));
      }
      if (ok) umma_commit(smem_u32(&bar_acc));
    }
  } else {
    // ------------------------------------------------------------ accumulator -> partial tile [row][feature]
    const int quad = warp & 3;
    pdl_wait();                       // as above; and the residual below is the predecessor's output, `out` may be its input
    if (mbar_wait(smem_u32(&bar_acc), 0, &s_abort, p.err, ERR_WAIT_TMEM_FULL)) {
      // every stage has been read by a finished MMA: the ring is free to hold the partial tile
      tc_fence_after();
      const uint32_t dst = smem_base + (quad * 32 + lane) * 4;
#pragma unroll 1
      for (int c = 0; c < NB && c < rows; c += 16) {
        uint32_t r[16];
        __syncwarp();
        tmem_ld_32x16(tmem_base + c + (static_cast<uint32_t>(quad * 32) << 16), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (c + j) * (SK_BM * 4)), "r"(r[j]) : "memory");
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (p.splits > 1) cluster_sync_all();
  if (warp < 2) pdl_wait();

  // ---------------------------------------------------------------- sum over the cluster, epilogue: 4 columns a thread
  const int cols = p.act == 3 ? SK_BM / 2 : SK_BM;           // output columns of the tile
  const int per_row = cols / 4;
  for (int u = rank * SK_THREADS + (int)threadIdx.x; u < rows * per_row; u += p.splits * SK_THREADS) {
    const int r = u / per_row, f = (u - r * per_row) * 4;
    const long long m = m0 + r;
    const int col = tile * cols + f;
    if (col >= p.N) continue;
    auto total = [&](int feature) {
      const uint32_t off = smem_base + (r * SK_BM + feature) * 4;
      float4 x[8];                      // every load in flight before the first addition
#pragma unroll
      for (int s = 0; s < 8; ++s)
        x[s] = s < p.splits ? ld_dsmem_f4(map_to_cta(off, s)) : make_float4(0.f, 0.f, 0.f, 0.f);
      float4 t = x[0];
#pragma unroll
      for (int s = 1; s < 8; ++s) { t.x += x[s].x; t.y += x[s].y; t.z += x[s].z; t.w += x[s].w; }
      return t;
    };
    const float4 t = total(f);
    float v[4] = {t.x, t.y, t.z, t.w};
    const bool whole = col + 4 <= p.N;
    if (p.act == 3) {
      const float4 up = total(SK_BM / 2 + f);
      const float w[4] = {up.x, up.y, up.z, up.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = v[j] / (1.f + __expf(-v[j])) * w[j];
    } else {
      if (p.bias) {
        if (whole) {
          const uint2 b = *reinterpret_cast<const uint2*>(p.bias + col);
          v[0] += bf16_lo(b.x); v[1] += bf16_hi(b.x); v[2] += bf16_lo(b.y); v[3] += bf16_hi(b.y);
        } else {
          for (int j = 0; j < 4; ++j) if (col + j < p.N) v[j] += __bfloat162float(p.bias[col + j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] *= p.out_scale;
        if (p.act == 1) v[j] = fmaxf(v[j], 0.f);
        else if (p.act == 2) v[j] = gelu_erf(v[j]);
      }
    }
    if (p.residual) {
      const __nv_bfloat16* rp = p.residual + m * p.ldr + col;
      if (whole) {
        const uint2 b = *reinterpret_cast<const uint2*>(rp);
        v[0] += bf16_lo(b.x); v[1] += bf16_hi(b.x); v[2] += bf16_lo(b.y); v[3] += bf16_hi(b.y);
      } else {
        for (int j = 0; j < 4; ++j) if (col + j < p.N) v[j] += __bfloat162float(rp[j]);
      }
    }
    if (p.out_fp32) {
      float* op = reinterpret_cast<float*>(p.out) + m * p.ldo + col;
      if (whole) {
        if (DZ_STORE_OK(op, 16)) *reinterpret_cast<float4*>(op) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        for (int j = 0; j < 4; ++j) if (col + j < p.N && DZ_STORE_OK(op + j, 4)) op[j] = v[j];
      }
    } else {
      __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(p.out) + m * p.ldo + col;
      if (whole) {
        if (DZ_STORE_OK(op, 8))
          *reinterpret_cast<uint2*>(op) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      } else {
        for (int j = 0; j < 4; ++j) if (col + j < p.N && DZ_STORE_OK(op + j, 2)) op[j] = __float2bfloat16(v[j]);
      }
    }
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync_all();      // nobody leaves while a peer may still read its partial tile
  if (warp == 1) {
    if (s_abort) {
      // error path: give copies and MMAs still in flight time to land before TMEM goes
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

static int sk_nb(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }

int skinny_map_w(CUtensorMap* map, const void* W, long long ldw, int rows, int K, bool swiglu) {
  return make_tmap_bf16_2d(map, W, rows, K, ldw, swiglu ? SK_BM / 2 : SK_BM, SK_BK, true);
}
int skinny_map_x(CUtensorMap* map, const void* A, long long lda, int M, int K) {
  return make_tmap_bf16_2d(map, A, M, K, lda, sk_nb(M), SK_BK, true);
}

// CTAs of a cluster that share a tile's K range: as many as keep the launch at 256 CTAs (of the 296 that fit, two per SM;
// larger clusters do not pack beyond that) with at least three 64-wide K blocks each.  Measured at one row, us: N 2048 K
// 8192 (16 tiles) 30.5 / 18.4 / 12.1 / 10.6 with 1 / 2 / 4 / 8 CTAs a tile; N 12288 K 4096 (96 tiles) 22.2 / 20.0 / 26.0
// with 1 / 2 / 3; N 6144 K 2048 (48 tiles) 8.7 / 13.1 with 4 / 6; N 20480 K 5120 (160 tiles) 36.5 / 43.5 with 1 / 2.
// A launch of a decoding step keeps to one CTA per SM, so that the next launch fits beside it and can fill its ring.
// (For 128-row tiles the caller chooses: split_pays in block_forward.cu.)
static int choose_splits(int tiles, int num_kb, bool in_step) {
  int s = (in_step ? sm_count() : 256) / (tiles > 0 ? tiles : 1);
  if (s > num_kb / 3) s = num_kb / 3;
  return s < 1 ? 1 : s > 8 ? 8 : s;
}

template <int NB>
static int launch_nb(const CUtensorMap& tmW, const CUtensorMap& tmX, const SkinnyArgs& a, int tiles, bool dependent,
                     cudaStream_t stream) {
  auto kern = skinny_gemm_kernel<NB>;
  static PerDeviceFlag configured;
  if (int rc = ensure_dyn_smem(configured, kern, SkinnySmem<NB>::TOTAL)) return rc;
  cudaError_t e = pdl_launch(kern, dim3((unsigned)(tiles * a.splits)), SK_THREADS, SkinnySmem<NB>::TOTAL, stream,
                             a.splits, dependent, tmW, tmX, a);
  return cuda_rc(e);
}

int skinny_launch(const CUtensorMap& tmW, const CUtensorMap& tmX, SkinnyArgs a, int splits, bool in_step, bool dependent,
                  cudaStream_t stream) {
  const int cols = a.act == 3 ? SK_BM / 2 : SK_BM;
  const int nb = sk_nb(a.M);
  a.num_n = (a.N + cols - 1) / cols;
  const long long tiles_ll = (long long)a.num_n * ((a.M + nb - 1) / nb);
  if (tiles_ll * 8 > 0x7fffffffLL) return DZ_ERR_TOO_LARGE;
  const int tiles = (int)tiles_ll;
  a.num_kb = (a.K + SK_BK - 1) / SK_BK;
  if (splits <= 0) splits = choose_splits(tiles, a.num_kb, in_step);
  if (splits > 8) splits = 8;
  a.kb_per_cta = (a.num_kb + splits - 1) / splits;
  a.splits = (a.num_kb + a.kb_per_cta - 1) / a.kb_per_cta;     // no CTA without a K block
  switch (nb) {
    case 16: return launch_nb<16>(tmW, tmX, a, tiles, dependent, stream);
    case 32: return launch_nb<32>(tmW, tmX, a, tiles, dependent, stream);
    case 64: return launch_nb<64>(tmW, tmX, a, tiles, dependent, stream);
    default: return launch_nb<128>(tmW, tmX, a, tiles, dependent, stream);
  }
}

}  // namespace dz

using namespace dz;
DZ_DEBUG_TU(skinny)

// Same contract as dz_gemm_bf16_tn (gemm_sm100.cu); act 3: W = gate rows | up rows (N each), out [M, N] =
// silu(A gate^T) * (A up^T), bf16, without bias, residual or scale.  splits: 0 = choose, else CTAs per tile (1 to 8).
extern "C" int dz_gemm_skinny(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo,
                              const void* bias, const void* residual, long long ldr, int M, int N, int K, int act,
                              int out_fp32, float out_scale, int splits, uint32_t* err, cudaStream_t stream) {
  if (!A || !W || !out || M <= 0 || N <= 0 || K <= 0 || act < 0 || act > 3 || splits < 0) return DZ_ERR_ARG;
  if ((K & 7) || (lda & 7) || (ldw & 7)) return DZ_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) return DZ_ERR_ALIGN;
  const int esz = out_fp32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(out) & 15) || ((ldo * esz) & 15)) return DZ_ERR_ALIGN;
  if (bias && (reinterpret_cast<uintptr_t>(bias) & 15)) return DZ_ERR_ALIGN;
  if (residual && ((reinterpret_cast<uintptr_t>(residual) & 15) || (ldr & 7))) return DZ_ERR_ALIGN;
  if (act == 3 && (bias || residual || out_fp32 || out_scale != 1.0f)) return DZ_ERR_ARG;
  if ((long long)N * 2 > 0x7fffffffLL) return DZ_ERR_TOO_LARGE;
  SkinnyArgs a{};
  a.M = M; a.N = N; a.K = K; a.out = out; a.ldo = ldo;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  a.ldr = ldr; a.act = act; a.out_fp32 = out_fp32; a.out_scale = out_scale; a.err = err;
  CUtensorMap tmW, tmX;
  int rc = skinny_map_w(&tmW, W, ldw, act == 3 ? 2 * N : N, K, act == 3);
  if (rc) return rc;
  rc = skinny_map_x(&tmX, A, lda, M, K);
  if (rc) return rc;
  return skinny_launch(tmW, tmX, a, splits, false, true, stream);
}
