// Host interface of the decode attention (decode_kernels.cu) inside the library.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dz {

// Keys of one (sequence, head), prefix rows among them.  The kernel itself keeps no scores; the bound on the length of a
// sequence is what the entry points refuse.
constexpr int DA_MAX_KEYS = 40 * 1024;

struct DecodeAttnArgs {
  const __nv_bfloat16* q;              // [B, ldq], head h at column h * hd
  long long ldq;
  const __nv_bfloat16 *k_new, *v_new;  // append mode: the new token's rows (row pitch ldq, H / rep heads), else null
  int rep;                             // query heads per key / value head of k_new, v_new
  const float2* rope;                  // append mode, optional: (cos, sin) [position][hd / 2]
  int rope_pos;
  __nv_bfloat16 *kc, *vc;              // cache [B][row][H * hd]; append mode writes row kv_len - 1
  long long ld_seq, ld_row;
  const __nv_bfloat16 *pk, *pv;        // prefix rows [n_prefix, ldp] or null
  long long ldp;
  int n_prefix;
  const int* pad_left;                 // [B] or null
  int kv_len, hd, splits;              // kv_len counts the new token
  float scale;
  __nv_bfloat16* out;                  // [B, ldo]
  long long ldo;
};

int decode_attn_launch(DecodeAttnArgs a, int B, int H, bool dependent, cudaStream_t stream);

}  // namespace dz
