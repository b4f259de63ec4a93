/* Projections of more than 128 tokens, and the fused qkv projection of any number: what the
 * entry points in gemm_f16.cu hand to gemm_pair.cu. */
#pragma once

#include <cuda_fp16.h>

#include "wst_common.cuh"

namespace wst {

struct PairGemm {
  const char *name = "wst_gemm_fp16";
  const void *w = nullptr; /* [out_f][in_f] fp16, or null: the packed form below */
  /* hierarchical int4: one 16-byte word of 32 nibbles and one byte of two 4-bit scale
   * indices per group of 32 along K, one (d, dmin) pair per row */
  const uint4 *qw = nullptr;     /* [out_f][in_f / 32] */
  const uint8_t *si = nullptr;   /* [out_f][in_f / 32]: ls | lm << 4 */
  const __half2 *sb = nullptr;   /* [out_f]: (d, dmin) */
  const void *x = nullptr;       /* [n][in_f] fp16 */
  const __half *bias = nullptr;  /* [out_f] or null */
  int in_f = 0, out_f = 0, n = 0;
  /* plain form */
  float *y = nullptr; /* [n][out_f] */
  int accum = 0;
  /* fused form (q_out set): the columns are the heads of the qkv row; they are normed,
   * rotated and stored where the attention reads them instead of going to y */
  __half *q_out = nullptr;           /* [n][n_q * hd] */
  __half *k_cache = nullptr;         /* [n_seq][n_kv][max_seq][hd] */
  __half *v_cache = nullptr;
  const float *cos_tab = nullptr;    /* [table_len][hd / 2] */
  const float *sin_tab = nullptr;
  const __half *q_gain = nullptr;    /* [hd] or null */
  const __half *k_gain = nullptr;
  const int32_t *seq_pos0 = nullptr; /* [n_seq] */
  int n_q = 0, n_kv = 0, hd = 0, n_per_seq = 0, max_seq = 0, table_len = 0;
  float eps = 0.f;
};

wst_status_t launch_gemm_pair(const PairGemm &g, int sm_count);

/* The plain form with int4 weights for up to 128 tokens (gemm_narrow.cu). */
wst_status_t launch_gemm_narrow(const PairGemm &g);

}  // namespace wst
