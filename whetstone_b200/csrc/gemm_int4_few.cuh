/* Launch interface of the int4-hier projection for a handful of tokens (gemm_int4_few.cu). */
#pragma once

#include "wst_common.cuh"

namespace wst {

constexpr int kInt4FewTokens = 32; /* the most tokens it takes */

/* Buffers aligned as wst_gemm_int4_hier checks; n <= kInt4FewTokens. */
wst_status_t launch_gemm_int4_few(const void *qw, const void *si, const void *sb, const void *x,
                                  const void *bias, void *y, int in_f, int out_f, int n, int accum,
                                  int sm_count);

}  // namespace wst
