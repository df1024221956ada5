// Interface of the f32 product on the tensor cores (gemm_f32_split.cu).
#pragma once
#include "gemm_plan.h"
#include "ugb_internal.h"

// c[j, i] = sum_k p[i, k] q[j, k], f32: p holds what is a column of c, q what is a row.  Both have a unit stride along their rows or
// along k.
struct ugb_f32_split_args {
  float *c;
  const float *p, *q;
  size_t batch, rows_p, rows_q, k;
  long long p_rs, p_ks, p_batch, q_rs, q_ks, q_batch;   // elements between rows, along k, between batch steps
  long long c_q, c_batch;                               // elements between rows of c, between batch steps
  bool pdl;
};

// On tiles of 128 x bn (32, 64 or 96; 64 where q's rows are contiguous), k split over clusters of `split` CTAs (up to 8).
// UGB_ERR_UNSUPPORTED (last_error untouched) for what it does not take.
int32_t ugb_f32_split(ugb_device *dev, const ugb_f32_split_args &a, int bn, int split);
