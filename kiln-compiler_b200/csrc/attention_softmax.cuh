// Maxima and probabilities of 32 scores, for the kernels whose rows are shared by two threads (attention.cu, attention_pairs.cuh).
#pragma once

#include <math_constants.h>

#include "attention.h"
#include "tc_common.cuh"

namespace kb200 {

namespace {

using namespace tc;

// Scores of one 32-column block -> probabilities, in place; returns their sum.  `first_col` is the
// block's first key relative to the query tile's first row (only used on the diagonal tile).
template <bool DIAGONAL>
__device__ __forceinline__ float probabilities32(float (&v)[32], float scale_log2, float m_use, int first_col, int row) {
  const float2 scale2 = make_float2(scale_log2, scale_log2), shift2 = make_float2(-m_use, -m_use);
  float2 sum2 = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    const float2 t = ffma2(make_float2(v[i], v[i + 1]), scale2, shift2);     // two exponents per instruction
    float2 pr = make_float2(ex2(t.x), ex2(t.y));
    if (DIAGONAL && first_col + i > row) pr.x = 0.0f;
    if (DIAGONAL && first_col + i + 1 > row) pr.y = 0.0f;
    v[i] = pr.x;
    v[i + 1] = pr.y;
    sum2 = fadd2(sum2, pr);
  }
  return sum2.x + sum2.y;
}
template <bool DIAGONAL>
__device__ __forceinline__ float row_max32(const float (&v)[32], float m, int first_col, int row) {
  if (DIAGONAL) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (first_col + i <= row) m = fmaxf(m, v[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; i += 2) m = fmax3(m, v[i], v[i + 1]);
  }
  return m;
}

}  // namespace

}  // namespace kb200
