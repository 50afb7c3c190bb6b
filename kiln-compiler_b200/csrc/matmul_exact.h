// Exact FP32 as products of float16 pairs on SM pairs (matmul_exact.cu), as matmul_tc.cu sees it, and the splitting of operands into such
// pairs (split_rows.cu).
#pragma once

#include "kb200_internal.h"

namespace kb200 {

struct ExactOperands {
  const void* a;             // [kLevels][2, M, pitch] float16, the plane of heads and that of tails of every level (see split16.cuh)
  const void* b;             // [2, N, pitch], rows along K
  int64_t pitch;
  const float* a_scale;      // [M] and [N]: what products of the terms are to be multiplied by
  const float* b_scale;
  const uint8_t* a_marks;    // [M rounded up to whole tiles]: the levels of A's rows
};

// Estimated cycles of a launch, or -1 when the kernel does not cover this matmul.
int64_t exact_cycles(const Plan& plan, const PlanKernel& k);
// Does this build of its kernel have the registers that its warps share out?  (With fewer those that ask for more would wait for ever.)
int exact_runs(const Plan& plan, const PlanKernel& k, bool* runs);
// *state stays null when the operands cannot be described; a non-zero return is an error.
int exact_bind(Plan& plan, PlanKernel& k, int kernel_index, const ExactOperands& ops, void** state);
int exact_launch(const Plan& plan, const void* state, cudaStream_t s);
bool exact_repoint(const PlanKernel& k, void* state);      // the operand pointers of `k` have moved
std::string exact_detail(const void* state);
bool exact_writes_tails(const void* state);
// Float16 pairs of the output into `to` as well, times `scale` by 32 columns, or only those.  False: not this launch.
bool exact_write_pairs(const PlanKernel& k, void* state, const PlanKernel::Planes& to, const float* scale, bool store32);
void exact_destroy(void* state);

// float32 rows of `cols` elements -> the two planes and the scales; with `marks` of every level.  A pass in front of a launch, or once for a weight.
int split_rows(const float* src, int64_t s_row, void* planes, int64_t pitch, float* scale, uint8_t* marks, int64_t rows, int64_t cols, bool pdl, cudaStream_t s);
// |LayerNorm(x) B + bias| per column of B [K, N] for any x, at most: of the normalised row, 1 / sqrt(inv_n) long, by Cauchy and Schwarz.  `bounds`: [n]
// on the host.  `near`: no column's result for a row of nearly equal elements (whose LayerNorm is next to beta) is below 2^-30 of its bound; else,
// without any biases as a rule, float16 pairs under the bound's power of two do not hold the results of rows of next to nothing.  Synchronises.
int layernorm_bounds(const float* b, int64_t b_k, int64_t b_n, int64_t k, int64_t n, const float* gamma, const float* beta, const float* bias, float inv_n, std::vector<float>* bounds, bool* near);
// Do float16 pairs hold this weight [K, N] as well as TF32 pairs would?  `scratch`: k + 1 words on the device.  Synchronises.
int split_suits(const float* b, int64_t b_k, int64_t b_n, int64_t k, int64_t n, uint32_t* scratch, bool* suits);

}  // namespace kb200
