// The tensor-core matmul for problems of few tiles (matmul_small.cu), as matmul_tc.cu sees it.
#pragma once

#include "kb200_internal.h"
#include "matmul_pair.h"

namespace kb200 {

// How the kernel takes A: through a tensor map of ops.a_base (a mirror or a copy, or A itself), through one of the float32 A
// for bf16 products, or through four, float32 at any pitch.
enum SmallA : int { SMALL_A_MAPPED, SMALL_A_FLOAT32, SMALL_A_GATHERED };

// Estimated cycles of a launch, or -1 when the kernel does not cover this matmul.
// `close`: exact FP32 as near to float64 as float32 sums on the CUDA cores.
int64_t small_cycles(const Plan& plan, const PlanKernel& k, bool b_kmajor, int64_t b_cols, SmallA form, bool close);
// Exact FP32: MMAs along K that go into one accumulator, where the kernel covers this matmul.
int small_sum_length(const Plan& plan, const PlanKernel& k);
// Tensor maps and launch parameters.  `b_tail`: exact FP32, the tails of B in the layout of ops.b_base.
// *state stays null when the operands cannot be described; a non-zero return is an error.
int small_bind(Plan& plan, PlanKernel& k, int kernel_index, const PairOperands& ops, const float* b_tail, SmallA form, bool close,
               void** state);
int small_launch(const Plan& plan, const void* state, cudaStream_t s);
bool small_repoint(const PlanKernel& k, void* state);     // the operand pointers of `k` have moved
std::string small_detail(const void* state);
bool small_writes_tails(const void* state);
void small_destroy(void* state);

}  // namespace kb200
