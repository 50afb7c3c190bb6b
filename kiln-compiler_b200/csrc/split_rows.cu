// Float32 operands of an exact matmul as two float16 terms: x 2^e = h + 2^-11 t, h the nearest float16 and t the nearest to what is left times
// 2^11, with one power of two per row that puts the row's largest element at 2^14 to 2^15.  Role of the operand precision of the reference's
// `tl.dot(..., input_precision="ieee")` (kiln/gpu/codegen.py:515).
//
// How much of x they hold: all but 2^-22 |x| (2^-24 in the mean) as long as h is a normal number, down to 2^-28 of the row's largest element; what is
// less comes under further powers of two, in planes of its own (levels, split16.cuh), as precisely down to 2^-84 of the largest.  Two TF32 terms,
// which have float32's exponents, hold all but 2^-22 to 2^-24 of every x.  (Under one power of two 2^-51 of the largest was what remained, with
// tails as they are 2^-40: of results that use none of the features 2^24 times the others, 1.8e-5 in that form.)  A weight has one level: those with
// elements below 2^-28 of their column's largest keep the kernels on TF32, and so do those whose rows' largest elements, max over n of
// |b[k, n]|, are more than 2^10 apart (`split_suits`).
//
// What bounds the pass: it is a launch of ~2.3 us in front of a matmul; 4 bytes read and 4 written per element.
#include <math.h>

#include "kb200_internal.h"
#include "matmul_exact.h"
#include "split16.cuh"

namespace kb200 {

namespace {

// One row per warp (WIDE: per block), N float4 a lane in registers; N = 0: rows of any width, read twice.
template <int N, bool WIDE>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ src, int64_t s_row, __half* __restrict__ heads,
                                                         int64_t plane, int64_t pitch, float* __restrict__ scales, uint8_t* __restrict__ marks, uint32_t rows, int units) {
  __shared__ uint32_t partial[2][8];
  const int lane = WIDE ? threadIdx.x : threadIdx.x & 31, lanes = WIDE ? 256 : 32;
  const uint32_t row = WIDE ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  if (row >= rows) return;
  const float4* const x = reinterpret_cast<const float4*>(src + (int64_t)row * s_row);
  float4 v[N > 0 ? N : 1];
  uint32_t most = 0, least = ~0u;
  auto look = [&](const float4& t) {
    const uint32_t a = magnitude_bits(t.x), b = magnitude_bits(t.y), c = magnitude_bits(t.z), d = magnitude_bits(t.w);
    most = max(max(most, max(a, b)), max(c, d));
    least = min(min(least, min(a - 1u, b - 1u)), min(c - 1u, d - 1u));
  };
  if constexpr (N > 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int j = lane + lanes * i;
      v[i] = j < units ? x[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) look(v[i]);
  } else {
    for (int j = lane; j < units; j += lanes) look(x[j]);
  }
  most = warp_umax(most);
  least = warp_umin(least);
  if constexpr (WIDE) {
    if ((threadIdx.x & 31) == 0) {
      partial[0][threadIdx.x >> 5] = most;
      partial[1][threadIdx.x >> 5] = least;
    }
    __syncthreads();
    most = warp_umax(partial[0][threadIdx.x & 7]);
    least = warp_umin(partial[1][threadIdx.x & 7]);
  }
  const RowScale scale(most);
  const uint32_t levels = marks != nullptr ? row_marks(most, least) : 0u;
  if (lane == 0) {
    scales[row] = scale.back;
    if (marks != nullptr) marks[row] = (uint8_t)levels;
  }
  __half* const h = heads + (int64_t)row * pitch;
  if constexpr (N > 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int j = lane + lanes * i;
      if (j < units) store_levels(h + 4 * j, plane, v[i], scale.by, levels);
    }
  } else {
    for (int j = lane; j < units; j += lanes) store_levels(h + 4 * j, plane, x[j], scale.by, levels);
  }
}

// The largest magnitude of a weight's elements at each k.
__global__ void __launch_bounds__(256) largest_kernel(const float* __restrict__ b, int64_t b_k, int64_t b_n, int n, uint32_t* __restrict__ out) {
  __shared__ uint32_t partial[8];
  const float* const row = b + blockIdx.x * b_k;
  uint32_t most = 0;
  for (int i = threadIdx.x; i < n; i += 256) most = max(most, __float_as_uint(row[i * b_n]) & 0x7FFFFFFFu);
  most = warp_umax(most);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = most;
  __syncthreads();
  most = warp_umax(partial[threadIdx.x & 7]);
  if (threadIdx.x == 0) out[blockIdx.x] = most;
}

// How many elements of a weight float16 pairs do not hold: not zero, and below 2^-28 of their column's largest.  One block per column.
__global__ void __launch_bounds__(256) low_kernel(const float* __restrict__ b, int64_t b_k, int64_t b_n, int k, uint32_t* __restrict__ count) {
  __shared__ uint32_t partial[8];
  const float* const column = b + blockIdx.x * b_n;
  uint32_t most = 0, low = 0;
  for (int i = threadIdx.x; i < k; i += 256) most = max(most, magnitude_bits(column[i * b_k]));
  most = warp_umax(most);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = most;
  __syncthreads();
  most = warp_umax(partial[threadIdx.x & 7]);
  for (int i = threadIdx.x; i < k; i += 256) low += row_marks(most, magnitude_bits(column[i * b_k]) - 1u) != 0 ? 1u : 0u;
  low = __reduce_add_sync(0xffffffffu, low);
  if ((threadIdx.x & 31) == 0 && low != 0) atomicAdd(count, low);
}

// One block per column of a weight: see layernorm_bounds.
__global__ void __launch_bounds__(256) bound_kernel(const float* __restrict__ b, int64_t b_k, int64_t b_n, int k, const float* __restrict__ gamma,
                                                    const float* __restrict__ beta, const float* __restrict__ bias, float length, float* __restrict__ out) {
  __shared__ float partial[3][8];
  const float* const column = b + blockIdx.x * b_n;
  float squares = 0.0f, shifts = 0.0f, rest = 0.0f;
  for (int i = threadIdx.x; i < k; i += 256) {
    const float w = column[i * b_k], g = gamma[i] * w;
    squares += g * g;
    shifts += fabsf(beta[i] * w);
    rest += beta[i] * w;
  }
  for (int o = 16; o > 0; o >>= 1) {
    squares += __shfl_xor_sync(0xffffffffu, squares, o);
    shifts += __shfl_xor_sync(0xffffffffu, shifts, o);
    rest += __shfl_xor_sync(0xffffffffu, rest, o);
  }
  if ((threadIdx.x & 31) == 0) {
    partial[0][threadIdx.x >> 5] = squares;
    partial[1][threadIdx.x >> 5] = shifts;
    partial[2][threadIdx.x >> 5] = rest;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      squares += partial[0][w];
      shifts += partial[1][w];
      rest += partial[2][w];
    }
    const float add = bias != nullptr ? bias[blockIdx.x] : 0.0f;
    out[blockIdx.x] = 1.01f * (length * sqrtf(squares) + shifts + fabsf(add));      // (1 %: float32 sums)
    out[gridDim.x + blockIdx.x] = fabsf(rest + add);
  }
}

}  // namespace

int layernorm_bounds(const float* b, int64_t b_k, int64_t b_n, int64_t k, int64_t n, const float* gamma, const float* beta, const float* bias, float inv_n, std::vector<float>* bounds, bool* near) {
  std::vector<float> both((size_t)n * 2);
  float* device = nullptr;
  KB200_CUDA(cudaMalloc(&device, both.size() * sizeof(float)));
  cudaError_t e = launch_kernel(false, bound_kernel, dim3((unsigned)n), dim3(256), 0, nullptr, b, b_k, b_n, (int)k, gamma, beta, bias, sqrtf(1.0f / inv_n), device);
  if (e == cudaSuccess) e = cudaMemcpy(both.data(), device, both.size() * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(device);
  if (e != cudaSuccess) return cuda_fail(e, "the bounds of a matmul's results");
  bounds->assign(both.begin(), both.begin() + n);
  *near = true;
  for (int64_t i = 0; i < n && *near; ++i) *near = both[i] == 0.0f || both[n + i] >= both[i] * 0x1p-30f;
  return KB200_OK;
}

int split_rows(const float* src, int64_t s_row, void* planes, int64_t pitch, float* scale, uint8_t* marks, int64_t rows, int64_t cols, bool pdl, cudaStream_t s) {
  __half* const heads = static_cast<__half*>(planes);
  const int64_t plane = rows * pitch;
  const int units = (int)(cols / 4), n = (units + 31) / 32;
  // a warp per row; rows of more than 1024 a block per row
  const int warps = rows >= 148 * 16 ? 8 : rows >= 148 * 4 ? 4 : 1;
  const dim3 grid((unsigned)((rows + warps - 1) / warps)), block(32 * warps), wide((unsigned)rows);
#define KB200_SPLIT(N, WIDE) launch_kernel(pdl, split_rows_kernel<N, WIDE>, WIDE ? wide : grid, WIDE ? dim3(256) : block, 0, s, src, s_row, heads, plane, pitch, scale, marks, (uint32_t)rows, units)
  if (n <= 2) KB200_CUDA(KB200_SPLIT(2, false));
  else if (n <= 4) KB200_CUDA(KB200_SPLIT(4, false));
  else if (n <= 6) KB200_CUDA(KB200_SPLIT(6, false));
  else if (n <= 8) KB200_CUDA(KB200_SPLIT(8, false));
  else if (n <= 16) KB200_CUDA(KB200_SPLIT(2, true));
  else if (n <= 32) KB200_CUDA(KB200_SPLIT(4, true));
  else KB200_CUDA(KB200_SPLIT(0, true));
#undef KB200_SPLIT
  return KB200_OK;
}

int split_suits(const float* b, int64_t b_k, int64_t b_n, int64_t k, int64_t n, uint32_t* device, bool* suits) {
  *suits = false;
  std::vector<uint32_t> most((size_t)k + 1);
  cudaError_t e = cudaMemsetAsync(device + k, 0, sizeof(uint32_t), nullptr);
  if (e == cudaSuccess) e = launch_kernel(false, largest_kernel, dim3((unsigned)k), dim3(256), 0, nullptr, b, b_k, b_n, (int)n, device);
  if (e == cudaSuccess) e = launch_kernel(false, low_kernel, dim3((unsigned)n), dim3(256), 0, nullptr, b, b_k, b_n, (int)k, device + k);
  if (e == cudaSuccess) e = cudaMemcpy(most.data(), device, most.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "the largest elements of a weight");
  // (Of normally distributed elements one in 2^26 is as small by chance, and is held to 2^-18 or better.)
  const bool held = most[(size_t)k] <= 1 + (uint64_t)k * n / (1 << 24);
  most.pop_back();
  uint32_t lo = 255, hi = 0;
  for (uint32_t m : most) {
    const uint32_t e2 = m >> 23;
    lo = e2 < lo ? e2 : lo;
    hi = e2 > hi ? e2 : hi;
  }
  // (2^-60 to 2^60: the epilogue multiplies by the columns' scales before the rows')
  *suits = held && hi - lo <= 10 && lo >= 127 - 60 && hi <= 127 + 60;
  return KB200_OK;
}

}  // namespace kb200
