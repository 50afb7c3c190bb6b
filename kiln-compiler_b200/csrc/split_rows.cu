// Float32 operands of an exact matmul as two float16 terms: x 2^e = h + 2^-11 t, h the nearest float16 and t the nearest to what is left times
// 2^11, with one power of two per row that puts the row's largest element at 2^14 to 2^15.  Role of the operand precision of the reference's
// `tl.dot(..., input_precision="ieee")` (kiln/gpu/codegen.py:515).
//
// How much of x they hold: all but 2^-22 |x| (2^-24 in the mean) as long as h is a normal number, down to 2^-28 of the row's largest element, and
// 2^-36 2^-e = 2^-51 to 2^-50 of that where x is less.  (With tails as they are, t is subnormal from 2^-15 of the largest element on and held 2^-40 of
// it: of results that use none of the features 2^24 times the others, 1.8e-5.)  Two TF32 terms, which have float32's exponents, hold all but
// 2^-22 to 2^-24 of every x; weights whose columns' largest elements along K, max over n of |b[k, n]|, are more than 2^10 apart keep
// the kernels that multiply those (`split_suits`).
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
                                                         int64_t plane, int64_t pitch, float* __restrict__ scales, uint32_t rows, int units) {
  __shared__ uint32_t partial[8];
  const int lane = WIDE ? threadIdx.x : threadIdx.x & 31, lanes = WIDE ? 256 : 32;
  const uint32_t row = WIDE ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  if (row >= rows) return;
  const float4* const x = reinterpret_cast<const float4*>(src + (int64_t)row * s_row);
  float4 v[N > 0 ? N : 1];
  uint32_t most = 0;
  auto look = [&](const float4& t) {
    const uint32_t a = __float_as_uint(t.x) & 0x7FFFFFFFu, b = __float_as_uint(t.y) & 0x7FFFFFFFu, c = __float_as_uint(t.z) & 0x7FFFFFFFu,
                   d = __float_as_uint(t.w) & 0x7FFFFFFFu;
    most = max(max(most, max(a, b)), max(c, d));
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
  if constexpr (WIDE) {
    if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = most;
    __syncthreads();
    most = warp_umax(partial[threadIdx.x & 7]);
  }
  const RowScale scale(most);
  if (lane == 0) scales[row] = scale.back;
  __half* const h = heads + (int64_t)row * pitch;
  if constexpr (N > 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int j = lane + lanes * i;
      if (j < units) store_terms(h + 4 * j, h + plane + 4 * j, v[i], scale.by);
    }
  } else {
    for (int j = lane; j < units; j += lanes) store_terms(h + 4 * j, h + plane + 4 * j, x[j], scale.by);
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

// One block per column of a weight: see layernorm_bounds.
__global__ void __launch_bounds__(256) bound_kernel(const float* __restrict__ b, int64_t b_k, int64_t b_n, int k, const float* __restrict__ gamma,
                                                    const float* __restrict__ beta, const float* __restrict__ bias, float length, float* __restrict__ out) {
  __shared__ float partial[2][8];
  const float* const column = b + blockIdx.x * b_n;
  float squares = 0.0f, shifts = 0.0f;
  for (int i = threadIdx.x; i < k; i += 256) {
    const float w = column[i * b_k], g = gamma[i] * w;
    squares += g * g;
    shifts += fabsf(beta[i] * w);
  }
  for (int o = 16; o > 0; o >>= 1) {
    squares += __shfl_xor_sync(0xffffffffu, squares, o);
    shifts += __shfl_xor_sync(0xffffffffu, shifts, o);
  }
  if ((threadIdx.x & 31) == 0) {
    partial[0][threadIdx.x >> 5] = squares;
    partial[1][threadIdx.x >> 5] = shifts;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      squares += partial[0][w];
      shifts += partial[1][w];
    }
    out[blockIdx.x] = 1.01f * (length * sqrtf(squares) + shifts + (bias != nullptr ? fabsf(bias[blockIdx.x]) : 0.0f));      // (1 %: float32 sums)
  }
}

}  // namespace

int layernorm_bounds(const float* b, int64_t b_k, int64_t b_n, int64_t k, int64_t n, const float* gamma, const float* beta, const float* bias, float inv_n, std::vector<float>* bounds) {
  bounds->assign((size_t)n, INFINITY);
  float* device = nullptr;
  KB200_CUDA(cudaMalloc(&device, (size_t)n * sizeof(float)));
  cudaError_t e = launch_kernel(false, bound_kernel, dim3((unsigned)n), dim3(256), 0, nullptr, b, b_k, b_n, (int)k, gamma, beta, bias, sqrtf(1.0f / inv_n), device);
  if (e == cudaSuccess) e = cudaMemcpy(bounds->data(), device, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(device);
  return e == cudaSuccess ? KB200_OK : cuda_fail(e, "the bounds of a matmul's results");
}

int split_rows(const float* src, int64_t s_row, void* planes, int64_t pitch, float* scale, int64_t rows, int64_t cols, bool pdl, cudaStream_t s) {
  __half* const heads = static_cast<__half*>(planes);
  const int64_t plane = rows * pitch;
  const int units = (int)(cols / 4), n = (units + 31) / 32;
  // a warp per row; rows of more than 1024 a block per row
  const int warps = rows >= 148 * 16 ? 8 : rows >= 148 * 4 ? 4 : 1;
  const dim3 grid((unsigned)((rows + warps - 1) / warps)), block(32 * warps), wide((unsigned)rows);
#define KB200_SPLIT(N, WIDE) launch_kernel(pdl, split_rows_kernel<N, WIDE>, WIDE ? wide : grid, WIDE ? dim3(256) : block, 0, s, src, s_row, heads, plane, pitch, scale, (uint32_t)rows, units)
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
  std::vector<uint32_t> most((size_t)k);
  cudaError_t e = launch_kernel(false, largest_kernel, dim3((unsigned)k), dim3(256), 0, nullptr, b, b_k, b_n, (int)n, device);
  if (e == cudaSuccess) e = cudaMemcpy(most.data(), device, (size_t)k * sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "the largest elements of a weight");
  uint32_t lo = 255, hi = 0;
  for (uint32_t m : most) {
    const uint32_t e2 = m >> 23;
    lo = e2 < lo ? e2 : lo;
    hi = e2 > hi ? e2 : hi;
  }
  // (2^-60 to 2^60: the epilogue multiplies by the columns' scales before the rows')
  *suits = hi - lo <= 10 && lo >= 127 - 60 && hi <= 127 + 60;
  return KB200_OK;
}

}  // namespace kb200
