// A float32 row as two float16 terms under a power of two: see split_rows.cu.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace kb200 {

__device__ __forceinline__ uint32_t magnitude_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// The scale of a row whose largest magnitude has these bits, and what its products are multiplied by.  (Rows below 2^-112 are not brought up
// all the way: `back` stays a normal number.)  A row with a NaN makes NaN of all its results, as float32 does.  One with
// infinities and no NaN is marked: NaN terms, and a `back` below zero that asks the matmul for sums of the operands themselves.
struct RowScale {
  float by, back;
  bool marked;
  __device__ __forceinline__ explicit RowScale(uint32_t largest) {
    const bool finite = largest < 0x7F800000u;
    const uint32_t e = largest >> 23, field = finite ? 268u - (e < 15u ? 15u : e) : 127u;
    marked = largest == 0x7F800000u;
    by = __uint_as_float(finite ? field << 23 : 0x7FFFFFFFu);
    back = __uint_as_float((254u - field) << 23 | (marked ? 0x80000000u : 0u));
  }
};

__device__ __forceinline__ uint32_t warp_umax(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }

// Tails are kept times 2^11, as large as their heads, so that they are normal numbers as long as those are.  Products of a head and a tail
// then are too, and are summed first; the accumulator is brought down by 2^11 with the first product of two heads (see umma_pair_onto).
constexpr int kTailBits = 11;
constexpr float kTailUp = 1 << kTailBits;

__device__ __forceinline__ void store_terms(__half* heads, __half* tails, const float4& x, float scale) {
  const float v[4] = {x.x * scale, x.y * scale, x.z * scale, x.w * scale};
  __half h[4], t[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    h[e] = __float2half_rn(v[e]);
    t[e] = __float2half_rn((v[e] - __half2float(h[e])) * kTailUp);
  }
  *reinterpret_cast<uint2*>(heads) = *reinterpret_cast<const uint2*>(h);
  *reinterpret_cast<uint2*>(tails) = *reinterpret_cast<const uint2*>(t);
}

}  // namespace kb200
