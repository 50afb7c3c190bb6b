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
__device__ __forceinline__ uint32_t warp_umin(uint32_t v) { return __reduce_min_sync(0xffffffffu, v); }

// Tails are kept times 2^11, as large as their heads, so that they are normal numbers as long as those are.  Products of a head and a tail
// then are too, and are summed first; the accumulator is brought down by 2^11 with the first product of two heads (see umma_pair_onto).
constexpr int kTailBits = 11;
constexpr float kTailUp = 1 << kTailBits;

// Elements far below their row's largest.  A head is a normal number down to 2^-14, 2^-28 of the largest; what is smaller goes into planes
// of its own, times 2^28 once more (level 1), or twice (level 2, which holds what is left as far as it can: all but 2^-107 of
// the largest), and is zero in the others.  A row's marks say which of these planes it has: bit 0 level 1, bit 1 level 2 as well.  The matmul
// then goes over K again for the tiles that hold such a row.
constexpr int kLevels = 3, kLevelBits = 28;
constexpr float kLevelUp = 1 << kLevelBits, kLevelFloor = 1.0f / (1 << 14);

// `least`: the bits of the smallest magnitude that is not zero, less one (zero: all ones).
__device__ __forceinline__ uint32_t row_marks(uint32_t most, uint32_t least) {
  const uint32_t e = most >> 23, top = e < 15u ? 15u : e, low = least >> 23;
  if (most >= 0x7F800000u || low + kLevelBits >= top) return 0;
  return low + 2 * kLevelBits >= top ? 1u : 3u;
}

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

// The planes of heads and of tails of every level that the row has, `plane` apart.
inline __device__ __noinline__ void store_apart(__half* heads, int64_t plane, float4 x, float scale, uint32_t marks) {
  float v[4] = {x.x * scale, x.y * scale, x.z * scale, x.w * scale};
#pragma unroll 1
  for (int level = 0; level < kLevels; ++level) {
    const bool more = (marks >> level & 1u) != 0;
    float here[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool taken = !more || fabsf(v[e]) >= kLevelFloor;
      here[e] = taken ? v[e] : 0.0f;
      v[e] = taken ? 0.0f : v[e] * kLevelUp;
    }
    store_terms(heads + 2 * level * plane, heads + (2 * level + 1) * plane, make_float4(here[0], here[1], here[2], here[3]), 1.0f);
    if (!more) break;
  }
}
__device__ __forceinline__ void store_levels(__half* heads, int64_t plane, const float4& x, float scale, uint32_t marks) {
  if (marks == 0) store_terms(heads, heads + plane, x, scale);
  else store_apart(heads, plane, x, scale, marks);
}

}  // namespace kb200
