// What the fused attention kernels share: the launch parameters of the tensor-core kernels and the entry points of
// the one for bf16 operands (attention_bf16.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace kb200 {

constexpr int kAttnRows = 128;               // queries per CTA and keys per tile
constexpr int kAttnHeadDim = 64;

struct AttnParams {
  int T, H, q_tiles;
  int B;                     // sequences in the graph (1 for the two-dimensional block); rows of Q, K, V and of the output are b * T + t
  float scale_log2;          // softmax scale times log2(e): exponentials are taken in base 2
  float* out;                // [T, H * 64] merged heads
  int64_t out_row_stride;
  bool out32;                // bf16 kernel: are the float32 rows written (someone reads them)?
  __nv_bfloat16* out16;      // optional bf16 copy of the merged heads, row stride H * 64, or null
  int64_t out16_row_stride;
  uint32_t idesc_qk, idesc_pv;
  int kernel_index;
  int* status;
  int split_from;            // query tiles from this one on are shared by two CTAs (q_tiles: none)
  float* partial;            // [split tile][2 halves][128 x 64 unnormalised output | 128 maxima | 128 sums]
  int* arrivals;             // [split tile][4 lane quadrants], zero between launches
  float* kept;               // bf16 kernel, items of more than kAttnRun key tiles: [CTA][a partial like those above], or null
  const unsigned short* order;   // with split tiles: (query tile << 1 | half) of the q_tiles + split tiles entries, heaviest first
};
constexpr int kAttnPartialFloats = kAttnRows * kAttnHeadDim + 2 * kAttnRows;
constexpr int kAttnRun = 16;                 // bf16 kernel: key tiles whose output adds up in tensor memory (see attention_bf16.cu)

#ifdef __CUDACC__
// A work item: one query tile of one head of one sequence, or (split tiles) one half of its key tiles.
struct AttnItem { int h, seq, q0, n_kv, qt, j0, half, slot; bool split; };

// This CTA's r-th item (-1: none).  Items are ordered heaviest first; rounds alternate direction over the CTAs, so that
// the CTA with the heaviest item of one round takes the lightest of the next (8 x 12 x 8 items: 24 key tiles at most per CTA instead of
// 27 on 148 CTAs, 13 instead of 15 on 296).
__device__ __forceinline__ int attn_nth_item(int r, int n_items) {
  const int w = r * (int)gridDim.x + ((r & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  return w < n_items ? w : -1;
}

// work item w -> (head, sequence, query tile): heaviest (longest causal prefix) tiles first, of every sequence.
// Query tiles from p.split_from on (the longest causal prefixes; none when split_from = q_tiles) are
// TWO items, one per half of their key tiles: each leaves its unnormalised rows and softmax state in
// a workspace, and the one that arrives second (a counter per tile and lane quadrant) merges them.
template <bool SPLIT>
__device__ __forceinline__ AttnItem attn_item(const AttnParams& p, int w) {
  AttnItem it;
  it.h = w % p.H;
  it.seq = (w / p.H) % p.B;
  const int v = w / (p.H * p.B);
  if (!SPLIT) {                                      // heaviest (longest causal prefix) first
    it.qt = p.q_tiles - 1 - v;
    it.half = 0;
  } else {                                           // whole tiles and halves in descending order of their key tiles (host table)
    const unsigned e = __ldg(p.order + v);
    it.qt = (int)(e >> 1);
    it.half = (int)(e & 1);
  }
  it.split = SPLIT && it.qt >= p.split_from;
  it.q0 = it.qt * kAttnRows;
  const int n = it.qt + 1;                           // causal: key tiles 0..qt
  it.j0 = it.split && it.half ? n >> 1 : 0;          // this item's key tiles: j0 .. j0 + n_kv - 1
  it.n_kv = (it.split && !it.half ? n >> 1 : n) - it.j0;
  it.slot = it.split ? (it.seq * p.H + it.h) * (p.q_tiles - p.split_from) + (it.qt - p.split_from) : 0;
  return it;
}

// 2^x for x <= 0 through the bare special-function instruction (exp2f adds a range fix-up for
// denormal results, which a probability does not need; the softmax is bound by this pipe).
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
#endif

// The items of one head, (query tile << 1 | half), by descending number of key tiles, so that the alternating rounds of the
// persistent CTAs pair a long item with a short one; query tiles from split_from on are two halves.
std::vector<int> attention_item_order(int q_tiles, int split_from);
int attention_item_tiles(int entry, int split_from);      // key tiles of an entry of that list
inline int64_t attention_bf16_ctas(bool alone, int sms) { return (alone ? 1 : 2) * (int64_t)sms; }

// How the kernel for bf16 operands spreads `heads` (sequences times heads) of q_tiles query tiles over the SMs.
struct AttnSchedule {
  int split_from;            // query tiles from this one on are shared by two CTAs
  bool alone;                // one CTA to an SM: a launch that cannot fill two on each would put them on half of the SMs
};
AttnSchedule attention_bf16_schedule(int64_t heads, int q_tiles, int sms, bool may_split);
bool attention_bf16_prepare();
cudaError_t attention_bf16_launch(bool pdl, dim3 grid, bool alone, cudaStream_t s, const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v,
                                  const CUtensorMap& out, const CUtensorMap& out16, const AttnParams& p);

}  // namespace kb200
