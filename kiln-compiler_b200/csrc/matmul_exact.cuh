// Exact FP32 on SM pairs for sm_100a: a Linear of more than 128 rows with float32 operands and float32 sums
// (`tl.dot(..., input_precision="ieee")`, kiln/gpu/codegen.py:515, 563-598), as float16 products.
//
// Every operand comes as two float16 terms under a power of two per row of A and column of B (split_rows.cu), which hold as many bits of
// it as the two TF32 terms of the other exact kernels: a b ~ h h + h t + t h.  Why float16: its products take half the tensor time of TF32's
// and a pair half of the bytes, and those two bounded the TF32 form (947 cycles for 128 x 128 x 32, 768 of them multiplying).
//
// Why the sums leave tensor memory after every 64 of K: the tensor core cuts off a bit of the accumulator with every MMA, ~4.5e-8 of it for 8 of K on
// the average, an error that adds up along the sign of what is in it (positive operands, 768 of K in one accumulator
// 4.2e-6, in two 2.3e-6).  The epilogue's warps, idle during a main loop, add every step's products up in registers, rounded as
// float32 sums are; the next steps go to other columns meanwhile.  The step's small products come first, while its accumulator is small; the first
// large one brings it down by 2^11, the power of two of the tails.
//
// Tiles are 256 x BN on the two SMs of a cluster (`.cta_group::2`), as in matmul_pair.cu, whose notes on pairs, producers and the leader's
// barriers hold here too; persistent, one CTA per SM, 384 threads:
//   warp 0      TMA producer: this CTA's 128 rows of A and its half of the columns of B, heads and tails, a stage per 64 of K
//   warp 1      tensor-memory allocation; in the leader the MMA issuer: eight small products, four large ones, a commit that hands the
//               stage back to both CTAs and one that hands the step's accumulator on
//   warps 4-11  two per tensor-memory lane quadrant; a lane has a row, warp h of a quadrant the 32-column blocks h, h + 2, ...: adds up
//               the steps, then scales, finishes and stores its blocks while the tensor cores work on the next tile
//
// Few tiles and a long K (SPLIT): a cluster of two to four pairs, each with its part of K for the same tile of 128 columns.  A pair finishes
// some of the tile's 32-column blocks: the sums of the others' are sent into their rings, idle by then, as bulk copies, and added up in the
// order of the pairs.
//
// Rows of A whose elements are more than 2^28 apart come in further levels (split16.cuh): their tiles go over K once more per level, with the planes of
// that level and the same ones of B, and the sums of its steps are multiplied by the level's power of two as they are added up, by 0 for rows
// that have none.  Why not per row: a tile multiplies 256 of them anyway.  1024 x 2304 x 768 15.5 us (with the pass), one such row 20.0, all 23.7, all with
// two levels 30.5; 4096^3 331, 365, 643, 984.  Of normally distributed rows of 768 one in 2 10^5 has such an element by chance.  (Where no row has
// one, asking costs a launch behind another ~0.2 us: 1024 x 768 block 75.6 -> 77.8.)
// Every wait is bounded: see matmul_pair.cu.
#pragma once

#include <cuda.h>

#include "device_math.cuh"
#include "kb200_internal.h"
#include "split16.cuh"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"
#include "tc_pair.cuh"

namespace kb200 {

namespace {

using namespace tc;

constexpr int kExactThreads = 384;
constexpr int kExactWarps = 8;                       // that add up and finish
constexpr int kExactFirstWarp = 4;
// Registers: 384 threads are launched with 168 each; the four warps in front, two of them idle, give up 112 of theirs, so that a thread
// of the others has room for the sums of a 256-column tile (128 x 56 + 256 x 224 = 384 x 168).
constexpr int kExactRegistersFew = 56, kExactRegistersMany = 224;
static_assert(128 * kExactRegistersFew + 256 * kExactRegistersMany == kExactThreads * 168, "what the launch brings");
constexpr int kExactMaxStages = 4;
constexpr int kExactMaxSums = 4;                     // accumulators of a step that tensor memory holds: 512 columns / BN
constexpr int kExactABytes = 128 * 128;              // one plane of A, 128 rows x 64 of K
constexpr int kExactSlot = 4096;                     // a staged block of 32 x 32
constexpr int kExactSmem = 224 * 1024;
constexpr int kExactStepK = 64;

enum : int { BAR_FULL = 0, BAR_EMPTY = kExactMaxStages, BAR_READY = 2 * kExactMaxStages, BAR_ADDED = BAR_READY + kExactMaxSums,
             BAR_RES = BAR_ADDED + kExactMaxSums, BAR_RECV = BAR_RES + kExactWarps, BAR_PEER = BAR_RECV + kExactWarps, BAR_COUNT = BAR_PEER + 1 };

enum : int { FIN_NONE = 0, FIN_BIAS, FIN_BIAS_GELU, FIN_BIAS_RES };

struct ExactParams {
  int bn, half_bn, stages, steps;
  int parts;             // SPLIT: pairs to a tile, two to four, each with its part of K
  int sums;              // accumulators in turn
  uint32_t idesc;
  int tiles_n, num_tiles;
  uint64_t magic_tn;
  int kernel_index;
  int* status;
  int M, N;
  const float* a_scale;  // what a row's products are to be multiplied by; below zero: the row holds infinities (see redo_row)
  const float* b_scale;
  const uint8_t* a_marks;      // by row, zero up to the last tile's end: the levels behind the first that it has
  const float* bias;
  const float* res;      // as the map of it, for redo_row
  int64_t res_row;
  const float* a;        // the operands as they are in memory, for redo_row
  const float* b;
  int64_t a_row, b_k, b_n, K;
  int stream_out;        // the output leaves L2 first: see streams_out
  int with_tail;         // the output minus its 19 leading bits is stored as well, for a consumer that splits it
  // ... or float16 pairs of it, times a power of two for every 32 columns: its bound is known (see layernorm_bounds), its rows hold no
  // infinities where those of A hold none, and the float32 output may be left out
  const float* pair_scale;
  int store32;
};

// Results of a row of A with infinities, whose float16 terms are NaN, done over as the CUDA cores do them, in the block of 32 x 32 that a
// warp has staged (this lane's row, m).
template <int FIN>
__device__ __noinline__ void redo_row(const ExactParams& p, uint8_t* block, int lane, int64_t m, int n0) {
  for (int c = 0; c < 32 && n0 + c < p.N; ++c) {
    const float* const a = p.a + m * p.a_row;
    const float* const b = p.b + (n0 + c) * p.b_n;
    float y = 0.0f;
#pragma unroll 8
    for (int64_t k = 0; k < p.K; ++k) y = fmaf(a[k], b[k * p.b_k], y);
    if (FIN != FIN_NONE) y += p.bias[n0 + c];
    if (FIN == FIN_BIAS_GELU) y = d_gelu_tanh(y);
    if (FIN == FIN_BIAS_RES) y += p.res[m * p.res_row + n0 + c];
    *reinterpret_cast<float*>(block + lane * 128 + (((c >> 2) ^ (lane & 7)) << 4) + (c & 3) * 4) = y;
  }
}

// This lane's row of a staged block added to v.
__device__ __forceinline__ void add_staged(float (&v)[32], const uint8_t* block, int lane) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float4 t = *reinterpret_cast<const float4*>(block + lane * 128 + ((q ^ (lane & 7)) << 4));
    const float2 a = fadd2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(t.x, t.y));
    const float2 b = fadd2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(t.z, t.w));
    v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = b.x; v[4 * q + 3] = b.y;
  }
}

// K in parts: the first of a tile's four blocks that pair `part` finishes (two, two | two, one, one | one each), a block's pair, and where in
// the area for it a part comes, in blocks of a lane quadrant.
__device__ __forceinline__ int first_block_of(int part, int parts) { return parts == 2 ? 2 * part : parts == 3 && part > 0 ? part + 1 : part; }
__device__ __forceinline__ int owner_of(int block, int parts) { return parts == 2 ? block >> 1 : parts == 3 && block > 0 ? block - 1 : block; }
__device__ __forceinline__ int received_at(int block, int from, int parts) { return (block * (parts - 1) + from) * 4; }

// The marks of a tile's 256 rows, a lane's eight of them, and the levels behind the first that a tile with these has.  (Both volatile: asked for in
// front of the tile's steps and looked at behind them, not ~700 cycles of L2 in front of the first.)
__device__ __forceinline__ uint2 tile_marks(const ExactParams& p, int tm, int lane) {
  uint2 marks;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(marks.x), "=r"(marks.y) : "l"(p.a_marks + (int64_t)tm * 256 + lane * 8) : "memory");
  return marks;
}
__device__ __forceinline__ int levels_behind(uint2 marks) {
  uint32_t any;
  asm volatile("or.b32 %0, %1, %2;" : "=r"(any) : "r"(marks.x), "r"(marks.y));
  any |= any >> 16;
  any |= any >> 8;
  return __popc(__reduce_or_sync(0xffffffffu, any & 3u));
}

// BLOCKS: 32-column blocks of a tile per warp, at most.
template <int BLOCKS, int FIN, bool SPLIT>
__global__ void __launch_bounds__(kExactThreads, 1)
mm_exact_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ CUtensorMap tma_out,
                const __grid_constant__ CUtensorMap tma_res, const __grid_constant__ CUtensorMap tma_tail, const __grid_constant__ ExactParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[BAR_COUNT];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) float columns[kExactWarps][2][32];      // scales and biases of the block a warp is finishing

  const uint32_t ring = smem_u32(smem_raw);          // 1024-byte aligned, as the 128-byte swizzle wants it
  const int b_plane = p.half_bn * 128, stage_bytes = 2 * (kExactABytes + b_plane);
  const uint32_t slots = ring + (uint32_t)(p.stages * stage_bytes);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  // with SPLIT the CTAs 0, 1 and 2, 3 (and so on) of a cluster are a pair each, `pair` counts clusters, and a cluster has one tile
  const uint32_t leader = SPLIT ? rank & 6u : 0u;
  rank &= 1u;
  const int parts = SPLIT ? p.parts : 1, part = (int)leader / 2;
  const int pair = SPLIT ? (int)blockIdx.x / (2 * parts) : blockIdx.x >> 1, num_pairs = SPLIT ? p.num_tiles : gridDim.x >> 1;
  const int step0 = SPLIT ? (part * p.steps + parts - 1) / parts : 0;                             // this pair's steps of K
  const int n_steps = SPLIT ? ((part + 1) * p.steps + parts - 1) / parts - step0 : p.steps;
  const uint16_t pair_ctas = (uint16_t)(3u << leader);
  const uint32_t bar0 = smem_u32(&bars[0]);
  const uint32_t full0 = bar0 + 8 * BAR_FULL, empty0 = bar0 + 8 * BAR_EMPTY, ready0 = bar0 + 8 * BAR_READY, added0 = bar0 + 8 * BAR_ADDED;

  if (threadIdx.x == 32) {
    prefetch_tensormap(&tma_a);
    prefetch_tensormap(&tma_b);
    prefetch_tensormap(&tma_out);
    if (FIN == FIN_BIAS_RES) prefetch_tensormap(&tma_res);
  }
  if (warp == 0) {
    if (lane == 0) abort_flag = 0;
    for (int b = lane; b < BAR_COUNT; b += 32)
      // (both CTAs' warps release an accumulator; a CTA of every other pair says that its ring is idle)
      mbar_init(bar0 + 8 * b, b >= BAR_ADDED && b < BAR_RES ? 2 * kExactWarps : SPLIT && b == BAR_PEER ? parts - 1 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  cluster_arrive_relaxed();           // every CTA's barriers exist once all have arrived (fence.mbarrier_init is what orders)
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_slot;         // (all 512 columns: the same address in both CTAs)
  cluster_wait();
  volatile int* abort_ptr = &abort_flag;
  auto give_up = [&](int site) {
    if (!*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | site); *abort_ptr = 1; }
  };
  // A role is walked by a whole warp; its waits end for all lanes or none.
  auto all_waited = [&](bool got, int site) {
    if (!got && lane == 0) give_up(site);
    return __all_sync(0xffffffffu, got ? 1 : 0) != 0;
  };
  const uint32_t full_leader0 = map_to_cta(full0, leader);
  // (One box brings both planes of an operand: issuing a bulk copy costs its warp ~200 cycles.)
  // The weights are nobody's output: their first stages are requested before the wait for the previous kernel.
  int ahead = 0;
  if (warp == 0 && pair < p.num_tiles) {
    const int tn = pair - pair_div(pair, p.magic_tn) * p.tiles_n;
    ahead = p.stages < n_steps ? p.stages : n_steps;
    if (elect_one()) {
      for (int s = 0; s < ahead; ++s) {
        if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (uint32_t)stage_bytes);
        tma_load_3d_pair(ring + (uint32_t)(s * stage_bytes + 2 * kExactABytes), &tma_b, full_leader0 + 8 * s, (step0 + s) * kExactStepK,
                         tn * p.bn + (int)rank * p.half_bn, 0);
      }
    }
    __syncwarp();
  }
  pdl_wait();                 // everything above may have overlapped the previous kernel's tail; from here on its output is read
  pdl_launch_dependents();

  if (warp < kExactFirstWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kExactRegistersFew));
    if (warp == 0) {
      // ---------------- TMA producer ----------------
      int s = 0;
      uint32_t parity = 1;
      bool ok = true;
      for (int tile = pair; tile < p.num_tiles && ok; tile += num_pairs) {
        const int tm = pair_div(tile, p.magic_tn), tn = tile - tm * p.tiles_n;
        const int m = tm * 256 + (int)rank * 128, n = tn * p.bn + (int)rank * p.half_bn;
        const uint2 marks = tile_marks(p, tm, lane);
        for (int level = 0, more = 0; level <= more && ok; ++level) {
          int k = step0 * kExactStepK;
          for (int i = 0; i < n_steps; ++i, k += kExactStepK) {
            ok = all_waited(mbar_wait_long(empty0 + 8 * s, parity, abort_ptr), 1);
            if (!ok) break;
            const bool b_here = ahead > 0;           // expected and requested above
            const uint32_t bar = full_leader0 + 8 * s, dst = ring + (uint32_t)(s * stage_bytes);
            if (elect_one()) {
              // the leader's barrier counts the bytes of both CTAs
              if (!b_here && rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (uint32_t)stage_bytes);
              tma_load_3d_pair(dst, &tma_a, bar, k, m, 2 * level);
              if (!b_here) tma_load_3d_pair(dst + 2 * kExactABytes, &tma_b, bar, k, n, 0);
            }
            __syncwarp();
            if (b_here) --ahead;
            if (++s == p.stages) { s = 0; parity ^= 1; }
          }
          if (level == 0) more = levels_behind(marks);
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer (leader CTA) ----------------
      if (rank == 0) {
        const int stages = p.stages, sums = p.sums, bn = p.bn;
        const uint32_t idesc = p.idesc;
        const uint64_t fixed = make_desc(0, 16, 1024);
        // (the 14-bit address field: the CTA rank in the upper bits of a cluster's shared window must not spill over.  Masked once: the ring
        // lies below the field's end.)
        const uint32_t first16 = (ring >> 4) & 0x3FFFu, stage16 = (uint32_t)stage_bytes >> 4, plane16 = (uint32_t)b_plane >> 4;
        const uint32_t fixed_lo = (uint32_t)fixed, fixed_hi = (uint32_t)(fixed >> 32);
        auto desc = [&](uint32_t at) { return ((uint64_t)fixed_hi << 32) | (fixed_lo + at); };
        int s = 0, sum = 0;
        uint32_t parity = 0, added_parity = 1;
        // (One loop over all steps: a level's or a tile's end is looked at behind its last one, off the path of the others.)
        int tile = pair, left = n_steps, level = 0, more = 0;
        uint2 marks = tile < p.num_tiles ? tile_marks(p, pair_div(tile, p.magic_tn), lane) : make_uint2(0, 0);
        while (tile < p.num_tiles) {
          // both CTAs' warps have added up what was here
          if (!all_waited(mbar_wait(added0 + 8 * sum, added_parity, abort_ptr), 4) || !all_waited(mbar_wait(full0 + 8 * s, parity, abort_ptr), 2)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t on = elect_one() ? 1u : 0u;
          const uint32_t a = first16 + (uint32_t)s * stage16, at = a + (kExactABytes >> 4), b = a + (2 * kExactABytes >> 4), bt = b + plane16;
          const uint32_t d = tmem + (uint32_t)(sum * bn);
#pragma unroll
          for (int k = 0; k < 8; k += 2) {
            umma_pair<true>(on, d, desc(at + k), desc(b + k), idesc, k != 0 ? 1u : 0u);
            umma_pair<true>(on, d, desc(a + k), desc(bt + k), idesc, 1u);
          }
#pragma unroll
          for (int k = 0; k < 8; k += 2) {
            if (k == 0) umma_pair_onto<kTailBits>(on, d, desc(a), desc(b), idesc);
            else umma_pair<true>(on, d, desc(a + k), desc(b + k), idesc, 1u);
          }
          if (on) {
            umma_pair_commit(empty0 + 8 * s, pair_ctas);
            umma_pair_commit(ready0 + 8 * sum, pair_ctas);
          }
          __syncwarp();
          if (++s == stages) { s = 0; parity ^= 1; }
          if (++sum == sums) { sum = 0; added_parity ^= 1; }
          if (--left == 0) {
            left = n_steps;
            if (level == 0) more = levels_behind(marks);
            if (level++ == more) {
              level = 0;
              tile += num_pairs;
              if (tile < p.num_tiles) marks = tile_marks(p, pair_div(tile, p.magic_tn), lane);
            }
          }
        }
      }
    }
  } else {
    // ---------------- warps 4..11 ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kExactRegistersMany));
    const int e = warp - kExactFirstWarp, quad = warp & 3, half = e >> 2;
    const uint32_t slot = slots + (uint32_t)(e * kExactSlot), lanes = (uint32_t)(quad * 32) << 16;
    const uint32_t res_bar = bar0 + 8 * (BAR_RES + e), recv_bar = bar0 + 8 * (BAR_RECV + e);
    const uint32_t added_leader0 = map_to_cta(added0, leader);
    const int blocks = p.bn / 32;
    // the blocks of a tile that this pair finishes
    const int first_block = SPLIT ? first_block_of(part, parts) : 0, end_block = SPLIT ? first_block_of(part + 1, parts) : blocks;
    const uint64_t policy = l2_policy(p.stream_out != 0);
    uint32_t res_phase = 0;
    int sum = 0;
    uint32_t ready_parity = 0;
    bool ok = true, dry = true;
    float sums[BLOCKS][32];
    constexpr int kAtOnce = BLOCKS < 4 ? 2 : 1;              // blocks loaded under one wait, as far as the registers go
    for (int tile = pair; tile < p.num_tiles && ok;) {
      const int tm = pair_div(tile, p.magic_tn), tn = tile - tm * p.tiles_n;
      const int m_first = tm * 256 + (int)rank * 128 + quad * 32, n0 = tn * p.bn;
      const bool rows_ok = m_first < p.M;
      const float row_scale = m_first + lane < p.M ? p.a_scale[m_first + lane] : 1.0f;
      const uint2 marks = tile_marks(p, tm, lane);
      // scales and biases of this warp's columns, a lane's of each block, before the sums are ready
      float scale_of[BLOCKS], bias_of[BLOCKS];
#pragma unroll
      for (int j = 0; j < BLOCKS; ++j) {
        const int n = n0 + 32 * (half + 2 * j) + lane;
        scale_of[j] = n < p.N ? __ldg(p.b_scale + n) : 0.0f;
        bias_of[j] = FIN != FIN_NONE && n < p.N ? __ldg(p.bias + n) : 0.0f;
      }
      const bool last = SPLIT || tile + num_pairs >= p.num_tiles;
      // a residual's first block is on its way while the products are summed
      int first_own = -1;
      if (rows_ok)
        for (int j = BLOCKS - 1; j >= 0; --j) {
          const int c = half + 2 * j;
          if (c >= first_block && c < end_block && n0 + 32 * c < p.N) first_own = j;
        }
      if (FIN == FIN_BIAS_RES && !dry && lane == 0 && first_own >= 0) {
        store_wait_read(0);
        mbar_expect_tx(res_bar, kExactSlot);
        tma_load_3d(slot, &tma_res, res_bar, n0 + 32 * (half + 2 * first_own), m_first, 0);
      }
#pragma unroll
      for (int j = 0; j < BLOCKS; ++j)
#pragma unroll
        for (int q = 0; q < 32; ++q) sums[j][q] = 0.0f;
      // The first pass over what finishes a tile is a rehearsal, as in matmul_pair.cu: its code is cold at every launch.
      float2 down = make_float2(1.0f, 1.0f);
      for (int level = 0, more = 0; level <= more && ok; ++level) {
        if (level > 0) {       // (rows that have no such level: whatever finite numbers its planes hold)
          const bool taken = (p.a_marks[m_first + lane] >> (level - 1) & 1u) != 0;
          down.x = down.y = !taken ? 0.0f : level == 1 ? 1.0f / kLevelUp : 1.0f / kLevelUp / kLevelUp;
        }
        for (int i = 0; i < n_steps && !dry; ++i) {
          if (!mbar_wait_long(ready0 + 8 * sum, ready_parity, abort_ptr)) give_up(3);
          ok = __shfl_sync(0xffffffffu, *abort_ptr ? 0 : 1, 0) != 0;
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = tmem + lanes + (uint32_t)(sum * p.bn + 32 * half);
#pragma unroll
          for (int j = 0; j < BLOCKS; j += kAtOnce) {
            if (half + 2 * j >= blocks) break;
            float w[kAtOnce][32];
            if (kAtOnce == 2 && j + 1 < BLOCKS && half + 2 * j + 2 < blocks) tmem_ld32x2(at + (uint32_t)(64 * j), at + (uint32_t)(64 * j + 64), w[0], w[kAtOnce - 1]);
            else tmem_ld32(at + (uint32_t)(64 * j), w[0]);
#pragma unroll
            for (int i = 0; i < kAtOnce && j + i < BLOCKS; ++i)
#pragma unroll
              for (int q = 0; q < 32; q += 2) {
                const float2 t = ffma2(make_float2(w[i][q], w[i][q + 1]), down, make_float2(sums[j + i][q], sums[j + i][q + 1]));
                sums[j + i][q] = t.x;
                sums[j + i][q + 1] = t.y;
              }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(added_leader0 + 8 * sum);
          if (++sum == p.sums) { sum = 0; ready_parity ^= 1; }
        }
        if (ok && level == 0) {
          more = levels_behind(marks);
          if (dry) break;
        }
      }
      if (!ok) break;
      auto pick = [&](float (&v)[32], int j) {
#pragma unroll
        for (int q = 0; q < 32; ++q) v[q] = sums[0][q];
#pragma unroll
        for (int i = 1; i < BLOCKS; ++i)
          if (j == i)
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] = sums[i][q];
      };
      // SPLIT: the sums of the other pairs' columns leave for their CTAs with the same rows, those of this one's columns (a block a warp, at most)
      // come from there.  The rings are idle: behind the four blocks that this CTA may send is what it gets, by block and pair.
      [[maybe_unused]] const uint32_t recv_area = (uint32_t)(blocks * 4 * 4096);
      if constexpr (SPLIT) {
        if (!dry) {
          if (e == 0 && lane < parts && lane != part) mbar_arrive_remote(map_to_cta(bar0 + 8 * BAR_PEER, 2 * lane + rank));      // this CTA's ring may be written
          if (lane == 0 && first_own >= 0) mbar_expect_tx(recv_bar, (uint32_t)(parts - 1) * 4096u);
          bool free = false;
#pragma unroll 1
          for (int j = 0; j < BLOCKS; ++j) {
            const int c = half + 2 * j;
            if (c >= blocks || !rows_ok || n0 + 32 * c >= p.N) break;
            if (c >= first_block && c < end_block) continue;
            const uint32_t at = (uint32_t)((c * 4 + quad) * 4096);
            float v[32];
            pick(v, j);
            uint8_t* const mine = smem_raw + at;
            stage_rows(mine, mine, v, lane, false);
            fence_async_smem();
            __syncwarp();
            if (!free) {
              free = all_waited(mbar_wait_cluster(bar0 + 8 * BAR_PEER, 0, abort_ptr), 7);
              if (!free) break;
            }
            if (lane == 0) {
              const int owner = owner_of(c, parts);
              const uint32_t to = recv_area + (uint32_t)(received_at(c - first_block_of(owner, parts), part < owner ? part : part - 1, parts) + quad) * 4096u;
              push_block(map_to_cta(ring + to, 2 * owner + rank), ring + at, 4096, map_to_cta(recv_bar, 2 * owner + rank));
            }
          }
        }
      }
      // Blocks are staged in the warp's slot, one after the other; on the last tile all but the first in the ring, idle by then.
      auto staging = [&](int j) {
        return j == first_own || !last ? slot : ring + (uint32_t)((e * (BLOCKS - 1) + j - first_own - 1) * kExactSlot);
      };
      // One block of the residual at a time, on the last tile one ahead (lane 0)
      [[maybe_unused]] auto request = [&](int j) {
        mbar_expect_tx(res_bar, kExactSlot);
        tma_load_3d(staging(j), &tma_res, res_bar, n0 + 32 * (half + 2 * j), m_first, 0);
      };
#pragma unroll 1
      for (int j = first_own; j >= 0 && j < BLOCKS; ++j) {
        const int c = half + 2 * j, n = n0 + 32 * c;
        if (c >= end_block || n >= p.N) break;          // uniform across the warp
        const uint32_t at = staging(j);
        uint8_t* const at_ptr = smem_raw + (at - ring);
        // What is staged in the slot may still be on its way out: with a short K a tile's sums are ready before the last tile's store has read
        // it.  (A residual's first block is there already, behind a wait of its own.)
        if (at == slot && lane == 0 && !(FIN == FIN_BIAS_RES && j == first_own)) {
          store_wait_read(0);
          if (FIN == FIN_BIAS_RES) request(j);
        }
        float scale = scale_of[0], bias = bias_of[0];
#pragma unroll
        for (int i = 1; i < BLOCKS; ++i)
          if (j == i) { scale = scale_of[i]; bias = bias_of[i]; }
        columns[e][0][lane] = scale;
        if (FIN != FIN_NONE) columns[e][1][lane] = bias;
        __syncwarp();
        float v[32];
        pick(v, j);
        if constexpr (SPLIT) {
          if (!dry) {
            if (!mbar_wait_cluster(recv_bar, 0, abort_ptr)) give_up(6);
            __syncwarp();
            for (int from = 0; from < parts - 1; ++from)
              add_staged(v, smem_raw + recv_area + (received_at(c - first_block, from, parts) + quad) * 4096, lane);
          }
        }
        // (the columns' scales first: their exponents are within 2^60, a row's need not be)
        const float2 of_row = make_float2(fabsf(row_scale), fabsf(row_scale));
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 t = *reinterpret_cast<const float4*>(&columns[e][0][4 * q]);
          float2 x = fmul2(fmul2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(t.x, t.y)), of_row);
          float2 y = fmul2(fmul2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(t.z, t.w)), of_row);
          if (FIN != FIN_NONE) {
            const float4 u = *reinterpret_cast<const float4*>(&columns[e][1][4 * q]);
            x = fadd2(x, make_float2(u.x, u.y));
            y = fadd2(y, make_float2(u.z, u.w));
          }
          v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = y.x; v[4 * q + 3] = y.y;
        }
        if (FIN == FIN_BIAS_GELU) gelu_tanh_pairs(v);
        __syncwarp();
        if (FIN == FIN_BIAS_RES) {
          if (!dry) {
            if (!mbar_wait(res_bar, res_phase, abort_ptr)) give_up(5);
            res_phase ^= 1u;
            __syncwarp();
            const int next = c + 2;
            if (last && lane == 0 && next < end_block && n0 + 32 * next < p.N) request(j + 1);
          }
          add_staged(v, at_ptr, lane);
        }
        __syncwarp();
        const bool redo = row_scale < 0.0f && !dry;
        if (p.store32) {
          stage_rows(at_ptr, at_ptr, v, lane, false);
          if (redo) redo_row<FIN>(p, at_ptr, lane, m_first + lane, n);
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && !dry) {
            tma_store_3d(&tma_out, at, n, m_first, 0, policy);
            tma_store_commit();
          }
        }
        if (p.pair_scale != nullptr) {
          if (p.store32 && lane == 0) store_wait_read(0);
          __syncwarp();
          stage_pairs(at_ptr, v, lane, __ldg(p.pair_scale + (n >> 5)));
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && !dry) {
            tma_store_3d(&tma_tail, at, n, m_first, 0);
            tma_store_3d(&tma_tail, at + 2048, n, m_first, 1);
            tma_store_commit();
          }
        }
        if (p.with_tail && !dry) {
          if (redo) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float4 t = *reinterpret_cast<const float4*>(at_ptr + lane * 128 + ((q ^ (lane & 7)) << 4));
              v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
            }
          }
#pragma unroll
          for (int q = 0; q < 32; ++q) v[q] -= __uint_as_float(__float_as_uint(v[q]) & 0xFFFFE000u);
          if (lane == 0) store_wait_read(0);
          __syncwarp();
          stage_rows(at_ptr, at_ptr, v, lane, false);
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tma_tail, at, n, m_first, 0);
            tma_store_commit();
          }
        }
        if (dry) break;
      }
      if (dry) dry = false;
      else tile += num_pairs;
    }
    if (lane == 0) store_wait_read(0);   // shared memory must outlive the stores that read it
  }

  // ---------------- common exit ----------------
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) let_copies_land();
  __syncwarp();
  // neither CTA leaves (or frees TMEM the other's MMAs write) before both are done
  cluster_arrive_relaxed();
  cluster_wait();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

}  // namespace

}  // namespace kb200
