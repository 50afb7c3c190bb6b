// Tensor-core matmul for problems of few tiles: one row of 128-row tiles (prompts of up to 128 tokens), or
// so few in all that most SMs would idle.  Same role as matmul_tc.cu for the Linears of a transformer
// (bias, bias + GELU, bias + residual; kiln/gpu/codegen.py:484-530, 563-598) in all three precisions.
//
// What bounds such a problem is latency: an SM takes ~64 bytes a clock from L2, so a lone CTA that walks
// 768 of K (24 slabs of 24 KB) needs 5 us for its operands however fast the tensor cores are, and every
// phase that runs once -- set-up, first copy, drain, exchange, epilogue -- costs its instruction fetches
// from a cold cache on top of its latencies.  So:
//   * K is split over the CTAs of a thread-block cluster until the SMs are used, and the whole K range of
//     a CTA is in flight at once where shared memory holds it;
//   * every warp sends the rows it has read from the accumulator to the CTA that finishes their band as
//     soon as it has staged them, data and arrival count in one bulk copy.  (matmul_tc.cu parks the whole
//     tile, passes a barrier and pushes bands: ~6000 cycles of a launch.)
//   * the epilogue is written for its chain, over float4 items in row order: bias and residual are
//     fetched before the accumulator is ready, stores cover whole lines;
//   * weights are requested before the wait for the previous kernel.
// The sum over the splits runs in rank order, so results do not depend on timing.
//
// Per CTA, 352 threads: warp 0 loads A, warp 10 loads B, warp 1 issues the MMAs, warps 2-9 (two per tensor-memory
// lane quadrant) move A to tensor memory, then drain, exchange and finish.  An A that is float32 where the MMAs want bf16 is rounded on that
// way; one whose rows are on no pitch of 16 bytes comes through four tensor maps (GATHER).  Waits are bounded as in matmul_tc.cu.
#include <cuda.h>
#include <cuda_bf16.h>

#include <type_traits>

#include "device_math.cuh"
#include "kb200_internal.h"
#include "matmul.h"
#include "matmul_small.h"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"

namespace kb200 {

namespace {

using namespace tc;

constexpr int kSmallM = 128;
constexpr int kSmallThreads = 352;
constexpr int kSmallEpiWarps = 8;
constexpr int kSmallMaxStages = 8;
constexpr int kSmallABytes = kSmallM * 128;      // one 128-byte K slab
constexpr int kSmallACols = 128;                 // tensor-memory columns for slabs of A
constexpr int kSmallSmem = 225 * 1024;
constexpr size_t kSmallAloneSmem = 164 * 1024;   // beside this, 228 KB an SM have less left than the 65 KB of the smallest clustered launch
constexpr int kSmallMaxSlots = 5;                // exact FP32: accumulators of 64 columns beside that of the small products and the slabs of A

// SMALL_BF16_A32: bf16 products of an A that is still float32, rounded on its way to tensor memory.  (A Linear of the caller's
// own input; a launch that made a bf16 copy of it cost ~2.3 us in front of this one.)
enum : int { SMALL_TF32 = 0, SMALL_BF16 = 1, SMALL_EXACT = 2, SMALL_BF16_A32 = 3 };
enum : int { FIN_NONE = 0, FIN_BIAS, FIN_BIAS_GELU, FIN_BIAS_RES };

struct SmallParams {
  int stages, num_steps, slab_k, splits;
  int b_kmajor, b_static;
  // Exact FP32: accumulators of the large products (that of the small ones is behind them); log2 of the MMAs of a step that go
  // into one, and, where that is all of them (2), the steps.
  int acc_slots, acc_shift, acc_steps;
  uint32_t b_lbo, b_sbo, b_layout, b_step16;
  uint32_t idesc;
  int tmem_cols;
  int tiles_n;
  int kernel_index;
  int* status;
  int M, N;
  const float* bias;
  const float* res;
  int64_t res_row;
  const float* a;                  // exact FP32: A as it is in memory, rows of K elements a_row apart
  int64_t a_row;
  const float* b;                  // exact FP32: B as it is in memory, and its strides along K and N
  int64_t b_k, b_n;
  int K;
  int a_rows;                      // rows of a box of A: the tile's, or M where that is less (GATHER: a quarter, in each map)
  float* out;                      // null: only the bf16 copy is stored
  __nv_bfloat16* out16;            // or null
  float* out_tail;                 // exact FP32: the output minus its 19 leading bits, for a consumer that splits it, or null
  int64_t out_row;                 // of both
  int vectors;                     // exact FP32: 0 where N or a row's start is off float4: bias, residual and output element by element
};

// 128-byte slabs of K per pipeline step.  A step costs the issuing warp ~400 cycles of wait, branches and commits
// beside ~25 per MMA; exact FP32 has twelve MMAs to a slab and, like the float32 A, no room for more.
__host__ __device__ constexpr int slabs_per_step(int mode) { return mode == SMALL_EXACT || mode == SMALL_BF16_A32 ? 1 : 2; }
// A stage: the slabs of A (one of float32 for bf16 products is two boxes of 32 columns), then those of B (exact FP32: and its tails)
__host__ __device__ constexpr int a_slab_bytes(int mode) { return mode == SMALL_BF16_A32 ? 2 * kSmallABytes : kSmallABytes; }
__host__ __device__ constexpr int gather_pitch_floats(int mode) { return mode == SMALL_EXACT ? 36 : 68; }      // of a row in shared memory, see GatherMaps
__host__ __device__ constexpr int a_stage_bytes(int mode, bool gather) {
  return gather ? kSmallM * gather_pitch_floats(mode) * 4 : slabs_per_step(mode) * a_slab_bytes(mode);
}
__host__ __device__ constexpr int b_boxes(int mode) { return mode == SMALL_BF16_A32 ? 1 : 2; }
__host__ __device__ constexpr int stage_bytes_of(int mode, int bn, bool gather) { return a_stage_bytes(mode, gather) + b_boxes(mode) * bn * 128; }

__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<uint32_t*>(&h);
}

// The rows of A on no pitch (GATHER): four tensor maps, of every fourth row each, whose pitch is four rows and so a multiple of 16 bytes.  A
// map's base is rounded down to 16 bytes, `shift` floats in front of its first row; boxes are four columns wider than a step and the warps
// that move A read from `shift` on.  Row 4 i + c of a tile is accumulator row 32 c + i: a warp's 32 rows are of one map and have one shift.
// (Rows of 36 or 68 floats in shared memory: an odd number of 16-byte units, so that a warp's loads have no bank conflicts.)
// (`count` and `shift` are here, not in SmallParams, whose other launches would pass them along.)
struct GatherMaps {
  CUtensorMap of[4];
  int count;
  int shift[4];
};
template <bool GATHER> __device__ __forceinline__ int matrix_row(int row) { return GATHER ? 4 * (row & 31) + (row >> 5) : row; }

// What a TF32 operand does not hold of x.
__device__ __forceinline__ float dropped_bits(float x) { return x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u); }

// Exact FP32: an infinite operand makes a NaN of its tail's products (inf x 0, inf - inf) where float32 has an infinity.  Results
// that are NaN, of the tile's accumulator rows `row`, row + rows_apart, ... below row_end and columns n to n + 3, done over as the CUDA cores do them.
template <int FIN, bool GATHER>
__device__ __noinline__ void redo_in_float32(const SmallParams& p, int m0, int row, int row_end, int rows_apart, int n) {
  for (; row < row_end; row += rows_apart) {
    const int m = m0 + matrix_row<GATHER>(row);
    if (m >= p.M) continue;
    for (int c = n; c < n + 4 && c < p.N; ++c) {
      float* const out = p.out + (int64_t)m * p.out_row + c;
      if (*out == *out) continue;
      const float* const a = p.a + m * p.a_row;
      const float* const b = p.b + c * p.b_n;
      float y = 0.0f;
#pragma unroll 8
      for (int k = 0; k < p.K; ++k) y = fmaf(a[k], b[k * p.b_k], y);
      if (FIN != FIN_NONE) y += p.bias[c];
      if (FIN == FIN_BIAS_GELU) y = d_gelu_tanh(y);
      if (FIN == FIN_BIAS_RES) y += p.res[(int64_t)m * p.res_row + c];
      *out = y;
      if (p.out_tail != nullptr) p.out_tail[(int64_t)m * p.out_row + c] = dropped_bits(y);
    }
  }
}

// BN: columns of a tile, 64, 96 or 128.  GATHER: rows of A on no pitch.  Of a Linear of 333 x 1000 x 771 the pass that copied A to aligned
// rows, and the one that made bf16 of a float32 A, was a launch of ~2.3 us in front of this one.
// DRAINS: exact FP32, more steps than the accumulators take.  (The adding up in the loop, and its registers, cost 3 % where it does
// nothing: 1024 x 768 x 3072 29.0 us, 27.9 without.)
template <int MODE, int FIN, int BN, bool GATHER, bool DRAINS>
__global__ void __launch_bounds__(kSmallThreads, 1)
mm_small_kernel(const __grid_constant__ std::conditional_t<GATHER, GatherMaps, CUtensorMap> tma_a, const __grid_constant__ CUtensorMap tma_b,
                const __grid_constant__ CUtensorMap tma_bt, const __grid_constant__ SmallParams p) {
  constexpr bool EXACT = MODE == SMALL_EXACT;
  constexpr int kSmallBBytes = BN * 128;
  constexpr int kTileBytes = kSmallM * BN * 4;
  constexpr int kABuffers = 2;                                  // steps of A in tensor memory, 64 columns each
  constexpr int kBlocks = BN / 32;                              // 32-column blocks of the tile, the first (or only) half of them to the first group of four warps
  constexpr int kSlabs = slabs_per_step(MODE);
  constexpr bool A32 = MODE == SMALL_BF16_A32, BF16 = MODE == SMALL_BF16 || A32;
  constexpr bool ALTERNATE = kSlabs == 1;                       // the two groups of warps that move A take alternate steps
  constexpr int kSlabA = a_slab_bytes(MODE), kBBoxes = b_boxes(MODE), kStage = stage_bytes_of(MODE, BN, GATHER), kStageA = a_stage_bytes(MODE, GATHER);
  constexpr int kGatherRow = gather_pitch_floats(MODE) * 4;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[3 * kSmallMaxStages + 4 + kSmallMaxSlots];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const uint32_t raw_at = smem_u32(smem_raw);
  const uint32_t ring = (raw_at + 1023u) & ~1023u;
  // This CTA's partial tile in 32 x 32 blocks of 4 KB: in the ring, idle by then, where it is large enough
  const bool in_ring = p.stages * kStage >= kTileBytes;
  const uint32_t recv = in_ring ? ring : ring + (uint32_t)(p.stages * kStage);
  // A cluster: the others' parts of this CTA's band
  const uint32_t parts0 = ring + (uint32_t)(p.stages * kStage) + (in_ring ? 0u : (uint32_t)kTileBytes);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kSmallMaxStages]), split0 = smem_u32(&bars[2 * kSmallMaxStages]);
  const uint32_t done = smem_u32(&bars[3 * kSmallMaxStages]), received = done + 8, tfree0 = done + 16, drained0 = done + 32;
  const int tile = blockIdx.x / p.splits;
  const int rank = blockIdx.x - tile * p.splits;                // in the cluster: its CTAs are consecutive
  const int tm = tile / p.tiles_n, tn = tile - tm * p.tiles_n;
  const int step0 = rank * p.num_steps / p.splits, n_steps = (rank + 1) * p.num_steps / p.splits - step0;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 2);
      mbar_init(empty0 + 8 * s, 1);
      mbar_init(split0 + 8 * s, ALTERNATE ? kSmallEpiWarps / 2 : kSmallEpiWarps);
    }
    mbar_init(done, 1);
    mbar_init(received, 1);
    for (int i = 0; i < kABuffers; ++i) mbar_init(tfree0 + 8 * i, 1);
    for (int i = 0; DRAINS && i < p.acc_slots; ++i) mbar_init(drained0 + 8 * i, kSmallEpiWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(received, (uint32_t)(kTileBytes / p.splits * (p.splits - 1)));     // (an arrival, too; a launch without a split does not use it)
  }
  if (threadIdx.x == 32) {
    if constexpr (GATHER) {
      for (int c = 0; c < 4; ++c) prefetch_tensormap(&tma_a.of[c]);
    } else {
      prefetch_tensormap(&tma_a);
    }
    prefetch_tensormap(&tma_b);
    if (EXACT) prefetch_tensormap(&tma_bt);
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // The next kernel's set-up may overlap all of this one (it waits for it to complete) -- from here on: its
  // CTAs must not take tensor memory that this one still has to allocate.
  pdl_launch_dependents();
  // Every CTA's barriers exist once all have arrived here; waited for in front of the exchange.  A launch
  // without a split is no cluster launch and keeps off the cluster instructions (a store to a mapped
  // address in one is an illegal instruction).
  const bool clustered = p.splits > 1;
  if (clustered) cluster_arrive_relaxed();        // (fence.mbarrier_init above is what orders)
  const uint32_t tmem = tmem_slot;
  [[maybe_unused]] const uint32_t tmem_a = tmem + (uint32_t)((EXACT ? p.acc_slots + 1 : 1) * BN);      // the slabs of A
  volatile int* abort_ptr = &abort_flag;
  auto give_up = [&](int site) {
    if (!*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | site); *abort_ptr = 1; }
  };
  // a frozen B is nobody's output: its producer does not wait for the previous kernel
  if (warp < 2 || (warp == 10 && !p.b_static)) pdl_wait();

  // A whole warp walks each of the three roles below; its waits end for all lanes or none.
  auto all_waited = [&](bool got, int site) {
    if (!got && lane == 0) give_up(site);
    return __all_sync(0xffffffffu, got ? 1 : 0) != 0;
  };
  if (warp == 0 || warp == 10) {
    // ---------------- TMA producers, one per operand ----------------
    const bool is_a = warp == 0;
    int s = 0, k_elem = step0 * kSlabs * p.slab_k;
    uint32_t parity = 1;
    for (int i = 0; i < n_steps; ++i) {
      if (i >= p.stages && !all_waited(mbar_wait(empty0 + 8 * s, parity, abort_ptr), 1)) break;
      const uint32_t bar = full0 + 8 * s, dst = ring + (uint32_t)(s * kStage), b_dst = dst + kStageA;
      if (elect_one()) {
        uint32_t a_bytes = kSlabs * (kSlabA / kSmallM) * p.a_rows;
        if constexpr (GATHER) a_bytes = tma_a.count * p.a_rows * kGatherRow;
        mbar_expect_tx(bar, is_a ? a_bytes : kBBoxes * kSmallBBytes);
        if constexpr (GATHER) {
          if (is_a)
            for (int c = 0; c < tma_a.count; ++c) tma_load_3d(dst + c * 32 * kGatherRow, &tma_a.of[c], bar, k_elem, tm * 32, 0);
        }
        // (a slab past the end of K, in the last step of an odd number, is a box outside the tensor: zeros)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int k = EXACT ? k_elem : A32 ? k_elem + j * 32 : k_elem + j * p.slab_k;
          if (is_a) {
            if constexpr (!GATHER)
              if (j < kSlabs || A32) tma_load_3d(dst + j * kSmallABytes, &tma_a, bar, k, tm * kSmallM, 0);
          } else if (j < kBBoxes) {
            const CUtensorMap* map = EXACT && j ? &tma_bt : &tma_b;
            if (p.b_kmajor) tma_load_3d(b_dst + j * kSmallBBytes, map, bar, k, tn * BN, 0);
            else tma_load_4d(b_dst + j * kSmallBBytes, map, bar, 0, k, tn * (BN / (BF16 ? 64 : 32)), 0);
          }
        }
      }
      __syncwarp();
      k_elem += kSlabs * p.slab_k;
      if (++s == p.stages) { s = 0; parity ^= 1; }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const uint64_t b_fixed = p.b_kmajor ? make_desc(0, 16, 1024) : make_desc(0, p.b_lbo, p.b_sbo, p.b_layout);
    const uint32_t b_step = p.b_step16, idesc = p.idesc;
    int s = 0, buf = 0;
    [[maybe_unused]] int slot = 0, in_slot = 0;
    [[maybe_unused]] uint32_t acc_at = tmem;       // the slot's columns
    [[maybe_unused]] bool again = false;           // the slots are being used again ...
    [[maybe_unused]] uint32_t refill = 1;          // ... and are free with this phase of `drained`
    uint32_t parity = 0;
    bool ok = true;
    for (int i = 0; i < n_steps && ok; ++i) {
      if (DRAINS && again && in_slot == 0) ok = all_waited(mbar_wait(drained0 + 8 * slot, refill, abort_ptr), 8);
      if (!ok) break;
      ok = all_waited(mbar_wait(split0 + 8 * s, parity, abort_ptr), 2);        // this step's A is in tensor memory (and so its B has landed)
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t b16 = (ring + (uint32_t)(s * kStage + kStageA)) >> 4;
      const uint32_t on = elect_one() ? 1u : 0u;
      // (the 14-bit address field: the CTA rank in the upper bits of a cluster's shared window must not spill over)
      auto desc = [&](uint32_t at) { return b_fixed | (uint64_t)(at & 0x3FFFu); };
      if constexpr (EXACT) {
        // a b ~ tail(a) b + a tail(b) + a b.  The tensor core truncates every accumulation, an error of ~2^-24 of what the
        // accumulator holds each time (positive operands, 3072 of K over eight CTAs, one accumulator: 2.7e-6).  So
        // no accumulator takes more than the host allows (see accumulate_as), and the warps below add them up in
        // float32.  The small products, whose error is 2^-11 of that, have one of their own.
        const uint32_t apart = tmem + (uint32_t)(p.acc_slots * BN);
        const uint32_t more = in_slot != 0 ? 1u : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t b = b16 + k * b_step, ta = tmem_a + (uint32_t)(buf * 64 + 8 * k);
          umma_ts_if(on, apart, ta + 32, desc(b), idesc, (i | k) != 0, false);
          umma_ts_if(on, apart, ta, desc(b + (kSmallBBytes >> 4)), idesc, 1u, false);
          umma_ts_if(on, acc_at, ta, desc(b), idesc, k == 0 ? more : p.acc_shift == 2 || (p.acc_shift == 1 && (k & 1)) ? 1u : 0u, false);
          if (p.acc_shift == 0 || (p.acc_shift == 1 && (k & 1))) acc_at += BN;
        }
        if (p.acc_shift == 2 && ++in_slot == p.acc_steps) {
          in_slot = 0;
          acc_at += BN;
          if (DRAINS && ++slot == p.acc_slots) { slot = 0; acc_at = tmem; again = true; refill ^= 1; }
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4 * kSlabs; ++k) {
          const uint32_t b = b16 + (k >> 2) * (kSmallBBytes >> 4) + (k & 3) * b_step, ta = tmem_a + (uint32_t)(buf * 64 + 8 * k);
          umma_ts_if(on, tmem, ta, desc(b), idesc, (i | k) != 0, BF16);
        }
      }
      if (on) {
        if (i + p.stages < n_steps) umma_commit(empty0 + 8 * s);
        if (i + kABuffers < n_steps) umma_commit(tfree0 + 8 * buf);
        if (i + 1 == n_steps) umma_commit(done);
      }
      __syncwarp();
      buf ^= 1;
      if (++s == p.stages) { s = 0; parity ^= 1; }
    }
  } else {
    // ---------------- warps 2..9 ----------------
    const int e = warp - 2, quad = warp & 3, half = e >> 2, t = threadIdx.x - 64;
    const int band_rows = kSmallM / p.splits;
    // The parameters are read through the constant cache, cold at every launch: touch what the end of the
    // kernel needs now, under the wait.
    asm volatile("" ::"l"(p.bias), "l"(p.res), "l"(p.res_row), "l"(p.out), "l"(p.out16), "l"(p.out_row), "r"(p.M), "r"(p.N), "r"(p.acc_slots), "r"(p.acc_steps) : "memory");
    // this thread's items of the band: float4 number t, t + 256, ... in row order, eight at a time
    constexpr int kUnits = BN / 4, kRowsAtOnce = 256 / kUnits;
    const int band0 = rank * band_rows, m0 = tm * kSmallM, n0 = tn * BN;
    const int u = t % kUnits, r0 = t < kUnits * kRowsAtOnce ? t / kUnits : kSmallM;      // (96 columns: 16 threads have none)
    const int n = n0 + 4 * u;
    pdl_wait();
    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load4 = [&](const float* from) {
      if (!EXACT || p.vectors) return *reinterpret_cast<const float4*>(from);
      return make_float4(from[0], n + 1 < p.N ? from[1] : 0.f, n + 2 < p.N ? from[2] : 0.f, n + 3 < p.N ? from[3] : 0.f);
    };
    if (FIN != FIN_NONE && n < p.N) bias = load4(p.bias + n);
    auto load_res = [&](int r) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      const int m = m0 + matrix_row<GATHER>(band0 + r);
      if (FIN == FIN_BIAS_RES && r < band_rows && m < p.M && n < p.N) x = load4(p.res + (int64_t)m * p.res_row + n);
      return x;
    };
    float4 res = load_res(r0);
    bool ok = true;
    // Exact FP32: this warp's rows of its half of the tile's columns, added up from the accumulators
    constexpr int kHalfBlocks = (kBlocks + 1) / 2;
    [[maybe_unused]] float sum[EXACT ? kHalfBlocks : 1][32];
    [[maybe_unused]] int drained = 0, drain_slot = 0;             // accumulators added so far, and the next one's slot
    [[maybe_unused]] auto add_slot = [&](int slot) {
#pragma unroll
      for (int c = 0; c < (EXACT ? kHalfBlocks : 0); ++c) {
        if (half * kHalfBlocks + c >= kBlocks) continue;
        float w[32];
        tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(slot * BN + (half * kHalfBlocks + c) * 32), w);
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[c][j] += w[j];
      }
    };
    [[maybe_unused]] auto drain = [&](bool free_it) {
      add_slot(drain_slot);
      if (free_it) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(drained0 + 8 * drain_slot);
      }
      ++drained;
      if (++drain_slot == p.acc_slots) drain_slot = 0;
    };
    if constexpr (EXACT) {
#pragma unroll
      for (int c = 0; c < kHalfBlocks; ++c)
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[c][j] = 0.0f;
    }
    {
      // A goes to tensor memory, 32 columns a slab (exact FP32: values and tails, what their 19 leading bits leave).
      // The tensor core reads an operand from shared memory at ~64 bytes a clock: with A there an MMA of 128
      // rows and 64 columns took 133 cycles, from tensor memory ~65, and in exact FP32, where A and its
      // tails were made in shared memory, a slab moved 136 KB through it (960 cycles a slab, now 690).
      // A lane has a row.  A slab is a chain of waits, loads, stores to tensor memory and an arrival, ~500 cycles
      // whatever its size: of two groups of four warps, one per lane quadrant, each takes one slab of a step,
      // or, one slab to a step, alternate steps.  (Every stage and buffer then belongs to one group, which
      // sees each phase of its barriers: an even number of stages where the ring is used again.)
      constexpr int kEvery = ALTERNATE ? 2 : 1;
      int s = ALTERNATE ? half : 0;
      uint32_t parity = 0;
      const int row = quad * 32 + lane;
      [[maybe_unused]] int shift = 0;
      if constexpr (GATHER) shift = tma_a.shift[quad];
      for (int i = s; i < n_steps && ok; i += kEvery) {
        const int buf = i % kABuffers;
        if (!mbar_wait(full0 + 8 * s, parity, abort_ptr)) give_up(7);
        // (loading and splitting A in front of this wait takes no less time: the issuing warp, in whose scheduler two of these
        // warps are, is held up by them then)
        if (i >= kABuffers && !mbar_wait(tfree0 + 8 * buf, ((i / kABuffers) & 1) ^ 1, abort_ptr)) give_up(6);
        ok = __shfl_sync(0xffffffffu, *abort_ptr ? 0 : 1, 0) != 0;
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint8_t* const src = smem_raw + (ring - raw_at) + s * kStage + (ALTERNATE ? 0 : half * (GATHER ? 128 : kSlabA)) + row * (GATHER ? kGatherRow : 128);
        float v[32];
        if constexpr (GATHER) {
          // the 32 (A32: 64) columns of this slab from `shift` on, a uniform number
          auto from = [&](auto first) {
            constexpr int S = decltype(first)::value;
            float raw[A32 ? 68 : 36];
#pragma unroll
            for (int q = 0; q < (A32 ? 17 : 9); ++q) {
              const float4 x = *reinterpret_cast<const float4*>(src + 16 * q);
              raw[4 * q] = x.x; raw[4 * q + 1] = x.y; raw[4 * q + 2] = x.z; raw[4 * q + 3] = x.w;
            }
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] = A32 ? __uint_as_float(pack_bf16(raw[(2 * q + S) % 68], raw[(2 * q + 1 + S) % 68])) : raw[(q + S) % 36];
          };
          if (shift == 0) from(std::integral_constant<int, 0>());
          else if (shift == 1) from(std::integral_constant<int, 1>());
          else if (shift == 2) from(std::integral_constant<int, 2>());
          else from(std::integral_constant<int, 3>());
        }
#pragma unroll
        for (int q = GATHER ? 16 : 0; q < (A32 ? 16 : 8); ++q) {
          const float4 x = *reinterpret_cast<const float4*>(src + (q >> 3) * kSmallABytes + (((q & 7) ^ (row & 7)) << 4));
          if (A32) {
            v[2 * q] = __uint_as_float(pack_bf16(x.x, x.y)); v[2 * q + 1] = __uint_as_float(pack_bf16(x.z, x.w));
          } else {
            v[(4 * q) & 31] = x.x; v[(4 * q + 1) & 31] = x.y; v[(4 * q + 2) & 31] = x.z; v[(4 * q + 3) & 31] = x.w;
          }
        }
        const uint32_t at = tmem_a + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * 64 + (ALTERNATE ? 0 : half * 32));
        tmem_st32(at, v);
        if constexpr (EXACT) {
#pragma unroll
          for (int q = 0; q < 32; ++q) v[q] = cut_tail(v[q]);
          tmem_st32(at + 32, v);
        }
        tmem_st_wait();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(split0 + 8 * s);
        // Accumulators that the ring of slots needs again: those whose steps end at i - 2, whose MMAs the wait for this
        // step's buffer of A has seen complete.
        if (DRAINS && n_steps > p.acc_slots * p.acc_steps)
          while ((drained + 1) * p.acc_steps + 1 <= i) drain(true);
        s += kEvery;
        if (s >= p.stages) { s -= p.stages; parity ^= 1; }
      }
    }
    if (ok && !mbar_wait(done, 0, abort_ptr)) give_up(3);
    ok = __shfl_sync(0xffffffffu, *abort_ptr ? 0 : 1, 0) != 0;
    __syncwarp();
    if (clustered) cluster_wait();              // every CTA's `received` exists
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if constexpr (EXACT) {
#pragma unroll 1
        for (const int all = (n_steps << (2 - p.acc_shift)) + p.acc_steps - 1; (drained + 1) * p.acc_steps <= all;) drain(false);
        add_slot(p.acc_slots);
      }
#pragma unroll(EXACT ? kHalfBlocks : 1)
      for (int c = 0; c < kHalfBlocks; ++c) {
        const int cb = half * kHalfBlocks + c;
        if (cb >= kBlocks) break;
        float v[32];
        if constexpr (EXACT) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = sum[c][j];
        } else {
          tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cb * 32), v);
        }
        // This 32 x 32 block goes to the CTA that finishes its rows (two CTAs, 16 rows each, with eight
        // splits): staged in 128-byte rows, the 16-byte unit XORed with the row, then one bulk copy per
        // destination that carries its arrival.  The rows of this CTA's own band stay where they are
        // staged.  (st.async straight from the registers, 16 bytes per lane and packet, took 3700 cycles
        // to land where these take ~1500.)
        const uint32_t block = (uint32_t)((cb * 4 + quad) * 4096);
        uint8_t* const mine = smem_raw + (recv - raw_at) + block + lane * 128;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<float4*>(mine + ((q ^ (lane & 7)) << 4)) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        if (clustered) {
          fence_async_smem();
          __syncwarp();
          const int pieces = band_rows < 32 ? 2 : 1, rows = band_rows < 32 ? 16 : 32;
          if (lane < pieces) {
            const int row = quad * 32 + lane * rows, dest = row / band_rows;
            if (dest != rank) {
              // in the destination's area: [source, the destination left out][32-column block][row of the band]
              const int source = rank < dest ? rank : rank - 1;
              const uint32_t to = parts0 + (uint32_t)((source * kBlocks + cb) * band_rows + (row - dest * band_rows)) * 128u;
              asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                           ::"r"(map_to_cta(to, (uint32_t)dest)), "r"(recv + block + (uint32_t)(lane * rows * 128)), "r"((uint32_t)(rows * 128)),
                             "r"(map_to_cta(received, (uint32_t)dest))
                           : "memory");
            }
          }
        }
      }
    }
    __syncwarp();
    if (clustered) {
      if (!mbar_wait_cluster(received, 0, abort_ptr)) give_up(5);
      __syncwarp();
      cluster_arrive_relaxed();
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");      // the eight warps have staged this CTA's own part
    ok = __shfl_sync(0xffffffffu, *abort_ptr ? 0 : 1, 0) != 0;
    if (ok) {
      // Item by item: row r0 + kRowsAtOnce * j, float4 number u.  A rolled loop: the code runs once, cold, and
      // eight unrolled items were 2000 to 3000 cycles of instruction fetches whatever their number.
      const uint8_t* const area = smem_raw + (parts0 - raw_at);
      const uint8_t* const own = smem_raw + (recv - raw_at);
      const int cb = u >> 3;
      [[maybe_unused]] bool any_nan = false;
#pragma unroll 1
      for (int r = r0; r < band_rows; r += kRowsAtOnce) {
        const float4 res_next = load_res(r + kRowsAtOnce);
        const int row = band0 + r, m = m0 + matrix_row<GATHER>(row);
        const int swizzled = ((u ^ r) & 7) << 4;
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        const uint8_t* part = area + (cb * band_rows + r) * 128 + swizzled;
#pragma unroll 1
        for (int s = 0; s < p.splits; ++s) {          // in rank order
          const bool mine = s == rank;
          const float4 b = *reinterpret_cast<const float4*>(mine ? own + (cb * 4 + (row >> 5)) * 4096 + (row & 31) * 128 + swizzled : part);
          if (!mine) part += kBlocks * band_rows * 128;
          y.x += b.x; y.y += b.y; y.z += b.z; y.w += b.w;
        }
        if (EXACT) {
          const float all = (y.x + y.y) + (y.z + y.w);
          any_nan = any_nan || all != all;
        }
        if (FIN != FIN_NONE) { y.x += bias.x; y.y += bias.y; y.z += bias.z; y.w += bias.w; }
        if (FIN == FIN_BIAS_GELU) {
          if (BF16) {
            y.x = f_gelu_tanh_approx(y.x); y.y = f_gelu_tanh_approx(y.y); y.z = f_gelu_tanh_approx(y.z); y.w = f_gelu_tanh_approx(y.w);
          } else {
            y.x = d_gelu_tanh(y.x); y.y = d_gelu_tanh(y.y); y.z = d_gelu_tanh(y.z); y.w = d_gelu_tanh(y.w);
          }
        }
        if (FIN == FIN_BIAS_RES) { y.x += res.x; y.y += res.y; y.z += res.z; y.w += res.w; }
        res = res_next;
        if (m >= p.M || n >= p.N) continue;
        if (EXACT && !p.vectors) {
          float* const to = p.out + (int64_t)m * p.out_row + n;
          to[0] = y.x;
          if (n + 1 < p.N) to[1] = y.y;
          if (n + 2 < p.N) to[2] = y.z;
          if (n + 3 < p.N) to[3] = y.w;
          continue;
        }
        if (p.out != nullptr) *reinterpret_cast<float4*>(p.out + (int64_t)m * p.out_row + n) = y;
        if (EXACT && p.out_tail != nullptr)
          *reinterpret_cast<float4*>(p.out_tail + (int64_t)m * p.out_row + n) = make_float4(dropped_bits(y.x), dropped_bits(y.y), dropped_bits(y.z), dropped_bits(y.w));
        if (p.out16 != nullptr) {
          __nv_bfloat162 lo = __floats2bfloat162_rn(y.x, y.y), hi = __floats2bfloat162_rn(y.z, y.w);
          uint2 packed;
          packed.x = *reinterpret_cast<uint32_t*>(&lo);
          packed.y = *reinterpret_cast<uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(p.out16 + (int64_t)m * p.out_row + n) = packed;
        }
      }
      if (EXACT && any_nan) redo_in_float32<FIN, GATHER>(p, m0, band0 + r0, band0 + band_rows, kRowsAtOnce, n);
    }
  }
  // (the warp has to be whole for an .aligned barrier)
  __syncwarp();
  if (clustered && (warp < 2 || warp == 10)) {
    cluster_wait();       // (the other warps have passed this phase above)
    cluster_arrive_relaxed();
  }
  // ---------------- exit ----------------
  if (abort_flag && threadIdx.x == 0) let_copies_land();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // Every CTA of the cluster has received everything: so every copy out of THIS shared memory has landed
  if (clustered) cluster_wait();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)p.tmem_cols) : "memory");
  }
}

using SmallKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, SmallParams);
using GatherKernel = void (*)(GatherMaps, CUtensorMap, CUtensorMap, SmallParams);

struct SmallState {
  CUtensorMap map_a, map_b, map_bt;
  GatherMaps maps_a;
  SmallParams params;
  SmallKernel kernel = nullptr;               // one of these two
  GatherKernel gather = nullptr;
  unsigned grid = 0;
  size_t smem = 0;
  int bias_slot = -1, res_slot = -1;
  int bn = 0;                                 // (these three for small_detail)
  SmallA form = SMALL_A_MAPPED;
  bool drains = false;
  bool a_moves = false, b_moves = false;      // the maps hold the operand's own address
};

template <int MODE, int BN, bool GATHER, bool DRAINS>
auto small_kernel_of(int fin) {
  switch (fin) {
    case FIN_BIAS: return &mm_small_kernel<MODE, FIN_BIAS, BN, GATHER, DRAINS>;
    case FIN_BIAS_GELU: return &mm_small_kernel<MODE, FIN_BIAS_GELU, BN, GATHER, DRAINS>;
    case FIN_BIAS_RES: return &mm_small_kernel<MODE, FIN_BIAS_RES, BN, GATHER, DRAINS>;
    default: return &mm_small_kernel<MODE, FIN_NONE, BN, GATHER, DRAINS>;
  }
}

template <int MODE, bool GATHER, bool DRAINS>
auto small_kernel_of(int fin, int bn) {
  return bn == 128 ? small_kernel_of<MODE, 128, GATHER, DRAINS>(fin) : bn == 96 ? small_kernel_of<MODE, 96, GATHER, DRAINS>(fin) : small_kernel_of<MODE, 64, GATHER, DRAINS>(fin);
}

SmallKernel small_kernel(int mode, int fin, int bn, bool drains) {
  switch (mode) {
    case SMALL_BF16: return small_kernel_of<SMALL_BF16, false, false>(fin, bn);
    case SMALL_BF16_A32: return small_kernel_of<SMALL_BF16_A32, false, false>(fin, bn);
    case SMALL_EXACT: return drains ? small_kernel_of<SMALL_EXACT, false, true>(fin, bn) : small_kernel_of<SMALL_EXACT, false, false>(fin, bn);
    default: return small_kernel_of<SMALL_TF32, false, false>(fin, bn);
  }
}

GatherKernel gather_kernel(int mode, int fin, int bn, bool drains) {
  switch (mode) {
    case SMALL_BF16_A32: return small_kernel_of<SMALL_BF16_A32, true, false>(fin, bn);
    case SMALL_EXACT: return drains ? small_kernel_of<SMALL_EXACT, true, true>(fin, bn) : small_kernel_of<SMALL_EXACT, true, false>(fin, bn);
    default: return small_kernel_of<SMALL_TF32, true, false>(fin, bn);
  }
}

// Floats between the 16-byte boundary in front of row c of A and the row.
int gather_shift(const DevOperand& a, int c) { return (int)(reinterpret_cast<uintptr_t>(a.ptr + c * a.stride[1]) / sizeof(float) % 4); }

int small_mode(int precision, SmallA form) {
  if (precision == KB200_PREC_FP32) return SMALL_EXACT;
  return precision != KB200_PREC_BF16 ? SMALL_TF32 : form == SMALL_A_MAPPED ? SMALL_BF16 : SMALL_BF16_A32;
}

// The chains this kernel finishes: nothing, + column, + column then GELU, + column + matrix.  `vectors`: whether all that it
// reads and writes there is in float4.
int finish_of(const PlanKernel& k, int* bias_slot, int* res_slot, bool* vectors) {
  const Chain& c = k.chain;
  const DevOperand& o = k.ops[c.out_slot];
  *vectors = k.N % 4 == 0 && o.stride[1] % 4 == 0 && aligned16(o.ptr);
  *bias_slot = *res_slot = -1;
  if (c.n == 0) return FIN_NONE;
  const ChainStep* s = c.steps;
  if (s[0].op != CH_ADD || s[0].slot < 0) return -1;
  const DevOperand& b = k.ops[s[0].slot];
  if (b.stride[1] != 0 || b.stride[2] != 1) return -1;
  *vectors = *vectors && aligned16(b.ptr);
  *bias_slot = s[0].slot;
  if (c.n == 1) return FIN_BIAS;
  if (c.n != 2) return -1;
  if (s[1].op == CH_GELU_TANH) return FIN_BIAS_GELU;
  if (s[1].op != CH_ADD || s[1].slot < 0) return -1;
  const DevOperand& r = k.ops[s[1].slot];
  if (r.stride[2] != 1 || r.stride[1] < k.N) return -1;
  *vectors = *vectors && r.stride[1] % 4 == 0 && aligned16(r.ptr);
  *res_slot = s[1].slot;
  return FIN_BIAS_RES;
}

// Clusters of `splits` CTAs, one CTA per SM, that fit the GPU at once (147 SMs in use at most: the SMs of
// a processing cluster need not be a multiple of the size).
int resident_clusters(const Plan& plan, int splits) {
  const int sm_count = plan.sm_count;
  if (splits == 1) return sm_count;
  int& known = plan.resident_clusters[splits];
  if (known == 0) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(splits * (sm_count / splits)), 1, 1);
    cfg.blockDim = dim3(kSmallThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmallSmem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const SmallKernel kernel = mm_small_kernel<SMALL_TF32, FIN_BIAS, 64, false, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = sm_count * 7 / 10 / splits;
    }
    known = n > 0 ? n : 1;
  }
  return known;
}

// Exact FP32: accumulators beside that of the small products and the slabs of A.
constexpr int exact_slots(int bn) { return (512 - kSmallACols) / bn - 1; }
static_assert(exact_slots(64) == kSmallMaxSlots, "barriers of the slots");

// How exact FP32 accumulates `most` steps of a CTA: at most `limit` MMAs along K into one accumulator.  Where the
// accumulators do not last for all steps, the warps that move A add them up as they go (`drains`).
struct Accumulate { int slots, shift, steps; bool drains; };

Accumulate accumulate_as(int most, int bn, int limit) {
  const int all = exact_slots(bn);
  Accumulate a{all, 2, 1, false};
  // few steps: an accumulator for every one, two or four MMAs
  a.shift = limit >= 4 ? 2 : limit >= 2 ? 1 : 0;
  while (a.shift > 0 && (most << (3 - a.shift)) <= all) --a.shift;
  if (most << (2 - a.shift) <= all) {
    a.slots = most << (2 - a.shift);
    return a;
  }
  a.shift = 2;
  const int steps = limit / 4 > 1 ? limit / 4 : 1;
  a.steps = (most + all - 1) / all;
  a.drains = a.steps > steps;
  if (a.drains) a.steps = steps;
  else a.slots = (most + a.steps - 1) / a.steps;
  return a;
}

// MMAs along K that may go into one accumulator: each adds 3.3e-8 to an error of ~5e-8 (positive operands).  Float32 sums
// over K on the CUDA cores, which take the operands that this kernel and no other may have (`close`), err by 1.5e-8 sqrt(K)
// (64: 1.3e-7; 768: 4.2e-7; 3072: 8.5e-7), matmul_tc.cu with K split over a cluster, up to 16 of its
// tiles, by 5.0e-7 to 6.2e-7 and else by 1.1e-6 and more.
int accumulate_limit(int64_t m, int64_t n, int64_t k, bool close) {
  const bool many = m > kSmallM && ((m + 127) / 128) * ((n + 127) / 128) > 16;
  if (many && !close) return 64;
  for (int limit : {12, 8, 4, 2})
    if ((limit + 1.5) * (limit + 1.5) <= 0.2 * (double)k) return limit;
  return 1;
}

struct SmallPlan { int bn, splits; int64_t cycles; };

// Bytes behind the ring: the others' parts of a band, and the own partial tile where the ring cannot hold it.
int exchange_bytes(int mode, int bn, bool gather, int splits, int stages) {
  const int tile_bytes = kSmallM * bn * 4;
  return tile_bytes / splits * (splits - 1) + (stages * stage_bytes_of(mode, bn, gather) >= tile_bytes ? 0 : tile_bytes);
}

// Stages of a CTA with `most` steps: all of them, as far as shared memory goes.
int ring_stages(int mode, int bn, bool gather, int splits, int most) {
  int stages = most < kSmallMaxStages ? most : kSmallMaxStages;
  while ((size_t)stages * stage_bytes_of(mode, bn, gather) + exchange_bytes(mode, bn, gather, splits, stages) + 1024 > (size_t)kSmallSmem) --stages;
  if (slabs_per_step(mode) == 1 && stages < most) stages &= ~1;              // a ring that is used again: see the warps that move A
  return stages;
}

// Tile width, K split and estimated cycles, from fits to measured launches (128 to 1024 rows, 768 and 3072 of K, each
// width and split).  A step, one 128-byte slab of K, is bound by shared memory: the operands land there
// at 128 bytes a clock and every MMA reads its operands again (exact FP32: twelve of them, A from tensor
// memory).  Everything that runs once, launch to exit, is the rest: tiles of 96 columns and
// more have two blocks to a warp to drain, eight CTAs more to exchange.  (Plans in flight are no argument: results must not depend on them.)
// 96 columns fit some row counts better than either neighbour (exact FP32: 1024 x 3072 x 768 36.4 -> 32.6 us,
// 1024 x 768 x 3072 31.2 -> 27.8, 364 x 768 x 3072 22.3 -> 16.4).
// GATHER: four copies to a step for one, and rows that start off the lines; with a ring of two stages (the other forms may have three in the
// same memory) a step waits for its copies.  Copies of A in front of the kernel -> four maps, 384 launches of 2 to 1000 rows: 333 x 1000 x 771 TF32
// 8.7 -> 7.0 us, 128 x 768 x 1537 BF16 7.7 -> 6.2, 600 x 1000 x 771 FP32 16.3 -> 13.3.
SmallPlan plan_small(int64_t m, int64_t n, int64_t k, int mode, bool gather, bool chunked, bool close, const Plan& plan) {
  const int64_t slab_k = mode == SMALL_BF16 || mode == SMALL_BF16_A32 ? 64 : 32, slabs = (k + slab_k - 1) / slab_k;
  SmallPlan best{64, 1, 0};
  const int64_t fetch = !gather ? 0 : 150;
  const int asked_bn = plan.few_tiles % 1000, asked_splits = plan.few_tiles / 1000 % 10;
  for (int bn : {64, 96, 128}) {
    if (asked_bn != 0 && bn != asked_bn) continue;
    if (bn == 96 && chunked) continue;                  // an N-major B comes in chunks of 64 bf16 columns
    const int64_t step = mode == SMALL_EXACT ? 435 + 4 * bn : mode == SMALL_BF16_A32 ? 450 + bn * 25 / 32 : 198 + bn * 13 / 8;
    const int64_t once = (bn == 64 ? 7500 : 10050) + (mode == SMALL_EXACT ? 600 : 0);
    const int64_t tiles = ((m + kSmallM - 1) / kSmallM) * ((n + bn - 1) / bn);
    for (int s : {1, 2, 4, 8}) {
      const int64_t steps = (slabs + slabs_per_step(mode) - 1) / slabs_per_step(mode);
      if (s > steps) break;
      if (asked_splits != 0 && s != asked_splits) continue;
      if (mode == SMALL_EXACT) {
        const Accumulate a = accumulate_as((int)((steps + s - 1) / s), bn, accumulate_limit(m, n, k, close));
        if (a.drains && (a.slots - 1) * a.steps < 2) continue;        // a slot would be needed before its steps are drained
      }
      const int64_t resident = resident_clusters(plan, s);
      const int64_t rounds = (tiles + resident - 1) / resident;
      const int64_t most = (steps + s - 1) / s;
      const int64_t short_ring = gather && most > 2 && ring_stages(mode, bn, gather, s, (int)most) < 3 ? slabs_per_step(mode) * step / 3 : 0;
      const int64_t cycles = rounds * (most * (slabs_per_step(mode) * step + fetch + short_ring) + once + (s == 8 ? 1000 : s > 1 ? 350 : 0));
      if (best.cycles == 0 || cycles < best.cycles) best = {bn, s, cycles};
    }
  }
  return best;
}

}  // namespace

int64_t small_cycles(const Plan& plan, const PlanKernel& k, bool b_kmajor, int64_t b_cols, SmallA form, bool close) {
  const kb200_kernel_desc& d = k.desc;
  const bool bf16 = d.precision == KB200_PREC_BF16;
  int bias_slot, res_slot;
  bool vectors;
  if (!k.has_chain || k.batch != 1 || finish_of(k, &bias_slot, &res_slot, &vectors) < 0) return -1;
  if (!vectors && d.precision != KB200_PREC_FP32) return -1;
  for (int i : {0, 1, 2, 3, 4, 6})
    if (d.cfg[i] != 0) return -1;                     // a tile, stage or split was asked for (how to store is not a question here)
  if (k.M >= (1 << 20) || k.N >= (1 << 24)) return -1;
  if (!b_kmajor && b_cols % (bf16 ? 64 : 32)) return -1;
  if (d.precision == KB200_PREC_FP32 && d.operands[d.b_slot].base_kind != KB200_BASE_CONST) return -1;
  const DevOperand& O = k.ops[k.chain.out_slot];
  if (O.stride[2] != 1 || O.stride[1] < k.N) return -1;
  if (((k.M + kSmallM - 1) / kSmallM) * ((k.N + 63) / 64) > 4096) return -1;
  return plan_small(k.M, k.N, k.K, small_mode(d.precision, form), form == SMALL_A_GATHERED, bf16 && !b_kmajor, close, plan).cycles;
}

int small_sum_length(const Plan& plan, const PlanKernel& k) {
  const SmallPlan how = plan_small(k.M, k.N, k.K, SMALL_EXACT, false, false, false, plan);
  const int64_t steps = (k.K + 31) / 32;
  const Accumulate a = accumulate_as((int)((steps + how.splits - 1) / how.splits), how.bn, accumulate_limit(k.M, k.N, k.K, false));
  return a.shift == 2 ? 4 * a.steps : 1 << a.shift;
}

int small_bind(Plan& plan, PlanKernel& k, int kernel_index, const PairOperands& ops, const float* b_tail, SmallA form, bool close, void** state) {
  *state = nullptr;
  if (k.desc.precision == KB200_PREC_FP32 && b_tail == nullptr)
    return fail(KB200_ERR_ARGUMENT, "matmul %s: the tails of B are missing", k.desc.name);
  SmallState* st = new SmallState();
  SmallParams& p = st->params;
  const kb200_kernel_desc& d = k.desc;
  const int mode = small_mode(d.precision, form);
  const bool gather = form == SMALL_A_GATHERED;
  bool vectors;
  const int fin = finish_of(k, &st->bias_slot, &st->res_slot, &vectors);
  p.vectors = vectors ? 1 : 0;
  const int slab_k = ops.bf16 ? 64 : 32, chunk = ops.bf16 ? 64 : 32;
  p.slab_k = slab_k;
  const int slabs = (int)((k.K + slab_k - 1) / slab_k), per_step = slabs_per_step(mode);
  p.num_steps = (slabs + per_step - 1) / per_step;
  const SmallPlan how = plan_small(k.M, k.N, k.K, mode, gather, ops.bf16 && !ops.b_kmajor, close, plan);
  const int bn = how.bn;
  st->bn = bn;
  st->form = form;
  p.splits = how.splits;
  p.tiles_n = (int)((k.N + bn - 1) / bn);
  const int64_t tiles = ((k.M + kSmallM - 1) / kSmallM) * p.tiles_n;
  const int stage_bytes = stage_bytes_of(mode, bn, gather);
  const int most = (p.num_steps + p.splits - 1) / p.splits;
  p.stages = ring_stages(mode, bn, gather, p.splits, most);
  st->smem = (size_t)p.stages * stage_bytes + exchange_bytes(mode, bn, gather, p.splits, p.stages) + 1024;
  st->grid = (unsigned)(tiles * p.splits);
  p.b_kmajor = ops.b_kmajor ? 1 : 0;
  p.b_static = ops.b_static ? 1 : 0;
  p.b_lbo = (uint32_t)(slab_k * 128);
  p.b_sbo = ops.bf16 ? 1024 : 512;
  p.b_layout = ops.bf16 ? 2 : 1;
  p.b_step16 = ops.b_kmajor ? 2u : (uint32_t)((ops.bf16 ? 16 : 8) * 128) >> 4;
  const uint32_t fmt = ops.bf16 ? 1u : 2u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((ops.b_kmajor ? 0u : 1u) << 16) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(kSmallM >> 4) << 24);
  p.acc_slots = 1;
  p.tmem_cols = 32;
  if (mode == SMALL_EXACT) {
    const Accumulate how_exact = accumulate_as(most, bn, accumulate_limit(k.M, k.N, k.K, close));
    p.acc_slots = how_exact.slots;
    p.acc_shift = how_exact.shift;
    p.acc_steps = how_exact.steps;
    st->drains = how_exact.drains;
  }
  while (p.tmem_cols < (mode == SMALL_EXACT ? p.acc_slots + 1 : 1) * bn + kSmallACols) p.tmem_cols *= 2;
  // Two clusters of plans on different streams must not share SMs where their tensor memory does not fit both: a CTA of each
  // could wait for columns that the other's neighbour holds, until the bounded waits end both.  Of 256 columns two fit (and
  // registers allow no third); with more, shared memory that leaves no room for the smallest such CTA keeps it away.
  if (p.splits > 1 && p.tmem_cols > 256 && st->smem < kSmallAloneSmem) st->smem = kSmallAloneSmem;
  p.kernel_index = kernel_index;
  p.status = plan.d_status;
  p.M = (int)k.M;
  p.N = (int)k.N;
  p.bias = st->bias_slot >= 0 ? k.ops[st->bias_slot].ptr : nullptr;
  p.res = st->res_slot >= 0 ? k.ops[st->res_slot].ptr : nullptr;
  p.res_row = st->res_slot >= 0 ? k.ops[st->res_slot].stride[1] : 0;
  const DevOperand& O = k.ops[k.chain.out_slot];
  p.out16 = static_cast<__nv_bfloat16*>(k.shadow_out);
  p.out = k.mirror_only && p.out16 ? nullptr : O.ptr;
  p.out_row = O.stride[1];
  p.out_tail = mode == SMALL_EXACT && vectors ? k.tail_out : nullptr;
  const DevOperand& A = k.ops[d.a_slot];
  p.a = mode == SMALL_EXACT ? A.ptr : nullptr;
  const DevOperand& B = k.ops[d.b_slot];
  p.b = B.ptr;
  p.b_k = B.stride[1];
  p.b_n = B.stride[2];
  p.a_row = A.stride[1];
  p.K = (int)k.K;
  // (Rows of shared memory that no box fills make accumulator rows that nobody reads.)
  p.a_rows = (int)(k.M < kSmallM ? k.M : kSmallM);
  st->a_moves = gather || form == SMALL_A_FLOAT32 || ops.a_base == A.ptr;
  st->b_moves = ops.b_base == k.ops[d.b_slot].ptr;
  bool ok = true;
  if (gather) {
    p.a_rows = (int)(k.M < kSmallM ? (k.M + 3) / 4 : kSmallM / 4);          // (rows that are not there cost a box as much as others)
    st->maps_a.count = (int)(k.M < 4 ? k.M : 4);
    for (int c = 0; c < st->maps_a.count && ok; ++c) {
      st->maps_a.shift[c] = gather_shift(A, c);
      ok = encode_map_rows(&st->maps_a.of[c], A.ptr + c * A.stride[1] - st->maps_a.shift[c], k.K + st->maps_a.shift[c], (k.M - c + 3) / 4, 4 * A.stride[1], gather_pitch_floats(mode), p.a_rows);
    }
    for (int c = st->maps_a.count; c < 4; ++c) {           // (not used)
      st->maps_a.of[c] = st->maps_a.of[0];
      st->maps_a.shift[c] = 0;
    }
  }
  if (!gather) ok = (form == SMALL_A_FLOAT32 ? encode_map(&st->map_a, false, A.ptr, k.K, k.M, 1, A.stride[1], 0, 32, p.a_rows, false)
                                               : encode_map(&st->map_a, ops.bf16, ops.a_base, k.K, k.M, 1, ops.a_row, 0, slab_k, p.a_rows, false));
  if (ok && ops.b_kmajor) ok = encode_map(&st->map_b, ops.bf16, ops.b_base, k.K, k.N, 1, ops.b_row, 0, slab_k, bn, false);
  else if (ok) ok = encode_map4(&st->map_b, ops.bf16, ops.b_base, chunk, k.K, ops.b_cols / chunk, 1, ops.b_row, 0, slab_k, bn / chunk, !ops.bf16);
  st->map_bt = st->map_b;
  if (ok && b_tail) ok = set_map_address(&st->map_bt, b_tail);
  if (!ok) { delete st; return KB200_OK; }
  if (gather) st->gather = gather_kernel(mode, fin, bn, st->drains);
  else st->kernel = small_kernel(mode, fin, bn, st->drains);
  const cudaError_t e = gather ? cudaFuncSetAttribute(st->gather, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem)
                               : cudaFuncSetAttribute(st->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem);
  if (e != cudaSuccess) { delete st; return cuda_fail(e, "cudaFuncSetAttribute(mm_small_kernel)"); }
  *state = st;
  return KB200_OK;
}

int small_launch(const Plan& plan, const void* state, cudaStream_t s) {
  const SmallState* st = static_cast<const SmallState*>(state);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(st->grid, 1, 1);
  cfg.blockDim = dim3(kSmallThreads, 1, 1);
  cfg.dynamicSmemBytes = st->smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (st->params.splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)st->params.splits;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (plan.pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  if (st->gather) KB200_CUDA(cudaLaunchKernelEx(&cfg, st->gather, st->maps_a, st->map_b, st->map_bt, st->params));
  else KB200_CUDA(cudaLaunchKernelEx(&cfg, st->kernel, st->map_a, st->map_b, st->map_bt, st->params));
  return KB200_OK;
}

bool small_repoint(const PlanKernel& k, void* state) {
  SmallState* st = static_cast<SmallState*>(state);
  if (st->bias_slot >= 0) st->params.bias = k.ops[st->bias_slot].ptr;
  if (st->res_slot >= 0) st->params.res = k.ops[st->res_slot].ptr;
  if (st->params.a) st->params.a = k.ops[k.desc.a_slot].ptr;
  if (st->params.out) st->params.out = k.ops[k.chain.out_slot].ptr;
  const DevOperand& A = k.ops[k.desc.a_slot];
  bool ok = true;
  for (int c = 0; st->gather && c < st->maps_a.count; ++c)      // (by a multiple of 16 bytes: the shifts stay)
    ok = ok && set_map_address(&st->maps_a.of[c], A.ptr + c * A.stride[1] - st->maps_a.shift[c]);
  return ok && (st->gather || !st->a_moves || set_map_address(&st->map_a, A.ptr)) &&
         (!st->b_moves || set_map_address(&st->map_b, k.ops[k.desc.b_slot].ptr));
}

std::string small_detail(const void* state) {
  const SmallState* st = static_cast<const SmallState*>(state);
  const char* const a = st->form == SMALL_A_GATHERED ? ", A gathered" : st->form == SMALL_A_FLOAT32 ? ", A float32" : "";
  return "mm_small " + std::to_string(st->bn) + " columns, " + std::to_string(st->params.splits) + " splits, " + std::to_string(st->params.stages) +
         " stages" + a + (st->drains ? ", drains" : "");
}

bool small_writes_tails(const void* state) { return static_cast<const SmallState*>(state)->params.out_tail != nullptr; }

void small_destroy(void* state) { delete static_cast<SmallState*>(state); }

}  // namespace kb200
