// CTA-pair tensor-core matmul for sm_100a: 256 x BN output tiles computed by the two SMs of a
// thread-block cluster with tcgen05.mma.cta_group::2.  Same role as matmul_tc.cu (the reference's
// matmul generator with a fused epilogue, kiln/gpu/codegen.py:484-530, 563-598) for problems with
// more than 128 rows in the TF32 and BF16 operand modes.
//
// Why pairs: one issuing thread drives the tensor cores of two SMs, every CTA stages only its own
// half of the B tile (half the shared-memory fill and half the B bytes per FLOP of a 128-row
// tile), and a 256 x 128 tile keeps each MMA instruction at 64 tensor cycles per SM, above the
// ~62 cycles an instruction occupies the pipe whatever its width.
//
// A cluster is two CTAs (ranks 0 = leader, 1 = peer), one per SM, persistent over a static list
// of tiles.  Per CTA, 512 threads:
//   warp 0      TMA producer (one lane): its CTA's 128 rows of A and its half of the B columns per
//               pipeline stage, plain (non-multicast) bulk tensor loads with .cta_group::2 so that
//               both CTAs' bytes complete on the LEADER's `full` barrier.
//   warp 1      TMEM allocation (both CTAs execute the .cta_group::2 alloc / dealloc); then, leader
//               only, the MMA issuer (one lane): tcgen05.mma.cta_group::2 (M = 256, N = BN) reads both
//               CTAs' stages and writes each CTA's 128 accumulator rows into that CTA's TMEM; one
//               multicast tcgen05.commit hands the stage back to both CTAs (`empty`) or the
//               accumulator on (`tfull`).
//   warps 2-13  epilogue of the CTA's own 128 rows, three warps per TMEM lane quadrant: tcgen05.ld
//               of a 32-column block, the fused chain with a lane per accumulator row, the block
//               staged in the warp's shared-memory slot and written by bulk tensor stores, float32
//               and / or the bf16 mirror.  A full-matrix operand of the chain (residual, mask) is
//               brought into the slot by a bulk tensor LOAD, so no warp ever gathers rows from
//               global memory.  Accumulators are double buffered in TMEM: the epilogue of tile i
//               runs under the main loop of tile i + 1; both CTAs' warps release the buffer on the
//               leader's `tempty` barrier.  (Warps 14 and 15 are idle: 512 threads are what leaves
//               the compiler 128 registers per thread.)
//
// Few tiles and a long K (SPLIT): the cluster is two pairs, each with half of K for the same tile.  Their accumulators meet
// through shared memory: every epilogue warp sends the 32 x 32 blocks of the other pair's half of the columns as bulk copies
// into that CTA's ring, idle by then, and finishes its own.
// Every mbarrier wait is bounded: on expiry the thread records (kernel, site) in the plan's status
// word, raises its CTA's abort flag, all roles fall through to the exit, which passes the cluster
// barrier (every path reaches it), frees TMEM and returns.  The other CTA's waits run out by themselves.
#include <cuda.h>
#include <cuda_bf16.h>


#include "device_math.cuh"
#include "kb200_internal.h"
#include "matmul.h"
#include "matmul_pair.h"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"
#include "tc_pair.cuh"

namespace kb200 {

namespace {

using namespace tc;

constexpr int kPairThreads = 512;
constexpr int kPairEpiWarps = 12;
constexpr int kPairFirstEpiWarp = 2;
constexpr int kPairWarpsPerQuad = kPairEpiWarps / 4;
constexpr int kPairBlocksPerWarp = (8 + kPairWarpsPerQuad - 1) / kPairWarpsPerQuad;   // 32-column blocks of a 256-column tile (narrower ones have fewer)
constexpr int kPairMaxStages = 8;
constexpr int kPairATileBytes = 128 * 128;        // 128 rows x one 128-byte K slab
constexpr int kPairSmemCeiling = 224 * 1024;      // opt-in ceiling, the same for every launch of the kernel
// barrier indices
constexpr int kBarFull = 0, kBarEmpty = kPairMaxStages, kBarTFull = 2 * kPairMaxStages, kBarTEmpty = kBarTFull + 2,
              kBarRes = kBarTEmpty + 2, kBarRecv = kBarRes + kPairEpiWarps, kBarPeer = kBarRecv + kPairEpiWarps, kBarCount = kBarPeer + 1;

// The chains of a transformer's Linears have epilogues of their own; any other runs step by step.  A step of
// the general form looks its descriptor up, branches on the operand's kind and jumps through a
// switch over every scalar op: ~700 instructions of straight-line code per 32 x 32 block of the GELU
// layer, which the warps fetched at ~25 cycles per 128-byte line (2000-2500 cycles per block, 14 000 per
// tile against 6 100 of its main loop).  Written for one chain, in packed arithmetic, it is ~200.
enum : int { EPI_CHAIN = 0, EPI_BIAS, EPI_BIAS_GELU, EPI_BIAS_RES };

enum : int { SIDE_NONE = 0, SIDE_IMM = 1, SIDE_COL = 2, SIDE_RES = 3 };

struct PairStep {
  int op;                // ChainOp
  int kind;              // SIDE_*
  float imm;
  const float* ptr;      // SIDE_COL: one value per column, contiguous
  int64_t batch_stride;  // SIDE_COL: elements between batch entries
};

struct PairParams {
  // what the producer and the MMA thread need comes first (constant-bank lines touched at start-up)
  int bn, half_bn, stages, num_kb, slab_k, kps, step_k;
  int first_kb;          // SPLIT: steps of the first pair
  int b_static;          // B is a frozen constant: its first stages are requested before the previous kernel has finished
  int b_kmajor;          // B is [N, K] with K contiguous (boxes like A); else [K, N], one 4-D box per stage
  int chunk_n;           // columns per 128-byte row of an N-major B chunk: 32 (tf32) or 64 (bf16)
  uint32_t b_lbo_bytes, b_sbo_bytes, b_layout, b_step16, b_slab16;
  uint32_t idesc;
  int tmem_cols;
  int tiles_n, tiles_per_batch, num_tiles;
  uint64_t magic_tn, magic_tpb;
  int kernel_index;
  int* status;
  // epilogue
  int64_t M, N;
  __nv_bfloat16* out16;  // bf16 mirror of the output (same strides), or null
  int stream_out;        // the float32 output leaves L2 first: see streams_out
  int store32;           // 0: only the mirror is stored (every reader of this output takes the mirror)
  int slots, slot_bytes;
  int res_step;          // chain step whose operand arrives by bulk tensor load, or -1
  int res_batched;       // that operand has one matrix per batch entry (else the same for all)
  int n_steps;
  PairStep steps[kMaxChain];
};

// One stage of this CTA's half of the B tile.
template <int KPS>
__device__ __forceinline__ void load_b_pair(const PairParams& p, const CUtensorMap* map, uint32_t dst, uint32_t bar, int k_elem, int n_col,
                                            int batch) {
  if (p.b_kmajor) {
    for (int j = 0; j < KPS; ++j) tma_load_3d_pair(dst + j * p.half_bn * 128, map, bar, k_elem + j * p.slab_k, n_col, batch);
  } else {
    tma_load_4d_pair(dst, map, bar, 0, k_elem, n_col / p.chunk_n, batch);
  }
}

template <bool BF16, int KPS, int EPI, bool SPLIT>
__global__ void __launch_bounds__(kPairThreads, 1)
mm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
               const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ CUtensorMap tma_out16,
               const __grid_constant__ CUtensorMap tma_res, const __grid_constant__ PairParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kBarCount];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ PairStep chain_steps[kMaxChain];     // looked up by a run-time index for every block
  __shared__ __align__(16) float columns[kPairEpiWarps][32];   // the bias of the block a warp is working on

  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;     // the 128-byte swizzle pattern repeats every 1024 bytes
  const int a_stage_bytes = KPS * kPairATileBytes;
  const int b_stage_bytes = KPS * p.half_bn * 128;
  const int stage_bytes = a_stage_bytes + b_stage_bytes;
  const uint32_t epi_base = tiles + (uint32_t)(p.stages * stage_bytes);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  // with SPLIT the CTAs 0, 1 and 2, 3 of a cluster are a pair each, `pair` counts clusters, and a cluster has one tile
  const uint32_t leader = SPLIT ? rank & 2u : 0u, cta = rank;
  rank &= 1u;
  const int pair = blockIdx.x >> (SPLIT ? 2 : 1), num_pairs = gridDim.x >> (SPLIT ? 2 : 1);
  const int first_kb = SPLIT && leader != 0 ? p.first_kb : 0;                                          // this pair's steps of K
  const int my_kb = !SPLIT ? p.num_kb : leader != 0 ? p.num_kb - p.first_kb : p.first_kb;
  const uint16_t pair_ctas = (uint16_t)(3u << leader);
  const uint32_t full0 = smem_u32(&bars[kBarFull]), empty0 = smem_u32(&bars[kBarEmpty]);
  const uint32_t tfull0 = smem_u32(&bars[kBarTFull]), tempty0 = smem_u32(&bars[kBarTEmpty]);

  if (threadIdx.x == 32) {
    prefetch_tensormap(&tma_a);
    prefetch_tensormap(&tma_b);
    prefetch_tensormap(&tma_out);
    if (p.out16 != nullptr) prefetch_tensormap(&tma_out16);
    if (p.res_step >= 0) prefetch_tensormap(&tma_res);
  }
  if (warp == 0) {
    if (lane == 0) abort_flag = 0;
    for (int b = lane; b < kBarCount; b += 32)
      mbar_init(full0 + 8 * b, b >= kBarTEmpty && b < kBarRes ? 2 * kPairEpiWarps : 1);   // both CTAs' epilogue warps release an accumulator
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The parameter block is read through the constant cache, cold at kernel start: touch the lines the
  // producer and the MMA thread need now, under the set-up, instead of in front of the first copy.
  // Both CTAs' barriers must exist before either signals the other: arrive on the cluster barrier as
  // soon as this CTA's are initialised, wait for it after the TMEM allocation below.
  cluster_arrive_relaxed();
  if (lane == 0 && warp < 2)
    asm volatile("" ::"r"(p.bn), "r"(p.idesc), "r"(p.num_tiles), "l"(p.magic_tn), "l"(p.magic_tpb), "l"(p.status) : "memory");
  if (warp == 2 && lane < kMaxChain) chain_steps[lane] = p.steps[lane];
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"((uint32_t)p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_slot;
  cluster_wait();
  volatile int* abort_ptr = &abort_flag;
  // The MMA instruction names one TMEM address for both CTAs: the two allocations must agree.
  if (threadIdx.x == 0 && rank == 1) {
    const uint32_t leader_base = ld_cluster_u32(map_to_cta(smem_u32(&tmem_base_slot), leader));
    if (leader_base != tmem_base) {
      atomicCAS(p.status, 0, (p.kernel_index << 8) | 9);
      *abort_ptr = 1;
    }
  }
  // A frozen B is nobody's output: the first stages' weights are requested before the wait for the
  // previous kernel, so that they are on their way, or here, when the activations are ready.
  const uint32_t full_leader0 = map_to_cta(full0, leader);
  int ahead = 0;                 // stages of the first tile whose B is requested already (producer warp)
  if (p.b_static && warp == 0 && pair < p.num_tiles) {
    const int batch = pair_div(pair, p.magic_tpb);
    const int rem = pair - batch * p.tiles_per_batch;
    const int n_col = (rem - pair_div(rem, p.magic_tn) * p.tiles_n) * p.bn + (int)rank * p.half_bn;
    ahead = p.stages < my_kb ? p.stages : my_kb;
    if (elect_one()) {
      for (int s = 0; s < ahead; ++s) {
        if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (uint32_t)stage_bytes);
        load_b_pair<KPS>(p, &tma_b, tiles + (uint32_t)(s * stage_bytes + a_stage_bytes), full_leader0 + 8 * s, (first_kb + s) * p.step_k, n_col, batch);
      }
    }
    __syncwarp();
  }
  // Everything above may have overlapped the previous kernel's tail; from here on its output is read.
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    // (like the MMA issuer's, a role that the whole warp walks, one lane issuing: see elect_one)
    const int stages = p.stages, num_tiles = p.num_tiles, num_kb = my_kb, slab_k = p.slab_k, step_k = p.step_k;
    const int bn = p.bn, half_bn = p.half_bn;
    int s = 0;
    uint32_t wait_parity = 1;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      const int batch = pair_div(tile, p.magic_tpb);
      const int rem = tile - batch * p.tiles_per_batch;
      const int tm_i = pair_div(rem, p.magic_tn);
      const int tn_i = rem - tm_i * p.tiles_n;
      const int m_row = tm_i * 256 + (int)rank * 128;
      const int n_col = tn_i * bn + (int)rank * half_bn;
      int k_elem = first_kb * step_k;
      for (int kb = 0; kb < num_kb; ++kb, k_elem += step_k) {
        const bool got = mbar_wait_long(empty0 + 8 * s, wait_parity, abort_ptr);
        if (!__all_sync(0xffffffffu, got ? 1 : 0)) {
          if (lane == 0 && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 1); *abort_ptr = 1; }
          ok = false;
          break;
        }
        // the leader's barrier counts the bytes of both CTAs (the peer's may land first: the phase
        // cannot complete before this arrival)
        const bool b_here = ahead > 0;           // expected and requested above
        const uint32_t bar = full_leader0 + 8 * s;
        const uint32_t dst = tiles + (uint32_t)(s * stage_bytes);
        if (elect_one()) {
          if (!b_here && rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (uint32_t)stage_bytes);
#pragma unroll
          for (int j = 0; j < KPS; ++j) tma_load_3d_pair(dst + j * kPairATileBytes, &tma_a, bar, k_elem + j * slab_k, m_row, batch);
          if (!b_here) load_b_pair<KPS>(p, &tma_b, dst + a_stage_bytes, bar, k_elem, n_col, batch);
        }
        __syncwarp();
        if (b_here) --ahead;
        if (++s == stages) { s = 0; wait_parity ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA) ----------------
    // A step is one barrier probe, 4 * KPS MMAs whose descriptor words advance by additions, and ONE commit
    // for both CTAs (a commit costs about as much as two MMAs).
    if (rank == 0) {
      const int stages = p.stages, num_tiles = p.num_tiles, num_kb = my_kb, bn = p.bn;
      const uint32_t idesc = p.idesc;
      const uint64_t a_fixed = make_desc(0, 16, 1024);
      const uint64_t b_fixed = p.b_kmajor ? make_desc(0, 16, 1024) : make_desc(0, p.b_lbo_bytes, p.b_sbo_bytes, p.b_layout);
      const uint32_t a_hi = (uint32_t)(a_fixed >> 32), b_hi = (uint32_t)(b_fixed >> 32);
      const uint32_t a_lo_fixed = (uint32_t)a_fixed, b_lo_fixed = (uint32_t)b_fixed;   // the bits of the low word above the start address
      const uint32_t b_step16 = p.b_step16, b_slab16 = p.b_slab16;
      // start addresses (16-byte units, 14 bits: the CTA rank in the upper bits of a cluster's shared
      // window address must not spill into the neighbouring fields) of stage 0
      const uint32_t a_first = (tiles >> 4) & 0x3FFFu, stage16 = (uint32_t)stage_bytes >> 4;
      const uint32_t b_first = a_first + ((uint32_t)a_stage_bytes >> 4);
      int s = 0, i = 0;
      uint32_t parity = 0, a16 = a_first, b16 = b_first;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++i) {
        const int acc = i & 1;
        const uint32_t aph = (i >> 1) & 1;
        // both CTAs' epilogue warps have drained this accumulator (two tiles ago)
        const bool drained = mbar_wait_long(tempty0 + 8 * acc, aph ^ 1, abort_ptr);
        if (!__all_sync(0xffffffffu, drained ? 1 : 0)) {
          if (lane == 0 && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 4); *abort_ptr = 1; }
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * bn);
        for (int kb = 0; kb < num_kb; ++kb) {
          const bool landed = mbar_wait(full0 + 8 * s, parity, abort_ptr);
          if (!__all_sync(0xffffffffu, landed ? 1 : 0)) {
            if (lane == 0 && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 2); *abort_ptr = 1; }
            ok = false;
            break;
          }
          // (the lane that issues is a predicate, not a branch: see umma_if)
          const uint32_t on = elect_one() ? 1u : 0u;
#pragma unroll
          for (int j = 0; j < KPS; ++j) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint64_t adesc = ((uint64_t)a_hi << 32) | (a_lo_fixed | ((a16 + (uint32_t)(j * (kPairATileBytes >> 4) + 2 * k)) & 0x3FFFu));
              const uint64_t bdesc = ((uint64_t)b_hi << 32) | (b_lo_fixed | ((b16 + (uint32_t)j * b_slab16 + (uint32_t)k * b_step16) & 0x3FFFu));
              umma_pair<BF16>(on, tmem_d, adesc, bdesc, idesc, (kb | j | k) != 0 ? 1u : 0u);
            }
          }
          if (on) {
            // the stage is free in both CTAs once these MMAs have read it
            umma_pair_commit(empty0 + 8 * s, pair_ctas);
            if (kb + 1 == num_kb) umma_pair_commit(tfull0 + 8 * acc, pair_ctas);
          }
          __syncwarp();
          a16 += stage16;
          b16 += stage16;
          if (++s == stages) { s = 0; parity ^= 1; a16 = a_first; b16 = b_first; }
        }
      }
    }
  } else if (warp >= kPairFirstEpiWarp && warp < kPairFirstEpiWarp + kPairEpiWarps) {
    // ---------------- epilogue (warps 2..13) ----------------
    // Three warps per TMEM lane quadrant (a warp may only touch lanes 32 * (warp % 4) ..+31); warp g of a
    // quadrant takes the 32-column blocks g, g + 3, g + 6 of the tile.  Twelve warps and not eight, because the epilogue is
    // bound by instruction issue and by the latencies inside a pass (tensor-memory load, the wait for
    // the slot's last store, the proxy fence): with two warps per scheduler the schedulers issued in
    // 46 % of the cycles, a probe of independent multiply-adds in 90 %.
    const int e = warp - kPairFirstEpiWarp, quad = warp & 3, group = e >> 2;
    const int slot_bytes = p.slot_bytes;
    const uint32_t slot0 = epi_base + (uint32_t)(e * slot_bytes);
    uint8_t* const slot0_ptr = smem_raw + (slot0 - raw);
    const uint32_t res_bar = smem_u32(&bars[kBarRes + e]);
    const uint32_t tempty_leader0 = map_to_cta(tempty0, leader);
    // the columns of a tile that this pair finishes
    const int c_first = SPLIT && leader != 0 ? p.half_bn : 0, c_end = SPLIT ? c_first + p.half_bn : p.bn;
    const bool has_res = p.res_step >= 0, with16 = p.out16 != nullptr, with32 = p.store32 != 0;
    // where the block's per-column operand passes through shared memory (-1: broadcast by shuffles)
    const int scratch_off = !has_res ? 0 : (with16 ? 4096 : -1);
    const int n_steps = p.n_steps;
    int col_step = -1;
    for (int s = 0; s < n_steps && col_step < 0; ++s)
      if (chain_steps[s].kind == SIDE_COL) col_step = s;
    const uint64_t out_policy = l2_policy(p.stream_out != 0);
    float col_pre[kPairBlocksPerWarp];
#pragma unroll
    for (int j = 0; j < kPairBlocksPerWarp; ++j) col_pre[j] = 0.0f;
    uint32_t res_phase = 0;
    bool ok = true;
    int i = 0;
    bool dry = true;               // the rehearsal pass described at the tile loop
    // The fused chain on one 32 x 32 block held a lane per row (v[q] = column n + q of this lane's row).
    auto run_chain = [&](float (&v)[32], float mine, int n, int batch) {
      for (int s = 0; s < n_steps; ++s) {
        const PairStep st = chain_steps[s];
        float side[32];
        if (st.kind == SIDE_RES) {
          if (!dry) {
            bool landed = mbar_wait(res_bar, res_phase, abort_ptr);
            if (!landed && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 5); *abort_ptr = 1; }
            res_phase ^= 1u;
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 t = *reinterpret_cast<const float4*>(slot0_ptr + lane * 128 + ((q ^ (lane & 7)) << 4));
            side[4 * q] = t.x; side[4 * q + 1] = t.y; side[4 * q + 2] = t.z; side[4 * q + 3] = t.w;
          }
        } else if (s == col_step && scratch_off >= 0) {
          const float4* col_smem = reinterpret_cast<const float4*>(slot0_ptr + scratch_off);
#pragma unroll
          for (int q = 0; q < 8; ++q) {        // every lane reads the same 16 bytes: a broadcast
            const float4 t = col_smem[q];
            side[4 * q] = t.x; side[4 * q + 1] = t.y; side[4 * q + 2] = t.z; side[4 * q + 3] = t.w;
          }
        } else if (s == col_step) {
#pragma unroll
          for (int q = 0; q < 32; ++q) side[q] = __shfl_sync(0xffffffffu, mine, q);
        } else if (st.kind == SIDE_COL) {
          const float4* base = reinterpret_cast<const float4*>(st.ptr + (int64_t)batch * st.batch_stride + n);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 t = n + 4 * q < p.N ? __ldg(base + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            side[4 * q] = t.x; side[4 * q + 1] = t.y; side[4 * q + 2] = t.z; side[4 * q + 3] = t.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; ++q) side[q] = st.imm;
        }
        chain_step32(st.op, v, side);
      }
    };
    // The first pass over the loop body is a rehearsal: while the first tile is still being multiplied
    // the warp runs one block of the same instructions on whatever tensor memory holds, waits for
    // nothing, requests nothing and stores nothing.  The kernel's code is cold at every launch, and the
    // instruction-cache misses of the first real epilogue would otherwise hold back the accumulator the
    // main loop needs two tiles later.
    for (int tile = pair; tile < p.num_tiles && ok;) {
      const int batch = pair_div(tile, p.magic_tpb);
      const int rem = tile - batch * p.tiles_per_batch;
      const int tm_i = pair_div(rem, p.magic_tn);
      const int tn_i = rem - tm_i * p.tiles_n;
      const int acc = dry ? 1 : (i & 1);
      const uint32_t aph = (i >> 1) & 1;
      const int m_first = tm_i * 256 + (int)rank * 128 + quad * 32;
      const int n0 = tn_i * p.bn;
      const bool rows_ok = m_first < p.M;
      // the first per-column operand of the chain (a bias) is fetched for this warp's blocks before the
      // accumulator is ready: lane l holds column l of each block, one coalesced 128-byte load per block
      if (col_step >= 0 && rows_ok) {
        const float* src = chain_steps[col_step].ptr + (int64_t)batch * chain_steps[col_step].batch_stride + n0 + lane;
#pragma unroll
        for (int j = 0; j < kPairBlocksPerWarp; ++j) {
          const int c = c_first + 32 * (group + kPairWarpsPerQuad * j);
          col_pre[j] = (c < c_end && n0 + c + lane < p.N) ? __ldg(src + c) : 0.0f;
        }
      }
      // the first block's matrix operand is requested before the accumulator is ready
      bool res_ready = false;
      if (has_res && !dry && rows_ok && c_first + 32 * group < c_end && n0 + c_first + 32 * group < p.N) {
        if (lane == 0) {
          store_wait_read(0);
          mbar_expect_tx(res_bar, 4096);
          tma_load_3d(slot0, &tma_res, res_bar, n0 + c_first + 32 * group, m_first, p.res_batched ? batch : 0);
        }
        res_ready = true;
      }
      if (!dry) {
        bool got = mbar_wait_long(tfull0 + 8 * acc, aph, abort_ptr);
        if (!got && lane == 0 && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 3); *abort_ptr = 1; }
        ok = __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0 && !*abort_ptr;
        if (!ok) break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // SPLIT: the sums of the other pair's columns leave for its CTA with the same rows, those of this one's columns come from
      // there.  The rings are idle: one half of this CTA's is what it sends, the other half what it gets.
      [[maybe_unused]] const uint32_t recv_bar = smem_u32(&bars[kBarRecv + e]);
      [[maybe_unused]] const uint32_t recv_area = (uint32_t)(p.half_bn / 32 * 4 * 4096);
      if constexpr (SPLIT) {
        if (!dry) {
          const uint32_t other = cta ^ 2u;
          if (e == 0 && lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&bars[kBarPeer]), other));      // this CTA's ring may be written
          uint32_t coming = 0;
          for (int c = 32 * group; c < p.half_bn; c += 32 * kPairWarpsPerQuad)
            if (rows_ok && n0 + c_first + c < p.N) coming += 4096;
          if (lane == 0 && coming != 0) mbar_expect_tx(recv_bar, coming);
          const int c_other = p.half_bn - c_first;
          bool free = false;
#pragma unroll 1
          for (int c = 32 * group; c < p.half_bn; c += 32 * kPairWarpsPerQuad) {
            if (!rows_ok || n0 + c_other + c >= p.N) break;
            const uint32_t at = (uint32_t)((c / 32 * 4 + quad) * 4096);
            float v[32];
            tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c_other + c), v);
            uint8_t* const mine = smem_raw + (tiles - raw) + at;
            stage_rows(mine, mine, v, lane, false);
            fence_async_smem();
            __syncwarp();
            if (!free) {
              const bool got = mbar_wait_cluster(smem_u32(&bars[kBarPeer]), 0, abort_ptr);
              if (!got && lane == 0 && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 7); *abort_ptr = 1; }
              free = __all_sync(0xffffffffu, got ? 1 : 0) != 0;
              if (!free) break;
            }
            if (lane == 0) push_block(map_to_cta(tiles + recv_area + at, other), tiles + at, 4096, map_to_cta(recv_bar, other));
          }
        }
      }
#pragma unroll 1
      for (int j = 0; j < kPairBlocksPerWarp; ++j) {
        const int c = c_first + 32 * (group + kPairWarpsPerQuad * j);
        const int n = n0 + c;
        if (c >= c_end || !rows_ok || n >= p.N) break;          // uniform across the warp
        float mine = col_pre[0];
#pragma unroll
        for (int q = 1; q < kPairBlocksPerWarp; ++q)
          if (j == q) mine = col_pre[q];
        // the slot's last bulk stores have finished reading it
        if (lane == 0) store_wait_read(0);
        __syncwarp();
        // a full-matrix operand of the chain (residual, mask) is brought INTO the slot by a bulk tensor
        // load, under the tensor-memory load below
        if (has_res && !dry && !(j == 0 && res_ready) && lane == 0) {
          mbar_expect_tx(res_bar, 4096);
          tma_load_3d(slot0, &tma_res, res_bar, n, m_first, p.res_batched ? batch : 0);
        }
        if (EPI != EPI_CHAIN) columns[e][lane] = mine;
        else if (col_step >= 0 && scratch_off >= 0) reinterpret_cast<float*>(slot0_ptr + scratch_off)[lane] = mine;
        float v[32];
        tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * p.bn + c), v);
        __syncwarp();
        if constexpr (SPLIT) {
          if (!dry) {
            const bool got = mbar_wait_cluster(recv_bar, 0, abort_ptr);
            if (!got && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 6); *abort_ptr = 1; }
            __syncwarp();
            const uint8_t* const theirs = smem_raw + (tiles - raw) + recv_area + ((c - c_first) / 32 * 4 + quad) * 4096;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float4 t = *reinterpret_cast<const float4*>(theirs + lane * 128 + ((q ^ (lane & 7)) << 4));
              const float2 a = fadd2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(t.x, t.y));
              const float2 b = fadd2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(t.z, t.w));
              v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = b.x; v[4 * q + 3] = b.y;
            }
          }
        }
        if constexpr (EPI == EPI_CHAIN) {
          run_chain(v, mine, n, batch);
        } else {
#pragma unroll
          for (int q = 0; q < 8; ++q) {        // every lane reads the same 16 bytes: a broadcast
            const float4 t = *reinterpret_cast<const float4*>(&columns[e][4 * q]);
            const float2 a = fadd2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(t.x, t.y));
            const float2 b = fadd2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(t.z, t.w));
            v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = b.x; v[4 * q + 3] = b.y;
          }
          if constexpr (EPI == EPI_BIAS_GELU) {
            if (BF16) gelu_tanh_approx_pairs(v);
            else gelu_tanh_pairs(v);
          }
          if constexpr (EPI == EPI_BIAS_RES) {
            if (!dry) {
              bool landed = mbar_wait(res_bar, res_phase, abort_ptr);
              if (!landed && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | 5); *abort_ptr = 1; }
              res_phase ^= 1u;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float4 t = *reinterpret_cast<const float4*>(slot0_ptr + lane * 128 + ((q ^ (lane & 7)) << 4));
              const float2 a = fadd2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(t.x, t.y));
              const float2 b = fadd2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(t.z, t.w));
              v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = b.x; v[4 * q + 3] = b.y;
            }
          }
        }
        __syncwarp();
        stage_rows(slot0_ptr, slot0_ptr + (with32 || has_res ? 4096 : 0), v, lane, with16, with32);
        fence_async_smem();
        __syncwarp();
        if (lane == 0 && !dry) {
          if (with32) tma_store_3d(&tma_out, slot0, n, m_first, batch, out_policy);
          if (with16) tma_store_3d(&tma_out16, slot0 + (with32 || has_res ? 4096u : 0u), n, m_first, batch);
          tma_store_commit();
        }
        if (dry) break;
      }
      if (dry) {
        dry = false;
        continue;
      }
      // this warp has read the accumulator: hand it back to the leader's MMA thread
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(tempty_leader0 + 8 * acc);
      tile += num_pairs;
      ++i;
    }
    if (lane == 0) store_wait_read(0);   // shared memory must outlive the stores that read it
  }

  // ---------------- common exit ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) let_copies_land();
  // neither CTA leaves (or frees TMEM the other's MMAs write) before both are done
  cluster_arrive_relaxed();
  cluster_wait();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
  }
}

using PairKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, PairParams);

template <bool BF16, int KPS, bool SPLIT>
PairKernel pair_kernel(int epilogue) {
  switch (epilogue) {
    case EPI_BIAS: return mm_pair_kernel<BF16, KPS, EPI_BIAS, SPLIT>;
    case EPI_BIAS_GELU: return mm_pair_kernel<BF16, KPS, EPI_BIAS_GELU, SPLIT>;
    case EPI_BIAS_RES: return mm_pair_kernel<BF16, KPS, EPI_BIAS_RES, SPLIT>;
    default: return mm_pair_kernel<BF16, KPS, EPI_CHAIN, SPLIT>;
  }
}

int epilogue_of(const PairParams& p) {
  const PairStep* s = p.steps;
  const bool bias = p.n_steps >= 1 && s[0].op == CH_ADD && s[0].kind == SIDE_COL;
  if (p.n_steps == 1 && bias) return EPI_BIAS;
  if (p.n_steps == 2 && bias && (s[1].op == CH_GELU_TANH || s[1].op == CH_GELU_TANH_APPROX)) return EPI_BIAS_GELU;
  if (p.n_steps == 2 && bias && s[1].op == CH_ADD && s[1].kind == SIDE_RES) return EPI_BIAS_RES;
  return EPI_CHAIN;
}

struct PairState {
  CUtensorMap map_a, map_b, map_out, map_out16, map_res;
  PairParams params;
  size_t smem_bytes = 0;
  dim3 grid;
  bool bf16 = false;
  bool split = false;      // clusters of two pairs, half of K each
  PairKernel kernel = nullptr;
};

// The chain step operands the epilogue can take: immediates, unary ops, per-column vectors readable
// with 128-bit loads, and at most one full matrix that a bulk tensor load can describe.
bool classify_steps(const PlanKernel& k, PairParams* p, const DevOperand** res_operand) {
  int n_res = 0;
  if (p) { p->res_step = -1; p->n_steps = k.chain.n; }
  for (int s = 0; s < k.chain.n; ++s) {
    const ChainStep& cs = k.chain.steps[s];
    PairStep ps{};
    ps.op = cs.op;
    ps.imm = cs.imm;
    if (cs.slot == -1) {
      ps.kind = SIDE_IMM;
    } else if (cs.slot < 0) {
      ps.kind = SIDE_NONE;
    } else {
      const DevOperand& o = k.ops[cs.slot];
      if (o.stride[1] == 0 && o.stride[2] == 1 && o.stride[0] % 4 == 0 && aligned16(o.ptr)) {
        ps.kind = SIDE_COL;
        ps.ptr = o.ptr;
        ps.batch_stride = o.stride[0];
      } else if (o.stride[2] == 1 && o.stride[1] >= k.N && o.stride[1] % 4 == 0 && o.stride[0] % 4 == 0 && o.stride[0] >= 0 &&
                 aligned16(o.ptr) && ++n_res == 1) {
        ps.kind = SIDE_RES;
        if (p) { p->res_step = s; p->res_batched = (k.batch > 1 && o.stride[0] != 0) ? 1 : 0; }
        if (res_operand) *res_operand = &o;
      } else {
        return false;
      }
    }
    if (p) p->steps[s] = ps;
  }
  return true;
}

}  // namespace

namespace {

// SM pairs this plan counts on: with several plans in flight (plan option CONCURRENCY) each takes its share.
int pair_share(const Plan& plan) {
  const int pairs = plan.sm_count / 2, share = plan.concurrency > 1 ? pairs / plan.concurrency : pairs;
  return share > 0 ? share : 1;
}

struct PairPlan { int bn; bool split; int64_t cycles; };

// Clusters of two pairs that fit the GPU at once.
int resident_quads(const Plan& plan) {
  int& known = plan.resident_quads;
  if (known == 0) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(plan.sm_count / 4 * 4), 1, 1);
    cfg.blockDim = dim3(kPairThreads, 1, 1);
    cfg.dynamicSmemBytes = kPairSmemCeiling;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 4;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const PairKernel kernel = mm_pair_kernel<true, 1, EPI_BIAS, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemCeiling) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known = n > 0 ? n : -1;
  }
  return known;
}

// Tile width and estimated cycles of a launch: 6700 once, and per round of tiles its drain and the cycles of its slabs, more of them the
// more of the pairs are at work (one SM gets 60 to 75 bytes a clock from L2; a slab of 256 columns has 512 cycles of multiplying).
// K in halves: the exchange and its own start instead.  Lines through 512 launches in TF32 and BF16, every width and both
// forms of each timed: 160 to 4096 rows of sixteen weights from 256 x 1024 to 4096 x 4096.  The choice is 0.1 % from the best on average,
// with the lines of the epilogue that released over the cluster it was 0.2 %, and against the few-tiles kernel 0.8
// and 0.5 % (TF32, BF16; 1024 x 2304 x 768 BF16 10.2 against 9.5 us, 256 x 4096 x 1000 TF32 10.6 against 9.7).
// The widths between 128 and 256 are for the last round: 2048 x 3072 x 768 TF32 21.2 us at 128 columns (three rounds, 64 of 74 pairs),
// 23.5 at 256 (96 tiles), 19.5 at 192 (128 tiles, two rounds); 8192 x 768 x 3072 BF16 66.2 at 256, 59.5 at 192 (with its pass
// over A); 8192 x 2304 x 768 36.1 at 256, 39.7 at 192.
struct PairWidth {
  int bn;
  int alone, full;                     // cycles of a slab with one pair at work | with all of them
  int drain;                           // of a round
  int half_alone, half_full, halves;   // K in halves: cycles of a slab, and of all that runs once (0: this width does not come in halves)
};
constexpr PairWidth kPairWidths[] = {
    {256, 490, 607, 3960, 505, 683, 12080}, {224, 430, 552, 3460, 0, 0, 0}, {192, 362, 485, 2730, 383, 496, 9970}, {160, 304, 412, 2570, 0, 0, 0}, {128, 256, 387, 2080, 0, 0, 0}};
constexpr int64_t kPairOnce = 6700, kPairHalvesBusy = 1860;      // (halves: with all pairs at work)
// A matrix operand of the epilogue arrives under the exchange of halves; without one it adds to the drain.  Of 156 launches with a
// residual behind another kernel, widths and halves of each timed, the choice is then 0.06 us from the best on average, 0.19 without
// (1400 x 768 x 768 TF32 15.5 us at 128 columns, 15.2 in halves; 1400 x 1024 x 4096 BF16 34.3 and 32.1).
constexpr int64_t kPairMatrixOperand = 1500;

int64_t slabs_of(const PlanKernel& k) {
  const int slab_k = k.desc.precision == KB200_PREC_BF16 ? 64 : 32;
  return (k.K + slab_k - 1) / slab_k;
}
int64_t tiles_of(const PlanKernel& k, const PairWidth& w) { return ((k.M + 255) / 256) * ((k.N + w.bn - 1) / w.bn) * k.batch; }
bool width_fits(const PlanKernel& k, const PairWidth& w, bool b_kmajor) {
  const int chunk_n = k.desc.precision == KB200_PREC_BF16 ? 64 : 32;      // an N-major B comes in whole chunks of columns
  return !(w.bn > 128 && w.bn / 2 >= k.N) && (b_kmajor || w.bn / 2 % chunk_n == 0);
}
// (one slab per step: what a step costs on its own shows where it multiplies for less)
int64_t one_slab(const PairWidth& w, bool two_slabs) { return w.bn == 128 && !two_slabs ? 125 : 0; }

// A launch that has the GPU to itself.  What decides the order of a matmul's sums -- whether K goes in halves, and by these cycles
// whether another kernel runs it -- is said here, by its shape and the GPU alone: results must not depend on plans in flight.
PairPlan plan_pair(const Plan& plan, const PlanKernel& k, bool two_slabs, bool b_kmajor) {
  const int64_t share = plan.sm_count / 2, slabs = slabs_of(k);
  const DevOperand* matrix = nullptr;
  classify_steps(k, nullptr, &matrix);
  const int64_t once = kPairOnce + (matrix != nullptr ? kPairMatrixOperand : 0);
  PairPlan best{0, false, 0};
  int64_t least = 0;                    // what `best` is compared by
  for (const PairWidth& w : kPairWidths) {
    if (!width_fits(k, w, b_kmajor)) continue;
    const int64_t tiles = tiles_of(k, w), rounds = (tiles + share - 1) / share;
    int64_t cycles = once + rounds * (slabs * (w.alone + one_slab(w, two_slabs)) + w.drain) + slabs * (w.full - w.alone) * tiles / share;
    // (Beyond ~80 us the GPU is at its power limit, where the bytes a tile moves for its work count: 4096^3 TF32 191 us at 256 columns, 201 at 192.)
    if (cycles > 150000) cycles += cycles * (256 - w.bn) / 2560;
    if (best.bn == 0 || cycles < least) best = {w.bn, false, cycles}, least = cycles;
    // K in halves on twice the pairs
    if (w.halves == 0 || slabs < 8 || 2 * tiles > share || tiles > resident_quads(plan)) continue;
    const int64_t halved = w.halves + (slabs + 1) / 2 * w.half_alone + ((slabs + 1) / 2 * (w.half_full - w.half_alone) + kPairHalvesBusy) * 2 * tiles / share;
    // (Of two that cost alike by the lines halves move fewer bytes: 1900 x 960 x 3840 TF32 25.8 us at 128 columns with its operands in L2 and up to 31
    // behind another matmul, 25.8 and 26.4 in halves of 256.  Of 264 launches of 300 to 3600 rows with 64 slabs and more, ten go by it, TF32 of 3840 and BF16 of
    // 7680 of K: 2 to 24 % less time each, 11 % on average.)
    const int64_t as = slabs < 64 ? halved : halved * 49 / 50;
    if (as < least) best = {w.bn, true, halved}, least = as;
  }
  return best;
}

// Tile width of a launch that shares the GPU, K in one go: any of them gives the same bits.  A plan with its share of the SM pairs goes
// by rounds of those.  Where other plans run beside it on all of them, they fill its last round, so the work of its tiles counts, and the
// tile that moves least for its work also takes the least power (the step of 64 contexts, eight modules in flight: 1377 us by
// rounds, mostly 192 columns, 1352 with 256).  The last drain is charged only where tiles do not cover the pairs, each has one
// and nothing to run under it: 2048 x 2304 x 768 TF32, four modules, 13.5 us at 192 columns (48 pairs, two tiles each), 14.4 at 256 (72 pairs); K = 256 7.8 and 9.8.
int width_in_flight(const Plan& plan, const PlanKernel& k, bool two_slabs, bool b_kmajor) {
  const int64_t share = pair_share(plan), slabs = slabs_of(k);
  int best = 0;
  int64_t least = 0;
  for (const PairWidth& w : kPairWidths) {
    if (!width_fits(k, w, b_kmajor)) continue;
    const int64_t tiles = tiles_of(k, w), slab = w.full + one_slab(w, two_slabs);
    const bool by_work = plan.others_in_flight && plan.concurrency == 1 && tiles >= share;
    const int64_t cycles = by_work ? tiles * slabs * slab / share : (tiles + share - 1) / share * slabs * slab + w.drain;
    if (best == 0 || cycles < least) best = w.bn, least = cycles;
  }
  return best;
}

}  // namespace

// (in the few-tiles kernel's cycles, which its estimate counts at 1.65 to the ns, this one's at 1.86: of 281 launches the choice is then 0.1 % (TF32)
// and 0.3 % (BF16) from the better kernel.  A GELU in float32 costs this kernel's last
// tile 0.9 us, that one's, spread over more warps, 0.55: 1002 x 1024 x 256 6.55 and 6.15, without it 5.5 both.  Of 140 TF32 launches with a GELU, 200 to 1700 rows, 17 go by it, K of 512
// and 768: 4 to 10 % less time each.)
int64_t pair_cycles(const Plan& plan, const PlanKernel& k, bool b_kmajor) {
  const bool gelu = k.desc.precision == KB200_PREC_TF32 && k.chain.n > 0 && k.chain.steps[k.chain.n - 1].op == CH_GELU_TANH;
  return (plan_pair(plan, k, true, b_kmajor).cycles + (gelu ? 700 : 0)) * 8 / 9;
}

bool pair_eligible(const Plan& plan, const PlanKernel& k, bool b_kmajor, int64_t b_cols) {
  const kb200_kernel_desc& d = k.desc;
  if (d.precision == KB200_PREC_FP32 || !k.has_chain) return false;
  if (d.cfg[0] == 128) return false;                       // the tuner asked for single-CTA tiles
  if (k.M <= 128 && d.cfg[0] != 256) return false;
  if (plan.sm_count < 2) return false;
  const bool bf16 = d.precision == KB200_PREC_BF16;
  const int chunk_n = bf16 ? 64 : 32;
  if (k.N < 128 || k.N % 4 || (!b_kmajor && b_cols % chunk_n)) return false;
  if (d.cfg[4] > 1) return false;                          // a forced split-K runs on the single-CTA kernel
  if (d.cfg[7] == 1 || d.cfg[7] == 2) return false;        // so do its epilogue variants
  if (((k.M + 255) / 256) * ((k.N + 127) / 128) * k.batch >= (int64_t(1) << 20)) return false;
  // bulk tensor stores: column-contiguous output, 16-byte aligned base and strides
  const DevOperand& O = k.ops[k.chain.out_slot];
  if (O.stride[2] != 1 || O.stride[1] % 4 || O.stride[1] < k.N || !aligned16(O.ptr)) return false;
  if (k.batch > 1 && (O.stride[0] % 4 || O.stride[0] <= 0)) return false;
  return classify_steps(k, nullptr, nullptr);
}

int pair_bind(Plan& plan, PlanKernel& k, int kernel_index, const PairOperands& ops, void** state) {
  const kb200_kernel_desc& d = k.desc;
  *state = nullptr;
  const DevOperand& O = k.ops[k.chain.out_slot];
  __nv_bfloat16* out16 = static_cast<__nv_bfloat16*>(k.shadow_out);
  if (out16 != nullptr && (O.stride[1] % 8 || (k.batch > 1 && O.stride[0] % 8) || !aligned16(out16))) return KB200_OK;
  PairState* st = new PairState();
  PairParams& p = st->params;
  const DevOperand* res = nullptr;
  if (!classify_steps(k, &p, &res)) { delete st; return KB200_OK; }
  st->bf16 = ops.bf16;
  if (ops.bf16)
    for (int s = 0; s < p.n_steps; ++s) {
      if (p.steps[s].op == CH_TANH) p.steps[s].op = CH_TANH_APPROX;
      else if (p.steps[s].op == CH_GELU_TANH) p.steps[s].op = CH_GELU_TANH_APPROX;
    }
  const int slab_k = ops.bf16 ? 64 : 32, chunk_n = ops.bf16 ? 64 : 32;
  // Tile width by the cost model above; K slabs per pipeline step below.
  int bn = d.cfg[1] == 128 || d.cfg[1] == 256 ? d.cfg[1] : 0;
  int kps = d.cfg[2] == 1 || d.cfg[2] == 2 ? d.cfg[2] : 0;
  const int share = pair_share(plan);
  const int64_t slabs = (k.K + slab_k - 1) / slab_k;
  if (bn == 0) {
    const PairPlan how = plan_pair(plan, k, kps != 1, ops.b_kmajor);
    st->split = how.split && d.cfg[3] == 0 && kps != 2;
    bn = st->split || (plan.concurrency == 1 && !plan.others_in_flight) ? how.bn : width_in_flight(plan, k, kps != 1, ops.b_kmajor);
  }
  while (bn == 256 && bn / 2 >= k.N) bn /= 2;
  // Staging per epilogue warp: one slot for a 32 x 32 block, float32 (also where a matrix operand of
  // the chain lands; left out when only the mirror is stored) and its bf16 copy.
  const bool store32 = !(k.mirror_only && out16 != nullptr);
  const int slot_bytes_wanted = ((store32 || p.res_step >= 0) ? 4096 : 0) + (out16 ? 2048 : 0);
  // two slabs per step where the ring still has three stages beside the staging slots
  if (kps == 0)
    kps = bn <= 128 && slabs >= 4 && 3 * 2 * (kPairATileBytes + bn / 2 * 128) + kPairEpiWarps * slot_bytes_wanted + 1024 <= kPairSmemCeiling ? 2 : 1;
  p.bn = bn;
  p.half_bn = bn / 2;
  p.slab_k = slab_k;
  p.kps = kps;
  p.step_k = kps * slab_k;
  p.num_kb = (int)((k.K + p.step_k - 1) / p.step_k);
  p.first_kb = (p.num_kb + 1) / 2;
  p.b_kmajor = ops.b_kmajor ? 1 : 0;
  p.b_static = ops.b_static ? 1 : 0;
  p.chunk_n = chunk_n;
  p.b_lbo_bytes = (uint32_t)(p.step_k * 128);              // N-major: bytes between the column chunks of a stage
  p.b_sbo_bytes = ops.bf16 ? 1024 : 512;
  // An N-major operand of 32-bit elements uses the 128-byte swizzle on 32-byte atoms (pattern of 4 rows);
  // 16-bit elements the ordinary 128-byte swizzle (8 rows).
  p.b_layout = ops.bf16 ? 2 : 1;
  p.b_step16 = ops.b_kmajor ? 2u : (uint32_t)((ops.bf16 ? 16 : 8) * 128) >> 4;
  p.b_slab16 = ops.b_kmajor ? (uint32_t)(p.half_bn * 128) >> 4 : 4u * p.b_step16;
  const uint32_t fmt = ops.bf16 ? 1u : 2u;
  // instruction descriptor: D = F32, A/B = BF16 or TF32, A K-major, B as bound, N = bn, M = 256 over the pair
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((ops.b_kmajor ? 0u : 1u) << 16) | ((uint32_t)(bn >> 3) << 17) | ((256u >> 4) << 24);
  p.tmem_cols = 32;
  while (p.tmem_cols < 2 * bn) p.tmem_cols *= 2;
  p.tiles_n = (int)((k.N + bn - 1) / bn);
  const int tiles_m = (int)((k.M + 255) / 256);
  p.tiles_per_batch = tiles_m * p.tiles_n;
  p.num_tiles = p.tiles_per_batch * (int)k.batch;
  p.magic_tn = ((uint64_t(1) << 40) + p.tiles_n - 1) / p.tiles_n;
  p.magic_tpb = ((uint64_t(1) << 40) + p.tiles_per_batch - 1) / p.tiles_per_batch;
  p.kernel_index = kernel_index;
  p.status = plan.d_status;
  p.M = k.M;
  p.N = k.N;
  p.out16 = out16;
  p.store32 = store32 ? 1 : 0;
  p.stream_out = streams_out(plan, k, k.chain.out_slot, k.batch * k.M * k.N) ? 1 : 0;
  p.slot_bytes = slot_bytes_wanted;
  p.slots = 1;
  const int stage_bytes = kps * (kPairATileBytes + p.half_bn * 128);
  const int epi_bytes = kPairEpiWarps * p.slot_bytes;
  int stages = d.cfg[3] > 0 ? d.cfg[3] : kPairMaxStages;
  if (stages > kPairMaxStages) stages = kPairMaxStages;
  while (stages > 2 && (size_t)stages * stage_bytes + epi_bytes + 1024 > (size_t)kPairSmemCeiling) --stages;
  if ((size_t)stages * stage_bytes + epi_bytes + 1024 > (size_t)kPairSmemCeiling) { delete st; return KB200_OK; }
  if (stages * stage_bytes < 2 * p.half_bn * 128 * 4) st->split = false;       // (what is sent and what is received lie in the ring)
  p.stages = stages;
  st->smem_bytes = (size_t)stages * stage_bytes + epi_bytes + 1024;
  // Persistent pairs: as many as there are tiles, up to this plan's share of the GPU.  With several
  // plans in flight a kernel that spread one tile to every pair would leave each pair's tensor cores
  // idle through its epilogue (bound by the store path, longer than the main loop at K = 768); on its
  // share of the pairs every pair walks several tiles and drains one while it multiplies the next.
  const int rounds = (p.num_tiles + share - 1) / share;
  const int n_pairs = (p.num_tiles + rounds - 1) / rounds;
  st->grid = dim3((unsigned)(st->split ? 4 * p.num_tiles : 2 * n_pairs), 1, 1);

  bool ok = encode_map(&st->map_a, ops.bf16, ops.a_base, k.K, k.M, k.batch, ops.a_row, ops.a_batch, slab_k, 128, false);
  if (ok) {
    if (ops.b_kmajor)
      ok = encode_map(&st->map_b, ops.bf16, ops.b_base, k.K, k.N, k.batch, ops.b_row, ops.b_batch, slab_k, p.half_bn, false);
    else
      ok = encode_map4(&st->map_b, ops.bf16, ops.b_base, chunk_n, k.K, ops.b_cols / chunk_n, k.batch, ops.b_row, ops.b_batch, p.step_k,
                       p.half_bn / chunk_n, !ops.bf16);
  }
  if (ok) ok = encode_map_store(&st->map_out, false, O.ptr, k.N, k.M, k.batch, O.stride[1], O.stride[0]);
  st->map_out16 = st->map_out;
  st->map_res = st->map_out;
  if (ok && out16) ok = encode_map_store(&st->map_out16, true, out16, k.N, k.M, k.batch, O.stride[1], O.stride[0]);
  if (ok && res) ok = encode_map_store(&st->map_res, false, res->ptr, k.N, k.M, p.res_batched ? k.batch : 1, res->stride[1], res->stride[0]);
  if (!ok) { delete st; return KB200_OK; }
  const int epilogue = epilogue_of(p);
  if (st->split) st->kernel = ops.bf16 ? pair_kernel<true, 1, true>(epilogue) : pair_kernel<false, 1, true>(epilogue);
  else if (kps == 2) st->kernel = ops.bf16 ? pair_kernel<true, 2, false>(epilogue) : pair_kernel<false, 2, false>(epilogue);
  else st->kernel = ops.bf16 ? pair_kernel<true, 1, false>(epilogue) : pair_kernel<false, 1, false>(epilogue);
  cudaError_t e = cudaFuncSetAttribute(st->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemCeiling);
  if (e != cudaSuccess) { delete st; return cuda_fail(e, "cudaFuncSetAttribute(mm_pair_kernel)"); }
  *state = st;
  return KB200_OK;
}

int pair_launch(const Plan& plan, const void* state, cudaStream_t s) {
  const PairState* st = static_cast<const PairState*>(state);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = st->grid;
  cfg.blockDim = dim3(kPairThreads, 1, 1);
  cfg.dynamicSmemBytes = st->smem_bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  attr[n_attr].id = cudaLaunchAttributeClusterDimension;
  attr[n_attr].val.clusterDim.x = st->split ? 4 : 2;
  attr[n_attr].val.clusterDim.y = 1;
  attr[n_attr].val.clusterDim.z = 1;
  ++n_attr;
  if (plan.pdl) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  KB200_CUDA(cudaLaunchKernelEx(&cfg, st->kernel, st->map_a, st->map_b, st->map_out, st->map_out16, st->map_res, st->params));
  KB200_CUDA(cudaGetLastError());
  return KB200_OK;
}

bool pair_repoint(const PlanKernel& k, void* state, const void* a, const void* b) {
  PairState* st = static_cast<PairState*>(state);
  bool ok = (!a || set_map_address(&st->map_a, a)) && (!b || set_map_address(&st->map_b, b)) &&
            set_map_address(&st->map_out, k.ops[k.chain.out_slot].ptr);
  for (int s = 0; s < st->params.n_steps && ok; ++s) {
    const int slot = k.chain.steps[s].slot;
    if (st->params.steps[s].kind == SIDE_COL) st->params.steps[s].ptr = k.ops[slot].ptr;
    if (st->params.steps[s].kind == SIDE_RES) ok = set_map_address(&st->map_res, k.ops[slot].ptr);
  }
  return ok;
}

std::string pair_detail(const void* state) {
  const PairState* st = static_cast<const PairState*>(state);
  return "mm_pair " + std::to_string(st->params.bn) + " columns, " + std::to_string(st->params.kps) + " slabs" + (st->split ? ", 2 splits" : "");
}

void pair_destroy(void* state) { delete static_cast<PairState*>(state); }

}  // namespace kb200
