// Fused causal attention in exact FP32 on float16 pairs: QK^T -> online softmax -> PV with float32 products, each of three float16 ones
// (x 2^e = h + 2^-11 t, see split_rows.cu; the probabilities are split here, times 2^14).  Role, items, pipeline and the softmax of two threads
// a row are attention_kernel's (attention.cu); what differs:
//   * Q, K and V come as two planes of float16 under a power of two per head, whose bound the plan knows (see result_bounds); both fit
//     shared memory twice, where the TF32 form's heads and tails fit once, and multiply at twice the rate;
//   * a group's probabilities lie over its own 64 scores, 32 columns of heads and 32 of tails, so both S buffers carry them;
//   * the tensor core cuts off a bit of an accumulator with every MMA: sums in it are over 64 keys (the head dimension in Q K^T), small
//     products first, and everything beyond is added up in float32 registers.
// From float64, merged heads of 12 heads: 1024 tokens 2.1e-7 (TF32 1.8e-6, the CUDA cores 2.6e-7), 2048 tokens 2.1e-7 (1.8e-6, 3.3e-7), 200 tokens
// 2.8e-7 (1.0e-6, 2.6e-7); with the projection's error, four seeds: 129 tokens 2.4e-7 (CUDA cores 2.1e-7), 333 2.7e-7 (2.5e-7), 512 2.7e-7 (2.6e-7), 1024
// 2.8e-7 (2.9e-7): what four MMAs of 16 dims cut off a score.  So it takes sequences of any length, which the TF32 form left to the CUDA cores: 12 heads of 1500 tokens
// 126 -> 25 us, of 333 tokens 18.1 -> 11.3 with the pass, 96 heads of 1024 tokens 128 (TF32) -> 53.  What bounds a tile is the softmax warps (a score costs
// them a maximum, an exponential, four conversions and their stores) beside 36 MMAs of ~50 cycles of issue.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "attention.h"
#include "attention_softmax.cuh"
#include "device_math.cuh"
#include "kb200_internal.h"
#include "split16.cuh"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"

namespace kb200 {

namespace {

using namespace tc;

constexpr int kPairsPlane = kAttnRows * 128;            // [128 rows x 64 dims] of heads, or of tails
constexpr int kPairsTile = 2 * kPairsPlane;
constexpr int kPairsSlot = 4096;                        // a warp's output block of 32 x 32
constexpr int kPairsExchange = 2 * (2 * 2 * kAttnRows * 4);
constexpr int kPairsSmem = 5 * kPairsTile + kPairsExchange + 8 * kPairsSlot + 1024;
constexpr int kPairsThreads = 320;
constexpr float kPairsUp = 16384.0f;                    // probabilities are at most 1: times 2^14.  (Not in the exponent, whose fraction would lose four bits.)

struct PairsParams {
  AttnParams a;
  const float* qk;          // by head: what a product of Q and K is to be multiplied by, times scale x log2(e)
  const float* v_back;      // ... and one with V, the probabilities' 2^14 included
  const float* out_scale;   // pairs of the merged heads leave as well, times *out_scale, through map_outh and map_outt; or null
  int store32;
};

// Probabilities of 32 keys as packed pairs: heads and tails of keys 2 i and 2 i + 1.
__device__ __forceinline__ void split_probabilities(const float (&v)[32], uint32_t* heads, uint32_t* tails) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float2 x = fmul2(make_float2(v[2 * i], v[2 * i + 1]), make_float2(kPairsUp, kPairsUp));
    const __half2 h = __floats2half2_rn(x.x, x.y);
    const float2 back = __half22float2(h);
    const float2 rest = ffma2(back, make_float2(-kTailUp, -kTailUp), fmul2(x, make_float2(kTailUp, kTailUp)));
    const __half2 t = __floats2half2_rn(rest.x, rest.y);
    heads[i] = *reinterpret_cast<const uint32_t*>(&h);
    tails[i] = *reinterpret_cast<const uint32_t*>(&t);
  }
}

__device__ __forceinline__ void tmem_st32u(uint32_t taddr, const uint32_t (&v)[32]) {
  float f[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]);
  tmem_st32(taddr, f);
}

template <bool SPLIT>
__global__ void __launch_bounds__(kPairsThreads, 1)
attention_pairs_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                       const __grid_constant__ CUtensorMap map_qt, const __grid_constant__ CUtensorMap map_kt, const __grid_constant__ CUtensorMap map_vt,
                       const __grid_constant__ CUtensorMap map_out, const __grid_constant__ CUtensorMap map_outh, const __grid_constant__ CUtensorMap map_outt,
                       const __grid_constant__ PairsParams params) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[20];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int arrived[4];                  // split items: was this lane quadrant's half the second to arrive?
  const AttnParams& p = params.a;
  constexpr int kRowsOf = kAttnRows;

  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t q_smem = (raw + 1023u) & ~1023u;
  const uint32_t k_smem = q_smem + kPairsTile, v_smem = k_smem + 2 * kPairsTile;      // rings of two tiles
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // bars: 0 q_full | 1,2 k_full | 3,4 k_empty | 5,6 v_full | 7,8 v_empty | 9,10 s_full | 11..14 p_full[group][s buffer] | 15,16 o_full[o buffer] | 19 q_empty
  const uint32_t q_full = smem_u32(&bars[0]), k_full = smem_u32(&bars[1]), k_empty = smem_u32(&bars[3]);
  const uint32_t v_full = smem_u32(&bars[5]), v_empty = smem_u32(&bars[7]);
  const uint32_t sfull0 = smem_u32(&bars[9]), pfull0 = smem_u32(&bars[11]), ofull0 = smem_u32(&bars[15]);
  const uint32_t q_empty = smem_u32(&bars[19]);
  const int n_items = p.B * p.H * (p.q_tiles + (SPLIT ? p.q_tiles - p.split_from : 0));

  if (threadIdx.x == 32) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    prefetch_tensormap(&map_qt);
    prefetch_tensormap(&map_kt);
    prefetch_tensormap(&map_vt);
    prefetch_tensormap(&map_out);
    prefetch_tensormap(&map_outh);
    prefetch_tensormap(&map_outt);
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < 20; ++i) mbar_init(q_full + 8 * i, i >= 11 && i < 15 ? 128 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // Everything above overlapped the previous kernel's tail; Q, K and V are its output.
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t tmem_base = tmem_base_slot;
  // columns: S0 0..127 | S1 128..255 | O_part[buffer][group] 256 + (2 buffer + group) 64
  const uint32_t tmem_o0 = tmem_base + 256;
  volatile int* abort_ptr = &abort_flag;
  auto give_up = [&](int site) {
    if (!*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | site); *abort_ptr = 1; }
  };
  // A whole warp walks each of the two roles below, one lane issuing (see elect_one); its waits end for all
  // lanes or none.
  auto all_waited = [&](bool got, int site) {
    if (!got && lane == 0) give_up(site);
    return __all_sync(0xffffffffu, got ? 1 : 0) != 0;
  };
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    int t = 0;                                     // key tiles loaded so far, over all items
    bool ok = true;
    auto load = [&](uint32_t dst, const CUtensorMap* heads, const CUtensorMap* tails, uint32_t bar, int token, int h, int seq) {
      if (elect_one()) {
        mbar_expect_tx(bar, kPairsTile);
        tma_load_4d(dst, heads, bar, 0, token, h, seq);
        tma_load_4d(dst + kPairsPlane, tails, bar, 0, token, h, seq);
      }
      __syncwarp();
    };
    for (int ii = 0; ok; ++ii) {
      const int w = attn_nth_item(ii, n_items);
      if (w < 0) break;
      const AttnItem it = attn_item<SPLIT>(p, w);
      // the Q tile is free once every Q K^T of the previous item has been executed
      if (!all_waited(mbar_wait(q_empty, (ii & 1) ^ 1, abort_ptr), 0x13)) break;
      load(q_smem, &map_q, &map_qt, q_full, it.q0, it.h, it.seq);
      for (int j = 0; j < it.n_kv; ++j, ++t) {
        const int s = t & 1;
        const uint32_t ph = (t >> 1) & 1;
        const int token = (it.j0 + j) * kRowsOf;
        if (!all_waited(mbar_wait(k_empty + 8 * s, ph ^ 1, abort_ptr), 0x11)) { ok = false; break; }
        load(k_smem + s * kPairsTile, &map_k, &map_kt, k_full + 8 * s, token, it.h, it.seq);
        if (!all_waited(mbar_wait(v_empty + 8 * s, ph ^ 1, abort_ptr), 0x12)) { ok = false; break; }
        load(v_smem + s * kPairsTile, &map_v, &map_vt, v_full + 8 * s, token, it.h, it.seq);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // Tiles are numbered over all items (t): ring slot, S buffer and O_part buffer are t & 1, phases (t >> 1) & 1.
    bool ok = true;
    auto issue_qk = [&](int t, bool last_of_item) {
      const int s = t & 1;
      ok = all_waited(mbar_wait(k_full + 8 * s, (t >> 1) & 1, abort_ptr), 0x22);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t kb = k_smem + s * kPairsTile;
      const uint32_t on = elect_one() ? 1u : 0u;
      // 32 bytes of the head dimension per instruction: tails x heads, heads x tails, heads x heads
#pragma unroll
      for (int pass = 0; pass < 3; ++pass) {
        const uint32_t qa = q_smem + (pass == 0 ? kPairsPlane : 0), ka = kb + (pass == 1 ? kPairsPlane : 0);
#pragma unroll
        for (int kd = 0; kd < 4; ++kd) {
          const uint64_t q_desc = make_desc(qa + kd * 32, 16, 1024), k_desc = make_desc(ka + kd * 32, 16, 1024);
          if (pass == 2 && kd == 0) umma_onto<kTailBits>(on, tmem_base + (uint32_t)s * 128, q_desc, k_desc, p.idesc_qk);
          else umma_if(on, tmem_base + (uint32_t)s * 128, q_desc, k_desc, p.idesc_qk, (pass | kd) != 0 ? 1u : 0u, true);
        }
      }
      if (on) {
        umma_commit(sfull0 + 8 * s);
        umma_commit(k_empty + 8 * s);
        if (last_of_item) umma_commit(q_empty);       // its last scores are issued: the Q tile is handed back
      }
      __syncwarp();
    };
    // P V of tile t, each group's 64 keys into an O_part of their own.  In-order execution of the tensor pipe keeps S[s] intact until these
    // reads of P are done (the next Q K^T into S[s] is issued later), and the buffers t & 1 were folded before P of tile t was published.
    auto issue_pv = [&](int t) {
      const int s = t & 1;
      const uint32_t ph = (t >> 1) & 1;
      ok = all_waited(mbar_wait(v_full + 8 * s, ph, abort_ptr), 0x23);
      if (!ok) return;
      const uint32_t vb = v_smem + s * kPairsTile;
      const uint32_t on = elect_one() ? 1u : 0u;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        ok = all_waited(mbar_wait(pfull0 + 8 * (g * 2 + s), ph, abort_ptr), 0x24);
        if (!ok) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t o_addr = tmem_o0 + (uint32_t)(s * 2 + g) * 64;
        // 16 keys = 8 columns of P and 16 128-byte rows of V per instruction
#pragma unroll
        for (int pass = 0; pass < 3; ++pass) {
          const uint32_t pa = tmem_base + (uint32_t)(s * 128 + g * 64 + (pass == 0 ? 32 : 0)), va = vb + (pass == 1 ? kPairsPlane : 0);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint64_t v_desc = make_desc(va + (uint32_t)(g * 4 + kk) * 2048, kPairsPlane, 1024, 2);
            if (pass == 2 && kk == 0) umma_ts_onto<kTailBits>(on, o_addr, pa, v_desc, p.idesc_pv);
            else umma_ts_if(on, o_addr, pa + (uint32_t)(kk * 8), v_desc, p.idesc_pv, (pass | kk) != 0 ? 1u : 0u, true);
          }
        }
      }
      if (on) {
        umma_commit(ofull0 + 8 * s);
        umma_commit(v_empty + 8 * s);
      }
      __syncwarp();
    };
    int t = 0;
    for (int ii = 0; ok; ++ii) {
      const int w = attn_nth_item(ii, n_items);
      if (w < 0) break;
      const int n_kv = attn_item<SPLIT>(p, w).n_kv;
      ok = all_waited(mbar_wait(q_full, ii & 1, abort_ptr), 0x21);
      if (!ok) break;
      issue_qk(t, n_kv == 1);
      for (int j = 0; j < n_kv && ok; ++j) {
        if (j + 1 < n_kv) issue_qk(t + j + 1, j + 2 == n_kv);      // the next scores are computed while the softmax warps work on tile j
        if (ok) issue_pv(t + j);
      }
      t += n_kv;
    }
  } else {
    // ---------------- softmax / output (warps 2..9): two threads share a query row, see attention.cu ----------------
    const int quad = warp & 3;
    const int group = (warp - 2) >> 2;
    const int row = quad * 32 + lane;              // row of the tile = TMEM lane
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const int c0 = group * 64;
    float* const xmax = reinterpret_cast<float*>(smem_raw + (v_smem - raw) + 2 * kPairsTile);
    float* const xsum = xmax + 4 * kRowsOf;
    uint8_t* const stage = reinterpret_cast<uint8_t*>(xmax) + kPairsExchange + (size_t)((warp - 2) * kPairsSlot);
    const int pair_barrier = 2 + quad;              // hardware barriers 2..5, 64 threads each
    // The pair's barrier also carries the abort flag (an OR over what the 64 threads read before they
    // arrived), so that both threads of a row take the same decision and neither waits for the other.
    auto pair_sync_aborted = [&]() {
      uint32_t any;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbar.red.or.pred q, %1, 64, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
          : "=r"(any)
          : "r"(pair_barrier), "r"((uint32_t)*abort_ptr)
          : "memory");
      return any != 0;
    };
    bool ok = true;
    int t0 = 0;                                      // tiles of the items before this one
    for (int ii = 0; ok; ++ii) {
      const int w = attn_nth_item(ii, n_items);
      if (w < 0) break;
      const AttnItem it = attn_item<SPLIT>(p, w);
      const int n_kv = it.n_kv;
      const float qk = __ldg(params.qk + it.h), v_back = __ldg(params.v_back + it.h);
      float o[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) o[i] = 0.0f;
      float m_run = -CUDART_INF_F, l_run = 0.0f, alpha_prev = 0.0f;
      // running output <- running output * alpha + this thread's 32 dims of the two O_parts of tile t
      auto fold = [&](int t, float alpha) {
        bool got = mbar_wait(ofull0 + 8 * (t & 1), (t >> 1) & 1, abort_ptr);
        if (!got) give_up(0x32);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float u[32], v[32];
        const uint32_t at = tmem_o0 + lane_addr + (uint32_t)((t & 1) * 128 + group * 32);
        tmem_ld32x2(at, at + 64, u, v);
        const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 r2 = ffma2(make_float2(o[i], o[i + 1]), alpha2, fadd2(make_float2(u[i], u[i + 1]), make_float2(v[i], v[i + 1])));
          o[i] = r2.x;
          o[i + 1] = r2.y;
        }
      };
      // Every thread of a pair passes the same barriers: a wait that ran out raises the CTA's flag and the
      // thread carries on to the next barrier, after which both see the flag and leave together.
      for (int j = 0; j < n_kv; ++j) {
        const int t = t0 + j;
        const int s = t & 1;
        const uint32_t ph = (t >> 1) & 1;
        if (!mbar_wait(sfull0 + 8 * s, ph, abort_ptr)) give_up(0x31);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t s_addr = tmem_base + lane_addr + (uint32_t)(s * 128 + c0);
        const bool diagonal = it.j0 + j == it.qt;
        float va[32], vb[32];
        tmem_ld32x2(s_addr, s_addr + 32, va, vb);       // both halves in flight, one wait
        // the scale is positive (checked when the chain was matched), so the maximum commutes with it
        float mx = -CUDART_INF_F;
        if (diagonal) {
          mx = row_max32<true>(va, mx, c0, row);
          mx = row_max32<true>(vb, mx, c0 + 32, row);
        } else {
          mx = row_max32<false>(va, mx, 0, 0);
          mx = row_max32<false>(vb, mx, 0, 0);
        }
        xmax[(s * 2 + group) * kRowsOf + row] = mx;
        if (pair_sync_aborted()) { ok = false; break; }
        mx = fmaxf(mx, xmax[(s * 2 + (group ^ 1)) * kRowsOf + row]);
        // the first key of every tile at or below the diagonal is visible to every row, so the maximum is finite
        const float m_new = fmaxf(m_run, mx * qk);
        const float alpha = ex2(m_run - m_new);       // 0 while m_run = -inf
        float sum;
        if (diagonal) {
          sum = probabilities32<true>(va, qk, m_new, c0, row);
          sum += probabilities32<true>(vb, qk, m_new, c0 + 32, row);
        } else {
          sum = probabilities32<false>(va, qk, m_new, 0, 0);
          sum += probabilities32<false>(vb, qk, m_new, 0, 0);
        }
        uint32_t heads[32], tails[32];
        split_probabilities(va, heads, tails);
        split_probabilities(vb, heads + 16, tails + 16);
        tmem_st32u(s_addr, heads);
        tmem_st32u(s_addr + 32, tails);
        tmem_st_wait();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(pfull0 + 8 * (group * 2 + s));
        // fold the PREVIOUS tile's O_parts while the tensor pipe works on this one
        if (j > 0) fold(t - 1, alpha_prev);
        alpha_prev = alpha;
        l_run = l_run * alpha + sum;
        m_run = m_new;
      }
      if (ok) fold(t0 + n_kv - 1, alpha_prev);
      t0 += n_kv;
      // ---- the row sum is the two threads' partial sums; thread g normalises and stores dims g*32 .. g*32+31 ----
      xsum[((ii & 1) * 2 + group) * kRowsOf + row] = l_run;
      if (pair_sync_aborted()) ok = false;
      // ---- a split item: as in attention_kernel ----
      bool writes = ok;
      float l_tot = ok ? l_run + xsum[((ii & 1) * 2 + (group ^ 1)) * kRowsOf + row] : 1.0f;
      if (SPLIT && ok && it.split) {
        float* const mine = p.partial + ((size_t)it.slot * 2 + it.half) * kAttnPartialFloats;
        const float* const other = p.partial + ((size_t)it.slot * 2 + (it.half ^ 1)) * kAttnPartialFloats;
#pragma unroll
        for (int i = 0; i < 32; ++i) __stcg(mine + (group * 32 + i) * kRowsOf + row, o[i]);
        if (group == 0) {
          __stcg(mine + kRowsOf * kAttnHeadDim + row, m_run);
          __stcg(mine + kRowsOf * kAttnHeadDim + kRowsOf + row, l_tot);
        }
        __threadfence();
        if (pair_sync_aborted()) ok = false;          // the quadrant's 64 threads have written and fenced
        if (ok) {
          if (lane == 0 && group == 0) {
            arrived[quad] = atomicAdd(p.arrivals + it.slot * 4 + quad, 1);
            __threadfence();
          }
          if (pair_sync_aborted()) ok = false;
        }
        if (ok) {
          writes = arrived[quad] != 0;
          if (writes) {
            if (lane == 0 && group == 0) p.arrivals[it.slot * 4 + quad] = 0;      // for the next launch
            const float m2 = __ldcg(other + kRowsOf * kAttnHeadDim + row), l2 = __ldcg(other + kRowsOf * kAttnHeadDim + kRowsOf + row);
            const float m = fmaxf(m_run, m2);
            const float a1 = ex2(m_run - m), a2 = ex2(m2 - m);
            // (rounded one by one and then added: symmetric in the two halves)
            l_tot = __fadd_rn(__fmul_rn(l_tot, a1), __fmul_rn(l2, a2));
#pragma unroll
            for (int i = 0; i < 32; ++i)
              o[i] = __fadd_rn(__fmul_rn(o[i], a1), __fmul_rn(__ldcg(other + (group * 32 + i) * kRowsOf + row), a2));
          }
        }
      }
      if (ok && writes) {
        const float inv = 1.0f / l_tot;
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = o[i] * v_back * inv;
        // A lane holds 32 dims of one row: through the warp's slot by bulk tensor stores (the maps end at the sequence's last row).
        const int col = it.h * kAttnHeadDim + group * 32, first_row = it.q0 + quad * 32;
        if (first_row < p.T) {
          if (params.store32) {
            if (lane == 0) tma_store_wait_read();          // the slot's last stores have read it
            __syncwarp();
            stage_rows(stage, stage, o, lane, false, true);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_3d(&map_out, smem_u32(stage), col, first_row, it.seq);
              tma_store_commit();
            }
          }
          if (params.out_scale != nullptr) {
            if (lane == 0) tma_store_wait_read();
            __syncwarp();
            stage_pairs(stage, o, lane, __ldg(params.out_scale));
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_3d(&map_outh, smem_u32(stage), col, first_row, it.seq);
              tma_store_3d(&map_outt, smem_u32(stage) + 2048, col, first_row, it.seq);
              tma_store_commit();
            }
          }
        }
      }
    }
    if (lane == 0) tma_store_wait_read();    // shared memory must outlive the stores that read it
  }

  // ---------------- common exit ----------------
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) let_copies_land();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Q, K and V as pairs, where the projection in front does not write them: rows of `n` floats, times scale[column / 32].
__global__ void __launch_bounds__(256) attention_pairs_pass(const float* __restrict__ src, int64_t s_row, __half* __restrict__ heads, int64_t plane, int64_t pitch,
                                                            const float* __restrict__ scale, uint32_t rows, uint32_t n4) {
  pdl_wait();                 // the producer of Q, K and V has completed
  pdl_launch_dependents();
  const uint32_t total = rows * n4;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t row = i / n4, c = (i - row * n4) * 4;
    __half* const at = heads + (int64_t)row * pitch + c;
    store_terms(at, at + plane, *reinterpret_cast<const float4*>(src + (int64_t)row * s_row + c), __ldg(scale + (c >> 5)));
  }
}

}  // namespace

}  // namespace kb200
