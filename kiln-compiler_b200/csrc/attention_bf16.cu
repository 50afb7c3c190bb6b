// Fused causal attention on bf16 operands for sm_100a (BF16 mode; the chain it stands for and how it is matched:
// attention.cu).  Q, K and V come from the bf16 mirror of the QKV projection's output.
//
// What bounds it: the special-function unit takes 16 exponentials a clock, 1024 cycles for the 128 x 128 scores of a
// tile, where the tensor cores need 512 for both products.  One query tile per SM cannot get near that:
// its warps all wait for the same scores, take the same exponentials and store the same probabilities at the same time, and
// the unit idles through every one of those latencies (~1950 cycles per tile, with 8 or 16 softmax
// warps alike).  So an SM holds TWO CTAs, each with a query tile of its own and half of the tensor memory:
// one's exponentials run under the other's latencies.  What that asks of a CTA:
//   * 256 columns of tensor memory: scores 0..127, probabilities (two bf16 a column) 128..191, output 192..255.  The scores are
//     in registers before the probabilities are written, so the next tile's Q K^T starts as soon as they were read.
//   * 168 registers a thread: one thread holds the 128 scores of a query row, and the output rows stay in tensor memory.  P V
//     accumulates there over the tiles of an item; a warp rescales its rows where the maximum of one of them has grown.  (Only
//     where it has grown by 2^8 would save 0.6 of 27.8 us, but the largest probability of a row would no longer be 1, which bf16
//     holds exactly: error 2.4e-4 -> 3.3e-4 for rows that a few keys dominate.  The sum over the rounded
//     probabilities mends that for 2.5 us more.)  Nothing crosses between threads: no barrier among the softmax warps.
//   * The tensor core cuts off what does not fit a sum, once per 16 keys, so a sum that only ever grew there would be short by
//     more the longer the sequence (values around 1, 16384 keys: 3.8e-5 short, error 6.1e-5; with rounded float32 additions 0.3e-5
//     and 5.4e-5).  An item of more than kAttnRun key tiles (LONG) is therefore finished as often, and each thread adds its row to
//     the one it keeps in a workspace of its CTA's in float32: 0.5e-5 and 5.4e-5, for 84.0 instead of 78.6 us at two
//     sequences of 4096 tokens and 12 heads.
//   * 112 KB of shared memory: two tiles each of Q, K and V, a 4 KB staging slot per softmax warp.
// 32-key blocks above the diagonal are not computed (3/8 of a diagonal tile's exponentials); an item's rows are finished behind
// the first exponentials of the next.  Eight sequences of 1024 tokens and 12 heads: 39.4 us with one query tile per SM, 27.5 now
// (the exponentials alone: 11.3); 2048 tokens of one sequence 22.6 -> 20.9, six sequences of 333 tokens 9.4 -> 8.5.
//
// 192 threads: warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 softmax, one per tensor-memory lane quadrant.  CTAs are
// persistent, items as in attention.cu.  Every wait is bounded (see matmul_tc.cu).
#include <algorithm>
#include <vector>

#include "attention.h"
#include "kb200_internal.h"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"

namespace kb200 {

namespace {

using namespace tc;

constexpr int kThreads = 64 + 128;
constexpr int kTile = kAttnRows * 128;       // [128 rows x 64 bf16], 128-byte swizzled
constexpr int kStage = 4096;                 // a warp's output rows: 32 x 32 float32 or 32 x 64 bf16
constexpr int kSmem = 6 * kTile + 4 * kStage;              // two CTAs of it, with 1 KB each of barriers and of the system's, are all an SM has
constexpr int kSmemAlone = 120 * 1024;       // ... one to an SM
constexpr uint32_t kColumns = 256, kColP = 128, kColO = 192;

// The 128 columns of this thread's lane: four loads in flight, one wait.  (As one load of 128 registers in a row it
// left the stores below no room for rows of their own: 82 registers spilled.)
__device__ __forceinline__ void tmem_ld128(uint32_t addr, float (&v)[128]) {
  uint32_t r[128];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%128];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%129];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%64, %65, %66, %67, %68, %69, %70, %71, %72, %73, %74, %75, %76, %77, %78, %79, %80, %81, %82, %83, %84, %85, %86, %87, %88, %89, %90, %91, %92, %93, %94, %95}, [%130];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%96, %97, %98, %99, %100, %101, %102, %103, %104, %105, %106, %107, %108, %109, %110, %111, %112, %113, %114, %115, %116, %117, %118, %119, %120, %121, %122, %123, %124, %125, %126, %127}, [%131];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63]),
        "=r"(r[64]), "=r"(r[65]), "=r"(r[66]), "=r"(r[67]), "=r"(r[68]), "=r"(r[69]), "=r"(r[70]), "=r"(r[71]),
        "=r"(r[72]), "=r"(r[73]), "=r"(r[74]), "=r"(r[75]), "=r"(r[76]), "=r"(r[77]), "=r"(r[78]), "=r"(r[79]),
        "=r"(r[80]), "=r"(r[81]), "=r"(r[82]), "=r"(r[83]), "=r"(r[84]), "=r"(r[85]), "=r"(r[86]), "=r"(r[87]),
        "=r"(r[88]), "=r"(r[89]), "=r"(r[90]), "=r"(r[91]), "=r"(r[92]), "=r"(r[93]), "=r"(r[94]), "=r"(r[95]),
        "=r"(r[96]), "=r"(r[97]), "=r"(r[98]), "=r"(r[99]), "=r"(r[100]), "=r"(r[101]), "=r"(r[102]), "=r"(r[103]),
        "=r"(r[104]), "=r"(r[105]), "=r"(r[106]), "=r"(r[107]), "=r"(r[108]), "=r"(r[109]), "=r"(r[110]), "=r"(r[111]),
        "=r"(r[112]), "=r"(r[113]), "=r"(r[114]), "=r"(r[115]), "=r"(r[116]), "=r"(r[117]), "=r"(r[118]), "=r"(r[119]),
        "=r"(r[120]), "=r"(r[121]), "=r"(r[122]), "=r"(r[123]), "=r"(r[124]), "=r"(r[125]), "=r"(r[126]), "=r"(r[127])
      : "r"(addr), "r"(addr + 32), "r"(addr + 64), "r"(addr + 96)
      : "memory");
#pragma unroll
  for (int i = 0; i < 128; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

// The largest of N scores of a row from the first-th on: eight chains of maxima at once.
template <int N>
__device__ __forceinline__ float row_max(const float (&v)[128], int first) {
  constexpr int kChains = N / 16 < 8 ? N / 16 * 2 : 8;
  float m[kChains];
#pragma unroll
  for (int q = 0; q < kChains; ++q) m[q] = fmaxf(v[first + 2 * q], v[first + 2 * q + 1]);
#pragma unroll
  for (int i = 2 * kChains; i < N; i += 2 * kChains)
#pragma unroll
    for (int q = 0; q < kChains; ++q) m[q] = fmax3(m[q], v[first + i + 2 * q], v[first + i + 2 * q + 1]);
#pragma unroll
  for (int n = kChains / 2; n >= 1; n /= 2)
#pragma unroll
    for (int q = 0; q < n; ++q) m[q] = fmaxf(m[q], m[q + n]);
  return m[0];
}

// N scores from the first-th on -> probabilities as bf16 pairs, added to the row's sum.
template <int N>
__device__ __forceinline__ void probabilities(const float (&v)[128], uint32_t (&packed)[64], int first, float2 scale2, float2 shift2, float2 (&sum2)[2]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 e = ffma2(make_float2(v[first + i], v[first + i + 1]), scale2, shift2);
    const float2 pr = make_float2(ex2(e.x), ex2(e.y));
    sum2[(i >> 1) & 1] = fadd2(sum2[(i >> 1) & 1], pr);
    __nv_bfloat162 h = __floats2bfloat162_rn(pr.x, pr.y);
    packed[(first + i) / 2] = *reinterpret_cast<uint32_t*>(&h);
  }
}

template <bool SPLIT, bool LONG>
__global__ void __launch_bounds__(kThreads, 2)
attention_bf16_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                      const __grid_constant__ CUtensorMap map_out16, const __grid_constant__ AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[16];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const uint32_t q_smem = smem_u32(smem_raw);      // two tiles each of Q, K and V, then the staging slots
  const uint32_t k_smem = q_smem + 2 * kTile, v_smem = k_smem + 2 * kTile;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // bars: 0,1 q_full | 2,3 q_empty | 4,5 k_full | 6,7 k_empty | 8,9 v_full | 10,11 v_empty | 12 s_full | 13 s_free | 14 p_full | 15 o_full
  const uint32_t q_full = smem_u32(&bars[0]), q_empty = smem_u32(&bars[2]), k_full = smem_u32(&bars[4]), k_empty = smem_u32(&bars[6]);
  const uint32_t v_full = smem_u32(&bars[8]), v_empty = smem_u32(&bars[10]);
  const uint32_t s_full = smem_u32(&bars[12]), s_free = smem_u32(&bars[13]), p_full = smem_u32(&bars[14]), o_full = smem_u32(&bars[15]);
  const int n_items = p.B * p.H * (p.q_tiles + (SPLIT ? p.q_tiles - p.split_from : 0));

  if (threadIdx.x == 32) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    if (p.out32) prefetch_tensormap(&map_out);
    if (p.out16 != nullptr) prefetch_tensormap(&map_out16);
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < 16; ++i) mbar_init(smem_u32(&bars[i]), i == 13 || i == 14 ? 4u : 1u);     // (s_free, p_full: a softmax warp each)
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // Everything above overlapped the previous kernel's tail; Q, K and V are its output.
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t tmem = tmem_base_slot;
  volatile int* abort_ptr = &abort_flag;
  // A wait that ends for all lanes of the warp or none; where it runs out the CTA gives up.  (The form that suspends: beside another
  // CTA's exponentials, polling warps take its issue slots, 27.9 us for eight sequences of 1024 tokens, 27.5 so.)
  auto wait = [&](uint32_t bar, uint32_t parity, int site) {
    const bool got = mbar_wait_cluster(bar, parity, abort_ptr);
    if (!got && !*abort_ptr) { atomicCAS(p.status, 0, (p.kernel_index << 8) | site); *abort_ptr = 1; }
    return __all_sync(0xffffffffu, got ? 1 : 0) != 0;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    int t = 0;                                     // key tiles loaded so far, over all items
    bool ok = true;
    auto load = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int token, const AttnItem& it) {
      if (elect_one()) {
        mbar_expect_tx(bar, kTile);
        tma_load_4d(dst, map, bar, 0, token, it.h, it.seq);
      }
      __syncwarp();
    };
    for (int ii = 0; ok; ++ii) {
      const int w = attn_nth_item(ii, n_items);
      if (w < 0) break;
      const AttnItem it = attn_item<SPLIT>(p, w);
      // a Q tile is free once every Q K^T of the item before the previous one has been executed
      const int qb = ii & 1;
      if (!wait(q_empty + 8 * qb, ((ii >> 1) & 1) ^ 1, 0x13)) break;
      load(q_smem + qb * kTile, &map_q, q_full + 8 * qb, it.q0, it);
      for (int j = 0; j < it.n_kv; ++j, ++t) {
        const int s = t & 1, token = (it.j0 + j) * kAttnRows;
        const uint32_t ph = (t >> 1) & 1;
        if (!(ok = wait(k_empty + 8 * s, ph ^ 1, 0x11))) break;
        load(k_smem + s * kTile, &map_k, k_full + 8 * s, token, it);
        if (!(ok = wait(v_empty + 8 * s, ph ^ 1, 0x12))) break;
        load(v_smem + s * kTile, &map_v, v_full + 8 * s, token, it);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // Tiles are numbered over all items (t): ring slot t & 1, ring phase (t >> 1) & 1; the other barriers complete once a tile.
    auto issue_qk = [&](int t, int item, bool first_of_item, bool last_of_item) {
      const int s = t & 1, qb = item & 1;
      if (first_of_item && !wait(q_full + 8 * qb, (item >> 1) & 1, 0x21)) return false;
      if (!wait(k_full + 8 * s, (t >> 1) & 1, 0x22)) return false;
      if (t > 0 && !wait(s_free, (t - 1) & 1, 0x25)) return false;       // the last tile's scores are in registers
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t qa = q_smem + qb * kTile, kb = k_smem + s * kTile;
      const uint32_t on = elect_one() ? 1u : 0u;
#pragma unroll
      for (int kd = 0; kd < 4; ++kd)
        umma_if(on, tmem, make_desc(qa + kd * 32, 16, 1024), make_desc(kb + kd * 32, 16, 1024), p.idesc_qk, kd != 0 ? 1u : 0u, true);
      if (on) {
        umma_commit(s_full);
        umma_commit(k_empty + 8 * s);
        if (last_of_item) umma_commit(q_empty + 8 * qb);       // its last scores are issued: the Q tile is handed back
      }
      __syncwarp();
      return true;
    };
    auto issue_pv = [&](int t, bool first_of_item) {
      const int s = t & 1;
      if (!wait(v_full + 8 * s, (t >> 1) & 1, 0x23)) return false;
      if (!wait(p_full, t & 1, 0x24)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t vb = v_smem + s * kTile;
      const uint32_t on = elect_one() ? 1u : 0u;
      // 16 keys = 8 columns of P and 16 128-byte rows of V per instruction
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_ts_if(on, tmem + kColO, tmem + kColP + kk * 8, make_desc(vb + kk * 2048, kTile, 1024, 2), p.idesc_pv,
                   !first_of_item || kk != 0 ? 1u : 0u, true);
      if (on) {
        umma_commit(o_full);
        umma_commit(v_empty + 8 * s);
      }
      __syncwarp();
      return true;
    };
    // The scores of a tile are computed under the exponentials of the one before, also those of an item's first tile.
    int t = 0;
    int w = attn_nth_item(0, n_items);
    int n_kv = w < 0 ? 0 : attn_item<SPLIT>(p, w).n_kv;
    bool ok = w >= 0 && issue_qk(0, 0, true, n_kv == 1);
    for (int ii = 0; ok && w >= 0; ++ii) {
      w = attn_nth_item(ii + 1, n_items);
      const int n_next = w < 0 ? 0 : attn_item<SPLIT>(p, w).n_kv;
      for (int j = 0; j < n_kv && ok; ++j, ++t) {
        if (j + 1 < n_kv) ok = issue_qk(t + 1, ii, false, j + 2 == n_kv);
        else if (w >= 0) ok = issue_qk(t + 1, ii + 1, true, n_next == 1);
        ok = ok && issue_pv(t, LONG ? j % kAttnRun == 0 : j == 0);
      }
      n_kv = n_next;
    }
  } else {
    // ---------------- softmax / output (warps 2..5): a thread per query row ----------------
    const int quad = warp & 3;
    const int row = quad * 32 + lane;              // row of the tile = tensor-memory lane
    const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
    uint8_t* const stage = smem_raw + 6 * kTile + quad * kStage;
    auto arrive = [&](uint32_t bar) {              // after this warp's last tensor-memory access that the barrier speaks of
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // One pass per tile, over all items, and one more for the last rows.  An item's rows are finished where its last P V has to be
    // waited for in any case: behind the next item's first exponentials.
    int t = 0, ii = 0, j = 0;
    int w = attn_nth_item(0, n_items);
    AttnItem it = attn_item<SPLIT>(p, w < 0 ? 0 : w), done = it;
    bool finished = false;                           // `done` is an item whose rows are still in tensor memory
    bool done_adds = false, done_ends = true;        // LONG: the run that is finished is not the first, is the last of its item
    float m_run = 0.0f, l_run = 0.0f, m_done = 0.0f, l_done = 0.0f;
    while (true) {
      uint32_t packed[64];                           // two keys per 32-bit column
      float alpha = 1.0f;
      bool rescale = false;                          // (of the whole warp)
      if (w >= 0) {
        if (!wait(s_full, t & 1, 0x31)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float v[128];
        tmem_ld128(lane_addr, v);
        arrive(s_free);
        // On the diagonal tile this warp's rows see the blocks of 32 keys up to their own, and of that one the first
        // lane + 1 keys.  The scale is positive (checked when the chain was matched), so the maximum commutes with it.
        const bool diagonal = it.j0 + j == it.qt;
        float mx;
        if (!diagonal) {
          mx = row_max<128>(v, 0);
        } else {
          mx = -CUDART_INF_F;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c > quad) continue;
            if (c == quad) {
#pragma unroll
              for (int i = 1; i < 32; ++i)
                if (i > lane) v[c * 32 + i] = -CUDART_INF_F;
            }
            mx = fmaxf(mx, row_max<32>(v, c * 32));
          }
        }
        mx *= p.scale_log2;
        // the first key of every tile at or below the diagonal is visible to every row, so the maximum is finite
        if (j == 0) {
          m_run = mx;
          l_run = 0.0f;
        } else if (LONG && j % kAttnRun == 0) {      // (the maximum goes on: a run of scores that are all -inf stays without weight)
          m_run = fmaxf(m_run, mx);
          l_run = 0.0f;
        } else {
          rescale = __any_sync(0xffffffffu, mx > m_run);
          if (rescale) {
            const float m_new = fmaxf(m_run, mx);
            alpha = ex2(m_run - m_new);
            m_run = m_new;
            l_run *= alpha;
          }
        }
        float2 sum2[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), shift2 = make_float2(-m_run, -m_run);
        if (!diagonal) {
          probabilities<128>(v, packed, 0, scale2, shift2, sum2);
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c <= quad) {
              probabilities<32>(v, packed, c * 32, scale2, shift2, sum2);
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) packed[c * 16 + i] = 0u;
            }
          }
        }
        l_run += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
      }
      if (t > 0) {
        // P V of the tile before has read P and written the output rows
        if (!wait(o_full, (t - 1) & 1, 0x32)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (finished) {
          finished = false;
          float oa[32], ob[32];
          tmem_ld32x2(lane_addr + kColO, lane_addr + kColO + 32, oa, ob);
          if constexpr (LONG) {
            float* const kept = p.kept + (size_t)blockIdx.x * kAttnPartialFloats + row;      // (read back by the thread that wrote it)
            if (done_adds) {
              const float earlier = ex2(__ldcg(kept + kAttnRows * kAttnHeadDim) - m_done);
              l_done = fmaf(__ldcg(kept + kAttnRows * kAttnHeadDim + kAttnRows), earlier, l_done);
#pragma unroll
              for (int i = 0; i < 32; ++i) oa[i] = fmaf(__ldcg(kept + i * kAttnRows), earlier, oa[i]);
#pragma unroll
              for (int i = 0; i < 32; ++i) ob[i] = fmaf(__ldcg(kept + (32 + i) * kAttnRows), earlier, ob[i]);
            }
            if (!done_ends) {
#pragma unroll
              for (int i = 0; i < 32; ++i) __stcg(kept + i * kAttnRows, oa[i]);
#pragma unroll
              for (int i = 0; i < 32; ++i) __stcg(kept + (32 + i) * kAttnRows, ob[i]);
              __stcg(kept + kAttnRows * kAttnHeadDim, m_done);
              __stcg(kept + kAttnRows * kAttnHeadDim + kAttnRows, l_done);
            }
          }
          // ---- a split item: leave this half's rows and state in the workspace; whoever arrives second merges.
          // Nobody waits for the other half.  The arrival is counted per lane quadrant, which is one warp here.
          bool writes = !LONG || done_ends;
          if (SPLIT && done.split && writes) {
            float* const mine = p.partial + ((size_t)done.slot * 2 + done.half) * kAttnPartialFloats;
            const float* const other = p.partial + ((size_t)done.slot * 2 + (done.half ^ 1)) * kAttnPartialFloats;
            // a column of the 64 after the other: a warp's 32 rows are one line
#pragma unroll
            for (int i = 0; i < 32; ++i) __stcg(mine + i * kAttnRows + row, oa[i]);
#pragma unroll
            for (int i = 0; i < 32; ++i) __stcg(mine + (32 + i) * kAttnRows + row, ob[i]);
            __stcg(mine + kAttnRows * kAttnHeadDim + row, m_done);
            __stcg(mine + kAttnRows * kAttnHeadDim + kAttnRows + row, l_done);
            __threadfence();
            __syncwarp();
            int arrived = 0;
            if (lane == 0) arrived = atomicAdd(p.arrivals + done.slot * 4 + quad, 1);
            arrived = __shfl_sync(0xffffffffu, arrived, 0);
            __threadfence();
            writes = arrived != 0;
            if (writes) {
              if (lane == 0) p.arrivals[done.slot * 4 + quad] = 0;      // for the next launch
              const float m2 = __ldcg(other + kAttnRows * kAttnHeadDim + row), l2 = __ldcg(other + kAttnRows * kAttnHeadDim + kAttnRows + row);
              const float m = fmaxf(m_done, m2);
              const float a1 = ex2(m_done - m), a2 = ex2(m2 - m);
              // Products rounded one by one and then added (no fused multiply-add): symmetric in the two
              // halves, so the bits do not depend on which of them merges.
              l_done = __fadd_rn(__fmul_rn(l_done, a1), __fmul_rn(l2, a2));
#pragma unroll
              for (int i = 0; i < 32; ++i) oa[i] = __fadd_rn(__fmul_rn(oa[i], a1), __fmul_rn(__ldcg(other + i * kAttnRows + row), a2));
#pragma unroll
              for (int i = 0; i < 32; ++i) ob[i] = __fadd_rn(__fmul_rn(ob[i], a1), __fmul_rn(__ldcg(other + (32 + i) * kAttnRows + row), a2));
            }
          }
          const int first_row = done.q0 + quad * 32;
          if (writes && first_row < p.T) {                 // (the maps end at the sequence's last row)
            const float inv = __fdividef(1.0f, l_done);
#pragma unroll
            for (int i = 0; i < 32; ++i) { oa[i] *= inv; ob[i] *= inv; }
            // A lane holds ONE row: the rows go through the warp's staging slot (128-byte rows, the 16-byte unit XORed
            // with the row against bank conflicts) and leave as bulk tensor stores.
            const int col = done.h * kAttnHeadDim;
            auto send = [&](auto&& fill, const CUtensorMap* map, int first_col) {
              if (lane == 0) tma_store_wait_read();        // the slot's last store has read it
              __syncwarp();
              fill();
              fence_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_store_3d(map, smem_u32(stage), first_col, first_row, done.seq);
                tma_store_commit();
              }
            };
            if (p.out16 != nullptr) send([&] { stage_rows_bf16x64(stage, oa, ob, lane); }, &map_out16, col);
            if (p.out32) {
              send([&] { stage_rows(stage, stage, oa, lane, false); }, &map_out, col);
              send([&] { stage_rows(stage, stage, ob, lane, false); }, &map_out, col + 32);
            }
          }
        } else if (rescale) {
          float oa[32], ob[32];
          tmem_ld32x2(lane_addr + kColO, lane_addr + kColO + 32, oa, ob);
          const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 a = fmul2(make_float2(oa[i], oa[i + 1]), alpha2), b = fmul2(make_float2(ob[i], ob[i + 1]), alpha2);
            oa[i] = a.x; oa[i + 1] = a.y; ob[i] = b.x; ob[i + 1] = b.y;
          }
          tmem_st32(lane_addr + kColO, oa);
          tmem_st32(lane_addr + kColO + 32, ob);
        }
      }
      if (w < 0) break;
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_st16(lane_addr + kColP + c * 16, packed + c * 16);
      tmem_st_wait();
      arrive(p_full);
      ++t;
      const bool ends = ++j == it.n_kv;
      if (ends || (LONG && j % kAttnRun == 0)) {
        finished = true;
        done = it;
        m_done = m_run;
        l_done = l_run;
        done_adds = j > kAttnRun;
        done_ends = ends;
      }
      if (ends) {
        j = 0;
        w = attn_nth_item(++ii, n_items);
        if (w >= 0) it = attn_item<SPLIT>(p, w);
      }
    }
    if (lane == 0) tma_store_wait_read();              // shared memory must outlive the stores that read it
  }

  // ---------------- common exit ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) let_copies_land();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kColumns) : "memory");
  }
}

using Kernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, AttnParams);
Kernel kernel_of(bool split, bool runs) {
  return split ? (runs ? attention_bf16_kernel<true, true> : attention_bf16_kernel<true, false>)
               : (runs ? attention_bf16_kernel<false, true> : attention_bf16_kernel<false, false>);
}

}  // namespace

std::vector<int> attention_item_order(int q_tiles, int split_from) {
  std::vector<int> order;
  for (int qt = 0; qt < q_tiles; ++qt) {
    order.push_back(qt << 1);
    if (qt >= split_from) order.push_back(qt << 1 | 1);
  }
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return attention_item_tiles(a, split_from) > attention_item_tiles(b, split_from); });
  return order;
}

int attention_item_tiles(int entry, int split_from) {
  const int n = (entry >> 1) + 1;
  return (entry >> 1) < split_from ? n : (entry & 1) ? n - (n >> 1) : n >> 1;
}

// Cycles from the first tile to the last of the longest SM, by walking the items the way the CTAs do.  Measured inside the
// kernel: a key tile takes a CTA 2300 cycles when it has the SM to itself, an item 1000 more (its
// rows' way out, its part of the copies' latency).  Beside another CTA a tile counts as 3300 (2900 inside the loop): fitted with the
// half's cost to 78 launches of 4 to 128 heads and 2 to 16 query tiles, every schedule of each timed.  The one it chooses is 0.5 % from
// the best on average and 5 % at most.  (With 2900: 1.7 %; 24 heads of 1024 tokens 15.0 us with halves on two CTAs an SM,
// 13.6 whole with one.)  A half costs 6500 (rows and state to the workspace, fence, counter, the other half's rows; one sequence
// of 256 tokens 5.7 -> 8.1 us), so only long items are worth it: 1024 tokens 12.3 -> 12.1 us, 2048 tokens 21.7 -> 20.4.
static int64_t schedule_cycles(int64_t heads, int q_tiles, int split_from, int sms, bool alone) {
  const std::vector<int> order = attention_item_order(q_tiles, split_from);
  const int64_t items = heads * (int64_t)order.size();
  const int64_t grid = std::min<int64_t>(items, alone ? sms : 2 * sms);
  std::vector<int64_t> work((size_t)grid, 0);
  for (int64_t w = 0; w < items; ++w) {
    const int64_t round = w / grid, at = w % grid;
    const int entry = order[(size_t)(w / heads)];
    work[(size_t)((round & 1) ? grid - 1 - at : at)] += 2300 * attention_item_tiles(entry, split_from) + 1000 + ((entry >> 1) >= split_from ? 6500 : 0);
  }
  int64_t longest = 0;
  for (int64_t i = 0; i < grid; ++i) {
    int64_t own = work[(size_t)i];
    if (!alone && i + sms < grid) {                  // the CTA beside it
      const int64_t other = work[(size_t)(i + sms)];
      own = std::min(own, other) * 33 / 23 + (std::max(own, other) - std::min(own, other));
    }
    longest = std::max(longest, own);
  }
  return longest;
}

AttnSchedule attention_bf16_schedule(int64_t heads, int q_tiles, int sms, bool may_split) {
  AttnSchedule best{q_tiles, false};
  if (heads * q_tiles > 8 * (int64_t)sms) return best;            // many rounds: nothing left to balance
  int64_t cycles = schedule_cycles(heads, q_tiles, q_tiles, sms, false);
  for (int from = may_split ? std::max(1, q_tiles / 2) : q_tiles; from <= q_tiles; ++from) {     // (halves of two key tiles at least)
    for (const bool alone : {true, false}) {
      const int64_t c = schedule_cycles(heads, q_tiles, from, sms, alone);
      if (c < cycles || (c == cycles && alone)) cycles = c, best = AttnSchedule{from, alone};
    }
  }
  return best;
}

bool attention_bf16_prepare() {
  for (const bool split : {false, true})
    for (const bool runs : {false, true})
      if (cudaFuncSetAttribute(kernel_of(split, runs), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemAlone) != cudaSuccess) return false;
  return true;
}

cudaError_t attention_bf16_launch(bool pdl, dim3 grid, bool alone, cudaStream_t s, const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v,
                                  const CUtensorMap& out, const CUtensorMap& out16, const AttnParams& p) {
  return launch_kernel(pdl, kernel_of(p.split_from < p.q_tiles, p.kept != nullptr), grid, dim3(kThreads), alone ? kSmemAlone : kSmem, s, q, k, v, out, out16, p);
}

}  // namespace kb200
