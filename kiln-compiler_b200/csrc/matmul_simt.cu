// Exact-FP32 batched matmul with a fused epilogue, on the FP32 pipes.  Role of the reference's
// matmul generator with input_precision="ieee" (kiln/gpu/codegen.py:484-530): arbitrary strided
// A [batch, M, K] and B [batch, K, N], FP32 accumulation over K, the epilogue applied to the
// accumulator while it is still in registers, out-of-range tile elements read as 0 and are not
// stored (codegen.py:513-517, 524).  tcgen05 has no IEEE-FP32 operand kind, so this is the path
// for allow_tf32=False; it is also the fallback for operands the tensor-core path cannot take.
#include <type_traits>

#include "device_math.cuh"
#include "kb200_internal.h"
#include "matmul.h"

namespace kb200 {

template <int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) mm_simt_kernel(const __grid_constant__ MatmulParams p) {
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  constexpr int NT = (BM / TM) * (BN / TN);
  __shared__ __align__(16) float As[BK][BM + 4];
  __shared__ __align__(16) float Bs[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int64_t tiles_n = (p.N + BN - 1) / BN;
  const int64_t m0 = (blockIdx.x / tiles_n) * BM, n0 = (blockIdx.x % tiles_n) * BN;
  const int64_t b = blockIdx.z;
  const float* A = p.ops[p.a_slot].ptr + b * p.ops[p.a_slot].stride[0];
  const float* B = p.ops[p.b_slot].ptr + b * p.ops[p.b_slot].stride[0];
  const int64_t a_sm = p.ops[p.a_slot].stride[1], a_sk = p.ops[p.a_slot].stride[2];
  const int64_t b_sk = p.ops[p.b_slot].stride[1], b_sn = p.ops[p.b_slot].stride[2];
  const bool a_kfast = a_sk == 1 || a_sm != 1;
  const bool b_nfast = b_sn == 1 || b_sk != 1;

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  for (int64_t k0 = 0; k0 < p.K; k0 += BK) {
#pragma unroll
    for (int e = tid; e < BM * BK; e += NT) {
      const int kk = a_kfast ? e % BK : e / BM;
      const int mm = a_kfast ? e / BK : e % BM;
      const int64_t gm = m0 + mm, gk = k0 + kk;
      As[kk][mm] = (gm < p.M && gk < p.K) ? A[gm * a_sm + gk * a_sk] : 0.0f;
    }
#pragma unroll
    for (int e = tid; e < BK * BN; e += NT) {
      const int nn = b_nfast ? e % BN : e / BK;
      const int kk = b_nfast ? e / BN : e % BK;
      const int64_t gn = n0 + nn, gk = k0 + kk;
      Bs[kk][nn] = (gn < p.N && gk < p.K) ? B[gk * b_sk + gn * b_sn] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], bb[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 t = *reinterpret_cast<const float4*>(&As[kk][ty * TM + i]);
        a[i] = t.x; a[i + 1] = t.y; a[i + 2] = t.z; a[i + 3] = t.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 t = *reinterpret_cast<const float4*>(&Bs[kk][tx * TN + j]);
        bb[j] = t.x; bb[j + 1] = t.y; bb[j + 2] = t.z; bb[j + 3] = t.w;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], bb[j], acc[i][j]);
    }
    __syncthreads();
  }

  // ---- epilogue ----
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int64_t gm = m0 + ty * TM + i;
    if (gm >= p.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int64_t gn = n0 + tx * TN + j;
      if (gn >= p.N) continue;
      epilogue_store(p, acc[i][j], b, gm, gn);
    }
  }
}

// Decode shape, M == 1: the weight matrix is read exactly once, so the kernel is bound by how many
// bytes it keeps in flight and by the latencies around that.  Each CTA owns 32 output columns; its 32 warps split K and
// combine through shared memory in warp order, which keeps the result deterministic.  A warp reads four rows of 128 bytes per
// instruction, up to 24 rows at once: all of K = 768, 9.4 MB over the 96 CTAs of a 3072-wide layer.  (Rows off a 16-byte pitch:
// VEC = 1, one row per instruction, 16 at once.)  Those of a frozen weight are requested before the wait for the previous kernel, whose
// tail they then arrive under.  The parameters are this kernel's own 0.4 KB: those of the general epilogue are 2.9 KB, which every
// launch pays for on the host and again in a cold constant cache.
constexpr int kGemvWarps = 32;
constexpr int kGemvCols = 32;
constexpr int kGemvRows = 24;        // rows of B a warp has in flight

struct GemvOperand {
  float* ptr;
  int64_t batch_stride, stride;      // elements per batch entry | per column (per k for A, per row for B)
};
struct GemvParams {
  int64_t N, K;
  GemvOperand a, b, out, side[kMaxChain];
  int frozen;                        // B is a constant: nobody before this kernel writes it
  int n_steps;
  int op[kMaxChain];
  float imm[kMaxChain];              // used where side[].ptr is null
};

// One column's sum -> the fused chain -> memory.
__device__ __forceinline__ void gemv_store(const GemvParams& p, float v, int64_t b, int64_t n) {
#pragma unroll 1
  for (int s = 0; s < p.n_steps; ++s) {
    const float* const side = p.side[s].ptr;
    v = apply_chain(p.op[s], v, side != nullptr ? side[b * p.side[s].batch_stride + n * p.side[s].stride] : p.imm[s]);
  }
  p.out.ptr[b * p.out.batch_stride + n * p.out.stride] = v;
}
// (an epilogue that is no chain)
__device__ __forceinline__ void gemv_store(const MatmulParams& p, float v, int64_t b, int64_t n) { epilogue_store(p, v, b, 0, n); }

__device__ __forceinline__ GemvOperand gemv_a(const GemvParams& p) { return p.a; }
__device__ __forceinline__ GemvOperand gemv_b(const GemvParams& p) { return p.b; }
__device__ __forceinline__ bool gemv_frozen(const GemvParams& p) { return p.frozen != 0; }
__device__ __forceinline__ GemvOperand gemv_a(const MatmulParams& p) { return {p.ops[p.a_slot].ptr, p.ops[p.a_slot].stride[0], p.ops[p.a_slot].stride[2]}; }
__device__ __forceinline__ GemvOperand gemv_b(const MatmulParams& p) { return {p.ops[p.b_slot].ptr, p.ops[p.b_slot].stride[0], p.ops[p.b_slot].stride[1]}; }
__device__ __forceinline__ bool gemv_frozen(const MatmulParams&) { return false; }

template <typename Params, int VEC>
__global__ void __launch_bounds__(kGemvWarps * 32) mm_gemv_kernel(const __grid_constant__ Params p) {
  __shared__ __align__(16) float part[kGemvWarps][kGemvCols];
  constexpr int kLanes = kGemvCols / VEC;         // lanes a row takes
  constexpr int kStep = 32 / kLanes;              // rows per instruction
  constexpr int kLoads = kGemvRows / kStep;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t b = blockIdx.z;
  const GemvOperand oa = gemv_a(p), ob = gemv_b(p);
  const int64_t n = (int64_t)blockIdx.x * kGemvCols + lane % kLanes * VEC;
  // this warp's part of K, counted from its first row: 32 bits are enough for that
  const int64_t k_per = (p.K + kGemvWarps - 1) / kGemvWarps, k_lo = warp * k_per;
  const int k_end = (int)(k_lo + k_per < p.K ? k_per : k_lo < p.K ? p.K - k_lo : 0);
  const int k_first = lane / kLanes;
  const float* const A = oa.ptr + b * oa.batch_stride + k_lo * oa.stride;
  const float* const B = ob.ptr + b * ob.batch_stride + k_lo * ob.stride + n;
  const bool live = n < p.N;                      // (VEC = 4: N is a multiple of four)
  float acc[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) acc[e] = 0.0f;
  if constexpr (VEC == 1) {
    // A row is one load of the warp, so whole blocks of rows go without a test of each: with one, 1 x 3001 x 2048 took 10.2 us,
    // 5.4 without; 1 x 4097 x 1537 10.2 and 4.7, 1 x 50257 x 768 60.5 and 47.8.
    pdl_wait();
    pdl_launch_dependents();
    auto block = [&](int k, auto rows) {
      constexpr int R = decltype(rows)::value;
      float w[R], a[R];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        w[u] = __ldg(B + (k + u) * ob.stride);
        a[u] = __ldg(A + (k + u) * oa.stride);
      }
#pragma unroll
      for (int u = 0; u < R; ++u) acc[0] = fmaf(a[u], w[u], acc[0]);
    };
    if (live) {
      int k = k_first;
      for (; k + 16 <= k_end; k += 16) block(k, std::integral_constant<int, 16>{});
      for (; k + 8 <= k_end; k += 8) block(k, std::integral_constant<int, 8>{});
      for (; k < k_end; ++k) block(k, std::integral_constant<int, 1>{});
    }
  } else {
    float w[kLoads][VEC];
    auto fetch = [&](int k0) {
      const float* row = B + k0 * ob.stride;
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        const float4 t = live && k0 + u * kStep < k_end ? __ldg(reinterpret_cast<const float4*>(row)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w[u][0] = t.x; w[u][1] = t.y; w[u][2] = t.z; w[u][3] = t.w;
        row += kStep * ob.stride;
      }
    };
    const bool early = gemv_frozen(p);
    if (early) fetch(k_first);
    pdl_wait();                 // the producer of this kernel's inputs has completed
    pdl_launch_dependents();    // the next kernel may begin its start-up
    if (!early) fetch(k_first);
    for (int k0 = k_first;;) {
      float a[kLoads];
      const float* x = A + k0 * oa.stride;
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        a[u] = k0 + u * kStep < k_end ? __ldg(x) : 0.0f;
        x += kStep * oa.stride;
      }
#pragma unroll
      for (int u = 0; u < kLoads; ++u)
        if (k0 + u * kStep < k_end) {               // (an infinite or NaN element of neither operand may meet a row that is not there)
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[e] = fmaf(a[u], w[u][e], acc[e]);
        }
      k0 += kGemvRows;
      if (k0 - lane / kLanes >= k_end) break;       // (the same for all lanes)
      fetch(k0);
    }
  }
  // the rows that a warp has read side by side
#pragma unroll
  for (int d = kLanes; d < 32; d *= 2)
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], d);
  if (lane < kLanes) {
    if constexpr (VEC == 4) *reinterpret_cast<float4*>(&part[warp][lane * 4]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    else part[warp][lane] = acc[0];
  }
  __syncthreads();
  if (threadIdx.x < kGemvCols) {
    const int64_t gn = (int64_t)blockIdx.x * kGemvCols + threadIdx.x;
    if (gn < p.N) {
      float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int i = 0; i < kGemvWarps; ++i) t[i & 3] += part[i][threadIdx.x];
      gemv_store(p, (t[0] + t[1]) + (t[2] + t[3]), b, gn);
    }
  }
}

void fill_matmul_params(const PlanKernel& k, MatmulParams* p) {
  const kb200_kernel_desc& d = k.desc;
  p->batch = k.batch;
  p->M = k.M;
  p->N = k.N;
  p->K = k.K;
  p->a_slot = d.a_slot;
  p->b_slot = d.b_slot;
  p->n_operands = k.n_ops;
  for (int o = 0; o < k.n_ops; ++o) p->ops[o] = k.ops[o];
  p->has_chain = k.has_chain ? 1 : 0;
  p->chain = k.chain;
  p->tape = k.tape;
}

static void launch_gemv(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  const int a_slot = k.desc.a_slot, b_slot = k.desc.b_slot;
  const dim3 grid((unsigned)((k.N + kGemvCols - 1) / kGemvCols), 1, (unsigned)k.batch), block(kGemvWarps * 32);
  const DevOperand& B = k.ops[b_slot];
  const bool vec = k.N % 4 == 0 && B.stride[1] % 4 == 0 && B.stride[0] % 4 == 0 && reinterpret_cast<uintptr_t>(B.ptr) % 16 == 0;
  if (!k.has_chain) {
    MatmulParams p{};
    fill_matmul_params(k, &p);
    launch_kernel(plan.pdl, vec ? mm_gemv_kernel<MatmulParams, 4> : mm_gemv_kernel<MatmulParams, 1>, grid, block, 0, s, p);
    return;
  }
  GemvParams g{};
  auto operand = [&](int slot, int d) { return GemvOperand{k.ops[slot].ptr, k.ops[slot].stride[0], k.ops[slot].stride[d]}; };
  g.N = k.N;
  g.K = k.K;
  g.a = operand(a_slot, 2);
  g.b = operand(b_slot, 1);
  g.out = operand(k.chain.out_slot, 2);
  g.frozen = k.desc.operands[b_slot].base_kind == KB200_BASE_CONST ? 1 : 0;
  g.n_steps = k.chain.n;
  for (int i = 0; i < k.chain.n; ++i) {
    g.op[i] = k.chain.steps[i].op;
    g.imm[i] = k.chain.steps[i].imm;
    if (k.chain.steps[i].slot >= 0) g.side[i] = operand(k.chain.steps[i].slot, 2);
  }
  launch_kernel(plan.pdl, vec ? mm_gemv_kernel<GemvParams, 4> : mm_gemv_kernel<GemvParams, 1>, grid, block, 0, s, g);
}

int launch_matmul_simt(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  if (k.impl == IMPL_MM_GEMV) {
    launch_gemv(plan, k, s);
  } else {
    MatmulParams p{};
    fill_matmul_params(k, &p);
    const int64_t big_tiles = ((p.M + 127) / 128) * ((p.N + 127) / 128) * p.batch;
    if (big_tiles >= plan.sm_count) {
      dim3 grid((unsigned)(((p.M + 127) / 128) * ((p.N + 127) / 128)), 1, (unsigned)p.batch);
      launch_kernel(plan.pdl, mm_simt_kernel<128, 128, 8, 8, 8>, grid, dim3(256), 0, s, p);
    } else {
      dim3 grid((unsigned)(((p.M + 63) / 64) * ((p.N + 63) / 64)), 1, (unsigned)p.batch);
      launch_kernel(plan.pdl, mm_simt_kernel<64, 64, 16, 4, 4>, grid, dim3(256), 0, s, p);
    }
  }
  KB200_CUDA(cudaGetLastError());
  return KB200_OK;
}

}  // namespace kb200
