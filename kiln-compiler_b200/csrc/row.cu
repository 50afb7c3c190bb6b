// Row kernels: reductions over the innermost dim fused with the elementwise ops that share the
// rows (LayerNorm, softmax, row centring ...).  Role of the reference's `row` generator
// (kiln/gpu/codegen.py:312-430).
//
//   row_generic    any tape: one CTA per row, one pass over the row per level of reduction with
//                  the elementwise values recomputed from the inputs in every pass -- the scheme of
//                  the reference's chunked rows (codegen.py:371-428), so memory use is constant for
//                  any row length.
//   row_layernorm  two-pass mean / variance LayerNorm with affine, one to 16 warps per row, the row
//   row_softmax    held in registers (128-bit loads where width and alignment allow, shuffle
//                  reductions): one read and one write of the tensor, HBM-bound.
#include <cuda_bf16.h>

#include <type_traits>

#include "device_math.cuh"
#include "kb200_internal.h"
#include "split16.cuh"

namespace kb200 {

constexpr int kRowThreads = 256;
constexpr int kMaxRowRed = 8;

struct RowParams {
  int rank;                       // row dims + 1
  int n_operands;
  int max_level;
  int64_t n_rows;
  int64_t inner;
  int64_t shape[KB200_MAX_RANK];
  DevOperand ops[KB200_MAX_OPERANDS];
  DevTape tape;
};

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* scratch) {
  v = is_max ? warp_max(v) : warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();                 // scratch may still be read from the previous reduction
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = lane < (kRowThreads / 32) ? scratch[lane] : (is_max ? -CUDART_INF_F : 0.0f);
  r = is_max ? warp_max(r) : warp_sum(r);
  return r;
}

__global__ void __launch_bounds__(kRowThreads) row_generic_kernel(const __grid_constant__ RowParams p) {
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  __shared__ float s_red[KB200_MAX_TAPE];
  __shared__ float s_scratch[kRowThreads / 32];
  float r[KB200_MAX_TAPE];
  int64_t rowoff[KB200_MAX_OPERANDS];
  const int inner_d = p.rank - 1;
  for (int64_t row = blockIdx.x; row < p.n_rows; row += gridDim.x) {
    for (int o = 0; o < p.n_operands; ++o) rowoff[o] = 0;
    int64_t rest = row;
    for (int d = inner_d - 1; d >= 0; --d) {
      int64_t i = rest % p.shape[d];
      rest /= p.shape[d];
      for (int o = 0; o < p.n_operands; ++o) rowoff[o] += i * p.ops[o].stride[d];
    }
    // pass `limit` evaluates every value below that level; the last pass also stores
    for (int limit = 1; limit <= p.max_level + 1; ++limit) {
      const bool final_pass = limit == p.max_level + 1;
      int red_idx[kMaxRowRed];
      float acc[kMaxRowRed];
      int n_red = 0;
      if (!final_pass) {
        for (int t = 0; t < p.tape.n; ++t) {
          const int oc = p.tape.ops[t].opcode;
          if ((oc == KB200_OP_RSUM || oc == KB200_OP_RMAX) && p.tape.ops[t].level == limit && n_red < kMaxRowRed) {
            red_idx[n_red] = t;
            acc[n_red] = oc == KB200_OP_RSUM ? 0.0f : -CUDART_INF_F;
            ++n_red;
          }
        }
      }
      for (int64_t col = threadIdx.x; col < p.inner; col += kRowThreads) {
        for (int t = 0; t < p.tape.n; ++t) {
          const kb200_tape_op op = p.tape.ops[t];
          if (op.opcode == KB200_OP_STORE) {
            if (final_pass) {
              const int64_t st = p.ops[op.b].stride[inner_d];
              if (st != 0 || col == 0) p.ops[op.b].ptr[rowoff[op.b] + col * st] = r[op.a];
            }
            continue;
          }
          if (op.level >= limit) continue;
          switch (op.opcode) {
            case KB200_OP_LOAD: r[t] = p.ops[op.a].ptr[rowoff[op.a] + col * p.ops[op.a].stride[inner_d]]; break;
            case KB200_OP_IMM: r[t] = op.imm; break;
            case KB200_OP_RSUM:
            case KB200_OP_RMAX: r[t] = s_red[t]; break;
            default: r[t] = apply_op(op.opcode, r[op.a], r[op.b]); break;
          }
        }
        for (int j = 0; j < n_red; ++j) {
          const kb200_tape_op op = p.tape.ops[red_idx[j]];
          const float v = r[op.a];
          acc[j] = op.opcode == KB200_OP_RSUM ? acc[j] + v : d_max(acc[j], v);
        }
      }
      for (int j = 0; j < n_red; ++j) {
        const bool is_max = p.tape.ops[red_idx[j]].opcode == KB200_OP_RMAX;
        const float total = block_reduce(acc[j], is_max, s_scratch);
        if (threadIdx.x == 0) s_red[red_idx[j]] = total;
      }
      __syncthreads();
    }
  }
}

// ---- register-resident rows: LayerNorm and softmax ----
struct RowFastParams {
  const float* x;
  float* out;
  const float* gamma;
  const float* beta;
  int affine_static;       // both are frozen constants: no kernel writes them
  int64_t n_rows;
  int64_t x_row_stride, out_row_stride;
  int inner;
  float inv_n, eps;
  __nv_bfloat16* out16;    // optional bf16 copy of the output (same row stride as `out`), or null
  int store32;             // 0: only that copy is stored (every reader of the output takes it)
  // Two row dims (a [batch * heads, tokens, inner] softmax whose mask varies with the token only):
  // row = i0 * rows_inner + i1, and every tensor has a stride for each.  rows_inner == 0: one row dim.
  int64_t rows_inner;
  int64_t x_stride1, out_stride1;
  // A short elementwise chain applied to the loaded row before the reductions (scale and additive
  // mask in front of a softmax, a residual add in front of a LayerNorm), and where to store its value.
  int n_pre;
  struct Pre {
    int op;                // ChainOp
    int kind;              // 0 unary, 1 immediate, 2 tensor
    float imm;
    const float* ptr;
    int64_t stride0, stride1;
    int inner_stride;      // 1, or 0 for one value per row
  } pre[kMaxRowPre];
  const float* x_end;      // behind x's last element
  float* pre_out;          // receives the chain's value (same shape as x), or null
  int64_t pre_out_stride0, pre_out_stride1;
};

// PLANES: and the rows as float16 pairs, see split_rows.cu.  (Of its own: 40 bytes more of parameters cost the other launches 0.35 us of host time.)
struct RowPlanesParams : RowFastParams {
  PlanKernel::Planes planes;
};

enum { ROW_LAYERNORM = 0, ROW_SOFTMAX = 1 };

// VEC consecutive floats as one access.
template <int VEC>
__device__ __forceinline__ void row_load(float (&v)[VEC], const float* p) {
  if (VEC == 1) {
    v[0] = *p;
  } else {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[VEC - 1] = t.w;
  }
}
template <int VEC>
__device__ __forceinline__ void row_store(float* p, const float (&v)[VEC]) {
  if (VEC == 1) *p = v[0];
  else *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[VEC - 1]);
}
template <int VEC>
__device__ __forceinline__ float row_fold(const float (&v)[VEC]) { return VEC == 1 ? v[0] : (v[0] + v[1]) + (v[2] + v[VEC - 1]); }

// N accesses of VEC floats per lane; the lanes of a row's warps take consecutive accesses, lane by
// lane.  WIDE: the block's warps share one row (their partial reductions meet in shared memory), else
// every warp has a row of its own.
//
// What bounds it is the memory system, so a row is read once and written once, all of its loads in flight
// together.  A row that does not fit one warp's registers gets more warps instead of a second pass,
// and a row that 128-bit accesses cannot take (an odd width puts every row on another alignment)
// keeps the scheme with single floats: a warp still moves whole 128-byte lines.  LayerNorm 2048 x
// 8192 and rows of odd width used to run on the tape interpreter above (1238 x 6944: 789 us,
// now 16).  PRE: a chain in front of the reductions; its
// switch over the scalar ops, unrolled over a lane's elements, costs a softmax of 512 columns 54
// registers instead of 32.
//
// SHIFT: rows that start off a 16-byte boundary by a number of floats that varies with the row (odd widths).
// The accesses are the aligned float4 that cover a row; of the first and last one only the row's own
// elements count, the neighbours' are read with them and left alone.  x and out have the same shift;
// the last float4 of the tensor is read element by element where it would reach past its end.
// Softmax only (16384 x 333: 18.0 us with single floats, 10.2; 16384 x 4093: 124, 114): the affine parameters of
// a LayerNorm would still come as single floats, four lanes apart, and 16384 x 771 took 30.9 us against 28.2.
//
// PLANES: a LayerNorm whose reader multiplies float16 pairs leaves its rows as such, their scale by a third reduction.
template <int MODE, int VEC, int N, bool WIDE, bool PRE, bool SHIFT, bool AHEAD, bool PLANES>
__global__ void __launch_bounds__(WIDE ? 512 : 256) row_kernel(const __grid_constant__ std::conditional_t<PLANES, RowPlanesParams, RowFastParams> p) {
  const int lane = WIDE ? threadIdx.x : (threadIdx.x & 31);
  const int lanes = WIDE ? blockDim.x : 32;
  const int64_t row = WIDE ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  static_assert(!SHIFT || (VEC == 4 && !PRE && MODE == ROW_SOFTMAX), "shifted rows come as float4, without operands beside them");
  const int units = SHIFT ? (p.inner + 6) >> 2 : VEC == 1 ? p.inner : p.inner >> 2;
  static_assert(!PLANES || (VEC == 4 && MODE == ROW_LAYERNORM), "pairs are made of float4");
  __shared__ float partial[WIDE ? 64 : 1];
  [[maybe_unused]] __shared__ uint32_t partial_most[WIDE && PLANES ? 32 : 1], partial_least[WIDE && PLANES ? 32 : 1];
  // Each reduction of a WIDE row has its own half of `partial`: no barrier between the reads of one and the writes of the next.
  auto across = [&](float v, bool is_max, int which) {
    v = is_max ? warp_max(v) : warp_sum(v);
    if (!WIDE) return v;
    const int warps = lanes >> 5, l = threadIdx.x & 31;
    if (l == 0) partial[32 * which + (threadIdx.x >> 5)] = v;
    __syncthreads();
    const float t = l < warps ? partial[32 * which + l] : (is_max ? -CUDART_INF_F : 0.0f);
    return is_max ? warp_max(t) : warp_sum(t);
  };
  // The affine parameters of a LayerNorm are mostly constants of the plan, not outputs of the previous
  // kernel: then they are fetched before this kernel waits for its producer, so their latency is off the
  // path (fetched after the two reductions they added a dependent memory round trip to every row).  Where other
  // rows on the SM cover that round trip their registers are worth more: in WIDE blocks, and with rows of
  // four or more float4 a lane in several waves, they are fetched where they are used (16384 x 768:
  // 19.6 -> 17.9 us).
  constexpr bool kAhead = MODE == ROW_LAYERNORM && AHEAD;
  float g[kAhead ? N : 1][VEC], b[kAhead ? N : 1][VEC];
  if (kAhead) {
    if (!p.affine_static) pdl_wait();
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int j = lane + lanes * i;
      if (j < units) {
        row_load<VEC>(g[i], p.gamma + VEC * j);
        row_load<VEC>(b[i], p.beta + VEC * j);
      }
    }
  }
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  if (row >= p.n_rows) return;
  int64_t i0 = row, i1 = 0;
  if (p.rows_inner > 0) { i0 = row / p.rows_inner; i1 = row - i0 * p.rows_inner; }
  const float* x = p.x + i0 * p.x_row_stride + i1 * p.x_stride1;
  int64_t out_off = i0 * p.out_row_stride + i1 * p.out_stride1;
  // element e of access j is column 4 j + e - shift
  const int shift = SHIFT ? (int)((reinterpret_cast<uintptr_t>(x) >> 2) & 3) : 0;
  x -= shift;
  out_off -= shift;
  auto column_ok = [&](int j, int e) { return !SHIFT || (unsigned)(4 * j + e - shift) < (unsigned)p.inner; };
  float* out = p.out + out_off;
  float v[N][VEC];
  bool live[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int j = lane + lanes * i;
    live[i] = SHIFT ? 4 * j - shift < p.inner : j < units;
    if (!live[i]) continue;
    if (!SHIFT || x + VEC * j + VEC <= p.x_end) {
      row_load<VEC>(v[i], x + VEC * j);
    } else {
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[i][e] = column_ok(j, e) ? x[VEC * j + e] : 0.0f;
    }
    if (SHIFT) {                 // what a neighbour's element must be for this row's reduction
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (!column_ok(j, e)) v[i][e] = -CUDART_INF_F;
    }
  }
  for (int s = 0; PRE && s < p.n_pre; ++s) {
    const RowFastParams::Pre st = p.pre[s];
    const float* side = st.kind == 2 ? st.ptr + i0 * st.stride0 + i1 * st.stride1 : nullptr;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (!live[i]) continue;
      float t[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) t[e] = st.imm;
      if (st.kind == 2) {
        if (st.inner_stride == 1) {
          row_load<VEC>(t, side + VEC * (lane + lanes * i));
        } else {
          const float one = __ldg(side);
#pragma unroll
          for (int e = 0; e < VEC; ++e) t[e] = one;
        }
      }
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[i][e] = apply_chain(st.op, v[i][e], t[e]);
    }
  }
  if (PRE && p.pre_out != nullptr) {
    float* z = p.pre_out + i0 * p.pre_out_stride0 + i1 * p.pre_out_stride1;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (live[i]) row_store<VEC>(z + VEC * (lane + lanes * i), v[i]);
  }
  if (MODE == ROW_LAYERNORM) {
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (live[i]) s += row_fold<VEC>(v[i]);
    const float mean = across(s, false, 0) * p.inv_n;
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (live[i]) {
        float sq[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          v[i][e] -= mean;
          sq[e] = v[i][e] * v[i][e];
        }
        q += row_fold<VEC>(sq);
      }
    }
    const float rstd = 1.0f / sqrtf(across(q, false, 1) * p.inv_n + p.eps);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (live[i]) {
        const int j = lane + lanes * i;
        float y[VEC];
        const int at = kAhead ? i : 0;
        if (!kAhead) {
          row_load<VEC>(g[0], p.gamma + VEC * j);
          row_load<VEC>(b[0], p.beta + VEC * j);
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) y[e] = v[i][e] * rstd * g[at][e] + b[at][e];
        if constexpr (PLANES) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) v[i][e] = y[e];
          continue;
        }
        if (p.store32) row_store<VEC>(out + VEC * j, y);
        if (p.out16 != nullptr) {
          if (VEC == 1) {
            p.out16[out_off + j] = __float2bfloat16_rn(y[0]);
          } else {
            __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[VEC > 1 ? 1 : 0]), hi = __floats2bfloat162_rn(y[VEC > 1 ? 2 : 0], y[VEC - 1]);
            uint2 packed;
            packed.x = *reinterpret_cast<uint32_t*>(&lo);
            packed.y = *reinterpret_cast<uint32_t*>(&hi);
            *reinterpret_cast<uint2*>(p.out16 + out_off + 4 * j) = packed;
          }
        }
      }
    }
    if constexpr (PLANES) {
      uint32_t most = 0, least = ~0u;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (live[i])
#pragma unroll
          for (int e = 0; e < VEC; ++e) {
            most = max(most, magnitude_bits(v[i][e]));
            least = min(least, magnitude_bits(v[i][e]) - 1u);
          }
      most = warp_umax(most);
      least = warp_umin(least);
      if constexpr (WIDE) {
        const int l = threadIdx.x & 31;
        if (l == 0) {
          partial_most[threadIdx.x >> 5] = most;
          partial_least[threadIdx.x >> 5] = least;
        }
        __syncthreads();
        most = warp_umax(l < (lanes >> 5) ? partial_most[l] : 0u);
        least = warp_umin(l < (lanes >> 5) ? partial_least[l] : ~0u);
      }
      const RowScale scale(most);
      const uint32_t marks = row_marks(most, least);
      if (lane == 0) {
        p.planes.scales[row] = scale.back;
        p.planes.marks[row] = (uint8_t)marks;
      }
      __half* const heads = static_cast<__half*>(p.planes.heads) + row * p.planes.pitch;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (!live[i]) continue;
        const int j = lane + lanes * i;
        store_levels(heads + 4 * j, p.planes.plane, make_float4(v[i][0], v[i][1], v[i][2], v[i][3]), scale.by, marks);
        if (p.store32 || scale.marked) row_store<VEC>(out + VEC * j, v[i]);
      }
    }
  } else {
    float m = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (live[i])
#pragma unroll
        for (int e = 0; e < VEC; ++e) m = fmaxf(m, v[i][e]);
    m = across(m, true, 0);
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (live[i]) {
        // one warp and 128-bit accesses: exp through ex2.approx (relative error 2^-22, what the reference's
        // tl.exp lowers to as well); the forms that took over from the tape interpreter keep its expf
#pragma unroll
        for (int e = 0; e < VEC; ++e) v[i][e] = VEC == 1 || WIDE || SHIFT ? expf(v[i][e] - m) : __expf(v[i][e] - m);
        s += row_fold<VEC>(v[i]);
      }
    }
    s = across(s, false, 1);
    const float inv = 1.0f / s;     // one IEEE division per row; the elements are scaled by it (within an ulp of dividing)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (live[i]) {
        float y[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) y[e] = v[i][e] * inv;
        const int j = lane + lanes * i;
        if (column_ok(j, 0) && column_ok(j, VEC - 1)) {
          row_store<VEC>(out + VEC * j, y);
        } else {
#pragma unroll
          for (int e = 0; e < VEC; ++e)
            if (column_ok(j, e)) out[VEC * j + e] = y[e];
        }
      }
    }
  }
}

// The widest row: 16 warps (more would halve the registers of a thread) of 8 float4 or 32 floats a lane.
constexpr int64_t kRowLimit = 512 * 32, kShiftedLimit = kRowLimit - 8;

enum { ROW_FLOATS = 0, ROW_VECTORS = 1, ROW_SHIFTED = 2 };      // how rows are accessed

template <int MODE, bool PRE, bool PLANES>
static void launch_rows(const std::conditional_t<PLANES, RowPlanesParams, RowFastParams>& p, int access, int sm_count, bool pdl, cudaStream_t s) {
  const bool vec = access != ROW_FLOATS;
  const int units = access == ROW_SHIFTED ? (p.inner + 6) / 4 : vec ? p.inner / 4 : p.inner;
  const int n = (units + 31) / 32;                  // accesses per lane if one warp takes the row
  unsigned grid, block;
#define KB200_ROW_CASE(VEC, N, WIDE, AHEAD) launch_kernel(pdl, row_kernel<MODE, VEC, N, WIDE, PRE, false, AHEAD, PLANES>, dim3(grid), dim3(block), 0, s, p)
#define KB200_SHIFT_CASE(N, WIDE) launch_kernel(pdl, row_kernel<MODE, 4, N, WIDE, false, true, false, false>, dim3(grid), dim3(block), 0, s, p)
  if (n <= (vec && MODE == ROW_LAYERNORM ? 6 : 8)) {
    // a warp per row; few rows spread over more blocks.  (A LayerNorm of 8 float4 a lane, or either of 12,
    // spills; four warps of a quarter each do not.  With a chain in front, a LayerNorm of four float4 and softmaxes of four or
    // six, or of eight floats, spill 4 to 20 bytes.)
    const int warps = p.n_rows >= (int64_t)sm_count * 16 ? 8 : (p.n_rows >= (int64_t)sm_count * 4 ? 4 : 1);
    grid = (unsigned)((p.n_rows + warps - 1) / warps);
    block = warps * 32;
    if constexpr (!PRE && MODE == ROW_SOFTMAX) {
      if (access == ROW_SHIFTED) {
        if (n <= 2) KB200_SHIFT_CASE(2, false);
        else if (n <= 4) KB200_SHIFT_CASE(4, false);
        else KB200_SHIFT_CASE(8, false);
        return;
      }
    }
    const bool few = MODE == ROW_SOFTMAX || p.n_rows < (int64_t)sm_count * 64;
    if (vec) {
      if (n <= 1) KB200_ROW_CASE(4, 1, false, true);
      else if (n <= 2) KB200_ROW_CASE(4, 2, false, true);
      else if (n <= 4 && few) KB200_ROW_CASE(4, 4, false, true);
      else if (n <= 4) KB200_ROW_CASE(4, 4, false, false);
      else if (n <= 6 && few) KB200_ROW_CASE(4, 6, false, true);
      else if (n <= 6) KB200_ROW_CASE(4, 6, false, false);
      else if constexpr (MODE == ROW_SOFTMAX) KB200_ROW_CASE(4, 8, false, true);
    } else if constexpr (!PLANES) {
      if (n <= 2) KB200_ROW_CASE(1, 2, false, true);
      else if (n <= 4) KB200_ROW_CASE(1, 4, false, true);
      else KB200_ROW_CASE(1, 8, false, true);
    }
    return;
  }
  // a block per row, of as many warps (up to 16) as 4 float4 or 8 floats a lane leave
  int per = vec ? 4 : 8;
  while (per * 16 < n) per *= 2;
  grid = (unsigned)p.n_rows;
  block = (unsigned)((n + per - 1) / per) * 32;
  if constexpr (!PRE && MODE == ROW_SOFTMAX) {
    if (access == ROW_SHIFTED) {
      if (per == 4) KB200_SHIFT_CASE(4, true);
      else KB200_SHIFT_CASE(8, true);
      return;
    }
  }
  if (vec && per == 4) KB200_ROW_CASE(4, 4, true, false);
  else if (vec) KB200_ROW_CASE(4, 8, true, false);
  else if constexpr (!PLANES) {
    if (per == 8) KB200_ROW_CASE(1, 8, true, false);
    else if (per == 16) KB200_ROW_CASE(1, 16, true, false);
    else KB200_ROW_CASE(1, 32, true, false);
  }
#undef KB200_ROW_CASE
#undef KB200_SHIFT_CASE
}

template <int MODE>
static void launch_row_fast(const RowFastParams& p, int access, int sm_count, bool pdl, cudaStream_t s) {
  const bool pre = p.n_pre > 0 || p.pre_out != nullptr;
  if (pre) launch_rows<MODE, true, false>(p, access, sm_count, pdl, s);
  else launch_rows<MODE, false, false>(p, access, sm_count, pdl, s);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int choose_row(Plan& plan, PlanKernel& k) {
  (void)plan;
  const kb200_kernel_desc& d = k.desc;
  k.impl = IMPL_ROW_GENERIC;
  k.launches = 1;
  // the generic kernel keeps at most kMaxRowRed running reductions per pass (one pass per level)
  int per_level[KB200_MAX_TAPE + 1] = {0};
  for (int t = 0; t < d.n_tape; ++t) {
    const int oc = d.tape[t].opcode;
    if (oc != KB200_OP_RSUM && oc != KB200_OP_RMAX) continue;
    const int level = d.tape[t].level;
    if (level < 0 || level > KB200_MAX_TAPE)
      return fail(KB200_ERR_ARGUMENT, "row kernel %s: reduction level %d out of range", d.name, level);
    if (++per_level[level] > kMaxRowRed)
      return fail(KB200_ERR_UNSUPPORTED, "row kernel %s: more than %d reductions at one level of the chain", d.name, kMaxRowRed);
  }
  const int64_t inner = d.iter_shape[d.iter_rank - 1];
  // register-resident rows: one or two row dims, every tensor contiguous (or one value per row) along the
  // innermost; 128-bit accesses where all of width, strides and bases allow them
  const int last = d.iter_rank - 1;
  if ((d.iter_rank != 2 && d.iter_rank != 3) || inner < 1 || inner > kRowLimit) return KB200_OK;
  bool vec = inner % 4 == 0;
  auto row_tensor_ok = [&](int slot) {
    const DevOperand& o = k.ops[slot];
    vec = vec && aligned16(o.ptr);
    for (int dd = 0; dd < last; ++dd) vec = vec && o.stride[dd] % 4 == 0;
    return o.stride[last] == 1 || inner == 1;
  };
  auto vector_ok = [&](int slot) {
    for (int dd = 0; dd < last; ++dd)
      if (k.ops[slot].stride[dd] != 0) return false;
    return row_tensor_ok(slot);
  };
  // operands of the chain in front of the reductions: a tensor like x, or one value per row
  auto pre_ok = [&]() {
    for (int st = 0; st < k.row_pre.n; ++st) {
      const int slot = k.row_pre.steps[st].slot;
      if (slot >= 0 && k.ops[slot].stride[last] != 0 && !row_tensor_ok(slot)) return false;
    }
    return k.pre_out_slot < 0 || row_tensor_ok(k.pre_out_slot);
  };
  k.row_pre.n = 0;
  k.pre_out_slot = -1;
  if (match_layernorm(d, &k)) {
    if (row_tensor_ok(k.x_slot) && row_tensor_ok(k.out_slot) && vector_ok(k.g_slot) && vector_ok(k.b_slot) && pre_ok())
      k.impl = IMPL_ROW_LAYERNORM;
  } else if (match_softmax(d, &k)) {
    if (row_tensor_ok(k.x_slot) && row_tensor_ok(k.out_slot) && pre_ok()) k.impl = IMPL_ROW_SOFTMAX;
  }
  k.row_vec = vec;
  return KB200_OK;
}

int launch_row(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  const kb200_kernel_desc& d = k.desc;
  const int64_t inner = d.iter_shape[d.iter_rank - 1];
  int64_t n_rows = 1;
  for (int i = 0; i < d.iter_rank - 1; ++i) n_rows *= d.iter_shape[i];
  if (k.impl == IMPL_ROW_LAYERNORM || k.impl == IMPL_ROW_SOFTMAX) {
    RowFastParams p{};
    p.store32 = 1;
    p.x = k.ops[k.x_slot].ptr;
    p.out = k.ops[k.out_slot].ptr;
    p.n_rows = n_rows;
    p.x_row_stride = k.ops[k.x_slot].stride[0];
    p.out_row_stride = k.ops[k.out_slot].stride[0];
    p.inner = (int)inner;
    const bool two = d.iter_rank == 3;
    p.rows_inner = two ? d.iter_shape[1] : 0;
    p.x_stride1 = two ? k.ops[k.x_slot].stride[1] : 0;
    p.out_stride1 = two ? k.ops[k.out_slot].stride[1] : 0;
    p.n_pre = k.row_pre.n;
    p.x_end = p.x + (n_rows > 0 ? k.ops[k.x_slot].stride[0] * (d.iter_shape[0] - 1) + p.x_stride1 * (two ? d.iter_shape[1] - 1 : 0) + inner : 0);
    for (int st = 0; st < k.row_pre.n; ++st) {
      const ChainStep& cs = k.row_pre.steps[st];
      RowFastParams::Pre& pr = p.pre[st];
      pr.op = cs.op;
      pr.imm = cs.imm;
      pr.kind = cs.slot == -2 ? 0 : (cs.slot == -1 ? 1 : 2);
      if (cs.slot >= 0) {
        const DevOperand& o = k.ops[cs.slot];
        pr.ptr = o.ptr;
        pr.stride0 = o.stride[0];
        pr.stride1 = two ? o.stride[1] : 0;
        pr.inner_stride = (int)o.stride[d.iter_rank - 1];
      }
    }
    // Softmax rows that do not start on 16 bytes: shifted float4, when x and the output are shifted alike in every
    // row and no chain in front brings operands of its own.
    int access = k.row_vec ? ROW_VECTORS : ROW_FLOATS;
    {
      const DevOperand &x = k.ops[k.x_slot], &o = k.ops[k.out_slot];
      bool alike = aligned16(x.ptr) && aligned16(o.ptr);
      for (int dd = 0; dd < d.iter_rank - 1; ++dd) alike = alike && (x.stride[dd] - o.stride[dd]) % 4 == 0;
      if (k.impl == IMPL_ROW_SOFTMAX && !k.row_vec && alike && k.row_pre.n == 0 && k.pre_out_slot < 0 && inner >= 32 && inner <= kShiftedLimit) access = ROW_SHIFTED;
    }
    p.pre_out = k.pre_out_slot >= 0 ? k.ops[k.pre_out_slot].ptr : nullptr;
    p.pre_out_stride0 = k.pre_out_slot >= 0 ? k.ops[k.pre_out_slot].stride[0] : 0;
    p.pre_out_stride1 = k.pre_out_slot >= 0 && two ? k.ops[k.pre_out_slot].stride[1] : 0;
    if (k.impl == IMPL_ROW_LAYERNORM) {
      p.gamma = k.ops[k.g_slot].ptr;
      p.affine_static = d.operands[k.g_slot].base_kind == KB200_BASE_CONST && d.operands[k.b_slot].base_kind == KB200_BASE_CONST;
      p.beta = k.ops[k.b_slot].ptr;
      p.inv_n = k.ln_inv_n;
      p.eps = k.ln_eps;
      p.out16 = static_cast<__nv_bfloat16*>(k.shadow_out);
      p.store32 = k.mirror_only && (p.out16 != nullptr || k.planes_out.heads != nullptr) ? 0 : 1;
      if (k.planes_out.heads != nullptr) {          // (rows of float4)
        RowPlanesParams with;
        static_cast<RowFastParams&>(with) = p;
        with.planes = k.planes_out;
        if (p.n_pre > 0 || p.pre_out != nullptr) launch_rows<ROW_LAYERNORM, true, true>(with, ROW_VECTORS, plan.sm_count, plan.pdl, s);
        else launch_rows<ROW_LAYERNORM, false, true>(with, ROW_VECTORS, plan.sm_count, plan.pdl, s);
      } else {
        launch_row_fast<ROW_LAYERNORM>(p, access, plan.sm_count, plan.pdl, s);
      }
    } else {
      launch_row_fast<ROW_SOFTMAX>(p, access, plan.sm_count, plan.pdl, s);
    }
  } else {
    RowParams p{};
    p.rank = d.iter_rank;
    p.n_operands = d.n_operands;
    p.n_rows = n_rows;
    p.inner = inner;
    p.max_level = 0;
    for (int t = 0; t < d.n_tape; ++t)
      if (d.tape[t].level > p.max_level) p.max_level = d.tape[t].level;
    for (int i = 0; i < d.iter_rank; ++i) p.shape[i] = d.iter_shape[i];
    for (int o = 0; o < d.n_operands; ++o) p.ops[o] = k.ops[o];
    p.tape = k.tape;
    int64_t cap = (int64_t)plan.sm_count * 8;
    launch_kernel(plan.pdl, row_generic_kernel, dim3((unsigned)(n_rows < cap ? n_rows : cap)), dim3(kRowThreads), 0, s, p);
  }
  KB200_CUDA(cudaGetLastError());
  return KB200_OK;
}

}  // namespace kb200
