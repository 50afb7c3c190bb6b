// Elementwise kernels: fused chains of scalar ops over strided / broadcast operands, and copies.
// Role of the reference's `elementwise` generator (kiln/gpu/codegen.py:284-310).
//
//   ew_generic      any tape, any strides: one element per thread, values in a per-thread file.
//   ew_chain_vec4   the tape is a chain and every operand is contiguous (or constant) along the
//                   innermost dim: 128-bit loads/stores, the running value stays in registers.
//                   HBM-bound: reads each input once, writes the output once.
//   ew_chain        the same for widths and alignments that 128 bits cannot take: float4 along the flat
//                   tensor where the output and the first input are dense, else one element per access.
//   ew_transpose    a chain whose first input is contiguous along a different dim than the output
//                   (head-split K^T copy, unfrozen weight transposes): 32x32 tiles through shared
//                   memory so both the read and the write are coalesced.
#include "device_math.cuh"
#include "kb200_internal.h"

namespace kb200 {

struct EwParams {
  int rank;
  int n_operands;
  int64_t numel;
  int64_t shape[KB200_MAX_RANK];
  DevOperand ops[KB200_MAX_OPERANDS];
  DevTape tape;
};

__global__ void __launch_bounds__(256) ew_generic_kernel(const __grid_constant__ EwParams p) {
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  float r[KB200_MAX_TAPE];
  int64_t off[KB200_MAX_OPERANDS];
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < p.numel; idx += step) {
    for (int o = 0; o < p.n_operands; ++o) off[o] = 0;
    int64_t rest = idx;
    for (int d = p.rank - 1; d >= 0; --d) {
      int64_t i = rest % p.shape[d];
      rest /= p.shape[d];
      for (int o = 0; o < p.n_operands; ++o) off[o] += i * p.ops[o].stride[d];
    }
    for (int t = 0; t < p.tape.n; ++t) {
      const kb200_tape_op op = p.tape.ops[t];
      switch (op.opcode) {
        case KB200_OP_LOAD: r[t] = p.ops[op.a].ptr[off[op.a]]; break;
        case KB200_OP_IMM: r[t] = op.imm; break;
        case KB200_OP_STORE: p.ops[op.b].ptr[off[op.b]] = r[op.a]; break;
        default: r[t] = apply_op(op.opcode, r[op.a], r[op.b]); break;
      }
    }
  }
}

// ---- vectorised chain ----
constexpr int kVecRank = 4;

struct EwChainParams {
  uint32_t nvec;                 // accesses in all: elements / VEC
  uint32_t shape[kVecRank];      // last entry = inner / VEC
  // Quotients by shape[d] through a multiplication: x / d = x * ceil(2^(31 + s) / d) >> (31 + s) with
  // 2^s >= d, exact for x < 2^31.
  uint32_t magic[kVecRank];
  int shift[kVecRank];
  int stream_out;                // a large result that only the caller reads: see streams_out
  float* ptr[KB200_MAX_OPERANDS];
  // element strides as 32-bit numbers (the host takes this kernel only when every offset fits),
  // the innermost one already multiplied by VEC: VEC (an access per index) or 0 (one scalar per row)
  int32_t stride[KB200_MAX_OPERANDS][kVecRank];
  Chain chain;
};

template <int RANK>
__device__ __forceinline__ uint32_t ew_offset(const EwChainParams& p, int slot, const uint32_t* idx) {
  uint32_t off = 0;
#pragma unroll
  for (int d = 0; d < RANK; ++d) off += idx[d] * (uint32_t)p.stride[slot][d];
  return off;
}

template <int RANK, int VEC>
__device__ __forceinline__ void ew_load(const EwChainParams& p, int slot, const uint32_t* idx, float* v) {
  const float* ptr = p.ptr[slot] + ew_offset<RANK>(p, slot, idx);
  if (VEC == 1) {
    *v = *ptr;
  } else if (p.stride[slot][RANK - 1] == 0) {
    v[0] = v[1] = v[2] = v[3] = __ldg(ptr);
  } else {
    const float4 x = *reinterpret_cast<const float4*>(ptr);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
}

// U accesses of VEC elements per thread, a block's accesses contiguous per u (coalesced).  The rank is a
// template parameter and all index arithmetic is 32-bit, its divisions multiplications: at 8 bytes moved
// per element the kernel must stay far below the instruction budget of the memory system (a generic
// 64-bit version of the same loop spent 75 instructions per element and ran at a third of the copy
// bandwidth).  Single elements take eight accesses per thread, for as many bytes in flight.
template <int RANK, int U, int VEC>
__global__ void __launch_bounds__(256) ew_chain_kernel(const __grid_constant__ EwChainParams p) {
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  const uint32_t nvec = p.nvec;
  const uint32_t step = gridDim.x * blockDim.x * U;
  for (uint32_t base = blockIdx.x * blockDim.x * U + threadIdx.x; base < nvec; base += step) {
    float v[VEC * U];
    uint32_t idx[U][RANK];
    bool live[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + (uint32_t)u * blockDim.x;
      live[u] = i < nvec;
      uint32_t rest = live[u] ? i : 0;
#pragma unroll
      for (int d = RANK - 1; d > 0; --d) {
        const uint32_t q = (uint32_t)(((uint64_t)rest * p.magic[d]) >> p.shift[d]);
        idx[u][d] = rest - q * p.shape[d];
        rest = q;
      }
      idx[u][0] = rest;
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[VEC * u + e] = 0.0f;
      if (live[u]) ew_load<RANK, VEC>(p, p.chain.first_slot, idx[u], v + VEC * u);
    }
    for (int s = 0; s < p.chain.n; ++s) {
      const ChainStep st = p.chain.steps[s];
      float side[VEC * U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) side[VEC * u + e] = st.imm;
        if (st.slot >= 0 && live[u]) ew_load<RANK, VEC>(p, st.slot, idx[u], side + VEC * u);
      }
      chain_step<VEC * U>(st.op, v, side);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!live[u]) continue;
      float* out = p.ptr[p.chain.out_slot] + ew_offset<RANK>(p, p.chain.out_slot, idx[u]);
      if (VEC == 1) *out = v[u];
      else {
        const float4 t = make_float4(v[VEC * u], v[VEC * u + 1], v[VEC * u + 2], v[VEC * u + VEC - 1]);
        if (p.stream_out) __stcs(reinterpret_cast<float4*>(out), t);
        else *reinterpret_cast<float4*>(out) = t;
      }
    }
  }
}

// Two dims, any width: the output and the first input are dense, so the tensor is walked as float4 whose elements
// may belong to two rows.  Other dense operands come the same way, the rest (a value per column or per
// row) element by element, from cache.  bias + GELU 8192 x 4093: 79.6 us as single elements, 51 % of
// the copy bandwidth.
struct EwFlatParams {
  uint32_t numel, inner, magic;
  int shift;
  float* ptr[KB200_MAX_OPERANDS];
  int32_t stride_row[KB200_MAX_OPERANDS], stride_col[KB200_MAX_OPERANDS];
  uint32_t dense;                // bit per operand
  Chain chain;
};

template <int U>
__global__ void __launch_bounds__(256) ew_flat_kernel(const __grid_constant__ EwFlatParams p) {
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  const uint32_t nvec = (p.numel + 3) >> 2, step = gridDim.x * blockDim.x * U;
  for (uint32_t base = blockIdx.x * blockDim.x * U + threadIdx.x; base < nvec; base += step) {
    float v[4 * U];
    uint32_t row[U] = {}, col[U] = {};
    auto load = [&](int slot, int u, float* x) {
      const uint32_t f = (base + (uint32_t)u * blockDim.x) * 4;
      if ((p.dense >> slot) & 1) {
        if (f + 4 <= p.numel) {
          const float4 t = *reinterpret_cast<const float4*>(p.ptr[slot] + f);
          x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = f + e < p.numel ? p.ptr[slot][f + e] : 0.0f;
        }
      } else {
        uint32_t r = row[u], c = col[u];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[e] = f + e < p.numel ? __ldg(p.ptr[slot] + r * (uint32_t)p.stride_row[slot] + c * (uint32_t)p.stride_col[slot]) : 0.0f;
          if (++c == p.inner) { c = 0; ++r; }
        }
      }
    };
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + (uint32_t)u * blockDim.x;
      if (i < nvec) {
        row[u] = (uint32_t)(((uint64_t)(i * 4) * p.magic) >> p.shift);
        col[u] = i * 4 - row[u] * p.inner;
        load(p.chain.first_slot, u, v + 4 * u);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[4 * u + e] = 0.0f;
      }
    }
    for (int s = 0; s < p.chain.n; ++s) {
      const ChainStep st = p.chain.steps[s];
      float side[4 * U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int e = 0; e < 4; ++e) side[4 * u + e] = st.imm;
        if (st.slot >= 0 && base + (uint32_t)u * blockDim.x < nvec) load(st.slot, u, side + 4 * u);
      }
      chain_step<4 * U>(st.op, v, side);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t f = (base + (uint32_t)u * blockDim.x) * 4;
      float* out = p.ptr[p.chain.out_slot] + f;
      if (f + 4 <= p.numel) {
        *reinterpret_cast<float4*>(out) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (f + e < p.numel) out[e] = v[4 * u + e];
      }
    }
  }
}

// ---- tiled transpose + chain ----
struct EwTransposeParams {
  int rank;                      // 2..kVecRank
  int tdim;                      // the dim along which the first input is contiguous (!= rank - 1)
  int64_t shape[kVecRank];
  int64_t outer;                 // product of the dims other than tdim and the last
  DevOperand ops[KB200_MAX_OPERANDS];
  Chain chain;
};

__global__ void __launch_bounds__(256) ew_transpose_kernel(const __grid_constant__ EwTransposeParams p) {
  pdl_wait();                 // the producer of this kernel's inputs has completed
  pdl_launch_dependents();    // the next kernel may begin its start-up
  __shared__ float tile[32][33];
  const int last = p.rank - 1;
  const int64_t n_t = p.shape[p.tdim], n_l = p.shape[last];
  const int64_t tiles_l = (n_l + 31) / 32, tiles_t = (n_t + 31) / 32;
  const int64_t total = tiles_l * tiles_t * p.outer;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
  for (int64_t tile_id = blockIdx.x; tile_id < total; tile_id += gridDim.x) {
    int64_t rest = tile_id;
    const int64_t tl = rest % tiles_l; rest /= tiles_l;
    const int64_t tt = rest % tiles_t; rest /= tiles_t;
    int64_t idx[kVecRank] = {0, 0, 0, 0};
#pragma unroll
    for (int d = kVecRank - 1; d >= 0; --d) {
      if (d < p.rank && d != p.tdim && d != last) {
        idx[d] = rest % p.shape[d];
        rest /= p.shape[d];
      }
    }
    int64_t in_base = 0;
#pragma unroll
    for (int d = 0; d < kVecRank; ++d)
      if (d < p.rank) in_base += idx[d] * p.ops[p.chain.first_slot].stride[d];
    const int64_t s_t = p.ops[p.chain.first_slot].stride[p.tdim], s_l = p.ops[p.chain.first_slot].stride[last];
    // read: threads run along tdim (contiguous in the input)
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      int64_t it = tt * 32 + tx, il = tl * 32 + ty + j;
      if (it < n_t && il < n_l) tile[ty + j][tx] = p.ops[p.chain.first_slot].ptr[in_base + it * s_t + il * s_l];
    }
    __syncthreads();
    // write: threads run along the last dim (contiguous in the output)
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      int64_t it = tt * 32 + ty + j, il = tl * 32 + tx;
      if (it < n_t && il < n_l) {
        idx[p.tdim] = it;
        idx[last] = il;
        float v = tile[tx][ty + j];
        for (int s = 0; s < p.chain.n; ++s) {
          const ChainStep st = p.chain.steps[s];
          float side = st.imm;
          if (st.slot >= 0) {
            int64_t off = 0;
#pragma unroll
            for (int d = 0; d < kVecRank; ++d)
              if (d < p.rank) off += idx[d] * p.ops[st.slot].stride[d];
            side = p.ops[st.slot].ptr[off];
          }
          v = apply_chain(st.op, v, side);
        }
        int64_t off = 0;
#pragma unroll
        for (int d = 0; d < kVecRank; ++d)
          if (d < p.rank) off += idx[d] * p.ops[p.chain.out_slot].stride[d];
        p.ops[p.chain.out_slot].ptr[off] = v;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------

static bool chain_slots(const Chain& c, int* slots, int* n) {
  *n = 0;
  if (c.first_slot < 0) return false;
  slots[(*n)++] = c.first_slot;
  for (int s = 0; s < c.n; ++s)
    if (c.steps[s].slot >= 0) slots[(*n)++] = c.steps[s].slot;
  slots[(*n)++] = c.out_slot;
  return true;
}

int choose_elementwise(Plan& plan, PlanKernel& k) {
  (void)plan;
  const kb200_kernel_desc& d = k.desc;
  k.impl = IMPL_EW_GENERIC;
  k.launches = 1;
  k.has_chain = extract_chain(d, &k.chain);
  if (!k.has_chain || d.iter_rank > kVecRank) return KB200_OK;
  int slots[kMaxChain + 2], n_slots;
  if (!chain_slots(k.chain, slots, &n_slots)) return KB200_OK;
  const int last = d.iter_rank - 1;
  const int64_t inner = d.iter_shape[last];
  // a chain of accesses along the innermost dim: every operand contiguous or constant there, every
  // element offset (and stride) within the kernel's 32-bit arithmetic; float4 accesses where width,
  // strides and bases allow, else single elements
  bool chain = numel_of(d) < (int64_t(1) << 31), vec = inner % 4 == 0;
  for (int i = 0; i < n_slots && chain; ++i) {
    const DevOperand& o = k.ops[slots[i]];
    const bool is_out = slots[i] == k.chain.out_slot;
    int64_t span = 0;
    for (int dd = 0; dd <= last && chain; ++dd) {
      if (o.stride[dd] < 0) chain = false;
      span += (d.iter_shape[dd] - 1) * o.stride[dd];
    }
    if (span >= (int64_t(1) << 31)) chain = false;
    if (o.stride[last] == 1) {
      vec = vec && (reinterpret_cast<uintptr_t>(o.ptr) & 15) == 0;
      for (int dd = 0; dd < last && vec; ++dd) vec = o.stride[dd] % 4 == 0;
    } else if (o.stride[last] != 0 || is_out) {
      chain = false;         // (an operand that is constant along the row is fine)
    }
  }
  if (chain) {
    k.impl = vec ? IMPL_EW_CHAIN_VEC4 : IMPL_EW_CHAIN;
    return KB200_OK;
  }
  // transpose: output contiguous along the last dim, first input contiguous along another one
  const DevOperand& in = k.ops[k.chain.first_slot];
  const DevOperand& out = k.ops[k.chain.out_slot];
  if (d.iter_rank >= 2 && out.stride[last] == 1 && in.stride[last] != 1) {
    for (int t = 0; t < last; ++t) {
      if (in.stride[t] == 1 && d.iter_shape[t] >= 8 && inner >= 8) {
        k.impl = IMPL_EW_TRANSPOSE;
        k.x_slot = t;   // reused field: the input's contiguous dim
        return KB200_OK;
      }
    }
  }
  return KB200_OK;
}

template <int U, int VEC>
static void launch_chain(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  const kb200_kernel_desc& d = k.desc;
  EwChainParams p{};
  const int rank = d.iter_rank;
  for (int i = 0; i < rank; ++i) {
    p.shape[i] = (uint32_t)d.iter_shape[i];
    if (i == rank - 1) p.shape[i] /= VEC;
    int log = 0;
    while ((uint64_t(1) << log) < p.shape[i]) ++log;
    p.shift[i] = 31 + log;
    p.magic[i] = (uint32_t)(((uint64_t(1) << p.shift[i]) + p.shape[i] - 1) / p.shape[i]);
  }
  p.nvec = (uint32_t)(numel_of(d) / VEC);
  for (int o = 0; o < d.n_operands; ++o) {
    p.ptr[o] = k.ops[o].ptr;
    for (int i = 0; i < rank; ++i) p.stride[o][i] = (int32_t)(k.ops[o].stride[i] * (i == rank - 1 ? VEC : 1));
  }
  p.chain = k.chain;
  p.stream_out = streams_out(plan, k, k.chain.out_slot, numel_of(d)) ? 1 : 0;
  int64_t blocks = ((int64_t)p.nvec + 256 * U - 1) / (256 * U);
  // beyond the cap every block takes the same number of grid-stride steps (no ragged last wave)
  const int64_t cap = (int64_t)plan.sm_count * 64;
  const int64_t steps = (blocks + cap - 1) / cap;
  const unsigned grid = (unsigned)((blocks + steps - 1) / (steps > 0 ? steps : 1));
  switch (rank) {
    case 1: launch_kernel(plan.pdl, ew_chain_kernel<1, U, VEC>, dim3(grid), dim3(256), 0, s, p); break;
    case 2: launch_kernel(plan.pdl, ew_chain_kernel<2, U, VEC>, dim3(grid), dim3(256), 0, s, p); break;
    case 3: launch_kernel(plan.pdl, ew_chain_kernel<3, U, VEC>, dim3(grid), dim3(256), 0, s, p); break;
    default: launch_kernel(plan.pdl, ew_chain_kernel<4, U, VEC>, dim3(grid), dim3(256), 0, s, p); break;
  }
}

// Does ew_flat_kernel take this chain (already known to fit 32-bit offsets)?
static bool flat_ok(const PlanKernel& k) {
  const kb200_kernel_desc& d = k.desc;
  if (d.iter_rank != 2 || numel_of(d) > (int64_t(1) << 30)) return false;
  for (int slot : {k.chain.first_slot, k.chain.out_slot}) {
    const DevOperand& o = k.ops[slot];
    if (o.stride[1] != 1 || o.stride[0] != d.iter_shape[1] || (reinterpret_cast<uintptr_t>(o.ptr) & 15)) return false;
  }
  return true;
}

static void launch_flat(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  const kb200_kernel_desc& d = k.desc;
  EwFlatParams p{};
  p.numel = (uint32_t)numel_of(d);
  p.inner = (uint32_t)d.iter_shape[1];
  int log = 0;
  while ((uint64_t(1) << log) < p.inner) ++log;
  p.shift = 31 + log;
  p.magic = (uint32_t)(((uint64_t(1) << p.shift) + p.inner - 1) / p.inner);
  for (int o = 0; o < d.n_operands; ++o) {
    const DevOperand& op = k.ops[o];
    p.ptr[o] = op.ptr;
    p.stride_row[o] = (int32_t)op.stride[0];
    p.stride_col[o] = (int32_t)op.stride[1];
    if (op.stride[1] == 1 && op.stride[0] == d.iter_shape[1] && (reinterpret_cast<uintptr_t>(op.ptr) & 15) == 0) p.dense |= 1u << o;
  }
  p.chain = k.chain;
  constexpr int U = 2;
  const int64_t blocks = ((int64_t)p.numel + 1024 * U - 1) / (1024 * U), cap = (int64_t)plan.sm_count * 64;
  const int64_t steps = (blocks + cap - 1) / cap;
  launch_kernel(plan.pdl, ew_flat_kernel<U>, dim3((unsigned)((blocks + steps - 1) / (steps > 0 ? steps : 1))), dim3(256), 0, s, p);
}

int launch_elementwise(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  const kb200_kernel_desc& d = k.desc;
  const int64_t numel = numel_of(d);
  if (k.impl == IMPL_EW_CHAIN_VEC4) {
    launch_chain<2, 4>(plan, k, s);
  } else if (k.impl == IMPL_EW_CHAIN) {
    if (flat_ok(k)) launch_flat(plan, k, s);
    else launch_chain<8, 1>(plan, k, s);
  } else if (k.impl == IMPL_EW_TRANSPOSE) {
    EwTransposeParams p{};
    p.rank = d.iter_rank;
    p.tdim = k.x_slot;
    p.outer = 1;
    for (int i = 0; i < d.iter_rank; ++i) {
      p.shape[i] = d.iter_shape[i];
      if (i != p.tdim && i != d.iter_rank - 1) p.outer *= d.iter_shape[i];
    }
    for (int o = 0; o < d.n_operands; ++o) p.ops[o] = k.ops[o];
    p.chain = k.chain;
    int64_t tiles = ((p.shape[p.tdim] + 31) / 32) * ((p.shape[p.rank - 1] + 31) / 32) * p.outer;
    int64_t cap = (int64_t)plan.sm_count * 16;
    launch_kernel(plan.pdl, ew_transpose_kernel, dim3((unsigned)(tiles < cap ? tiles : cap)), dim3(256), 0, s, p);
  } else {
    EwParams p{};
    p.rank = d.iter_rank;
    p.n_operands = d.n_operands;
    p.numel = numel;
    for (int i = 0; i < d.iter_rank; ++i) p.shape[i] = d.iter_shape[i];
    for (int o = 0; o < d.n_operands; ++o) p.ops[o] = k.ops[o];
    p.tape = k.tape;
    int64_t blocks = (numel + 255) / 256;
    int64_t cap = (int64_t)plan.sm_count * 8;
    launch_kernel(plan.pdl, ew_generic_kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), dim3(256), 0, s, p);
  }
  KB200_CUDA(cudaGetLastError());
  return KB200_OK;
}

}  // namespace kb200
