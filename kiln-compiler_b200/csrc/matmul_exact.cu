// Exact FP32 on SM pairs: which matmuls, tile widths, launches.  The kernel and why it is built as it is: matmul_exact.cuh.
#include <cuda.h>

#include "kb200_internal.h"
#include "matmul_exact.cuh"
#include "matmul_exact.h"

namespace kb200 {

namespace {

using ExactKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, ExactParams);

template <int BLOCKS, bool SPLIT>
ExactKernel exact_kernel(int fin) {
  switch (fin) {
    case FIN_BIAS: return mm_exact_kernel<BLOCKS, FIN_BIAS, SPLIT>;
    case FIN_BIAS_GELU: return mm_exact_kernel<BLOCKS, FIN_BIAS_GELU, SPLIT>;
    case FIN_BIAS_RES: return mm_exact_kernel<BLOCKS, FIN_BIAS_RES, SPLIT>;
    default: return mm_exact_kernel<BLOCKS, FIN_NONE, SPLIT>;
  }
}

struct ExactState {
  CUtensorMap map_a, map_b, map_out, map_res, map_tail;
  ExactParams params;
  ExactKernel kernel = nullptr;
  size_t smem = 0;
  unsigned grid = 0;
  int parts = 1;                         // of K
  int bias_slot = -1, res_slot = -1;
};

// The chains that are finished here: nothing, + column, + column then GELU, + column + matrix, all of it in float4 and 16-byte rows.
int finish_of(const PlanKernel& k, int* bias_slot, int* res_slot) {
  const Chain& c = k.chain;
  *bias_slot = *res_slot = -1;
  if (c.n == 0) return FIN_NONE;
  const ChainStep* s = c.steps;
  if (s[0].op != CH_ADD || s[0].slot < 0) return -1;
  const DevOperand& b = k.ops[s[0].slot];
  if (b.stride[1] != 0 || b.stride[2] != 1 || !aligned16(b.ptr)) return -1;
  *bias_slot = s[0].slot;
  if (c.n == 1) return FIN_BIAS;
  if (c.n != 2) return -1;
  if (s[1].op == CH_GELU_TANH) return FIN_BIAS_GELU;
  if (s[1].op != CH_ADD || s[1].slot < 0) return -1;
  const DevOperand& r = k.ops[s[1].slot];
  if (r.stride[2] != 1 || r.stride[1] < k.N || r.stride[1] % 4 || !aligned16(r.ptr)) return -1;
  *res_slot = s[1].slot;
  return FIN_BIAS_RES;
}

// Clusters of `parts` pairs that fit the GPU at once.
int resident_parts(const Plan& plan, int parts) {
  int& known = plan.resident_exact_parts[parts];
  if (known == 0) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(plan.sm_count / (2 * parts) * 2 * parts), 1, 1);
    cfg.blockDim = dim3(kExactThreads, 1, 1);
    cfg.dynamicSmemBytes = kExactSmem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2 * parts;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const ExactKernel kernel = mm_exact_kernel<2, FIN_BIAS, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kExactSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known = n > 0 ? n : -1;
  }
  return known;
}

struct ExactPlan { int bn, parts; int64_t cycles; };

// Tile width, parts of K and estimated cycles, the pass over A included: all that runs once, the steps of the rounds, what
// they cost more the more of the pairs are at work, and per round its drain.  Lines through 419 launches, and 336 for the parts of K: 160 to 4096 rows of
// eleven weights from 256 x 1024 to 4096 x 1024, every width timed (2 to 4 % off in the mean square); the choice is 0.2 % from the best on average.
// us with two, three and four parts: 333 x 768 x 3072 17.6, 15.2, 14.3 (26.7 in one); 512 x 768 x 3072 18.1, 16.0, 15.2; 1024 x 512 x 2048 15.7, 14.3.  (Of
// 24 tiles the clusters of three pairs do not all fit at once: 1024 x 768 x 3072 keeps halves.)  (A
// step of 256 columns has 1536 cycles of multiplying, of 128 columns 768, and the operands come in at 48 KB: 1024 x 2304 x 768 16.3 us at 128
// columns, 19.9 at 256; 4096 x 3072 x 768 54.1 at 256.)  Plans in flight are no argument: results must not depend on them.
struct ExactWidth { int bn, once, step, busy, drain; };
constexpr ExactWidth kExactWidths[] = {{256, 11060, 1497, 574, 4516}, {192, 11050, 1092, 496, 3039}, {160, 9770, 910, 342, 3575}, {128, 10565, 705, 374, 2543}};
// K in two, three and four parts on as many times the pairs
constexpr ExactWidth kExactParts[] = {{128, 12915, 706, 259, 1945}, {128, 12823, 736, 214, 3606}, {128, 10919, 625, 406, 7082}};

// (Of all that runs once, ~4300 are the pass, which a producer that splits A's rows takes over: 1024 x 2304 x 768 16.3 -> 13.0 us.)
ExactPlan plan_exact(const Plan& plan, int64_t m, int64_t n, int64_t k, bool split) {
  const int64_t pairs = plan.sm_count / 2, steps = (k + kExactStepK - 1) / kExactStepK, pass = split ? -4300 : m * k / 714;
  ExactPlan best{0, 1, 0};
  for (const ExactWidth& w : kExactWidths) {
    if (w.bn > 128 && w.bn / 2 >= n) continue;
    const int64_t tiles = ((m + 255) / 256) * ((n + w.bn - 1) / w.bn), rounds = (tiles + pairs - 1) / pairs;
    const int64_t cycles = w.once + pass + rounds * (steps * w.step + w.drain) + steps * w.busy * tiles / pairs;
    if (best.bn == 0 || cycles < best.cycles) best = {w.bn, 1, cycles};
  }
  for (int parts = 2; parts <= 4; ++parts) {
    const ExactWidth& h = kExactParts[parts - 2];
    const int64_t tiles = ((m + 255) / 256) * ((n + h.bn - 1) / h.bn), part = (steps + parts - 1) / parts;
    if (steps < 2 * parts || tiles * parts > pairs || tiles > resident_parts(plan, parts)) continue;
    const int64_t cycles = h.once + pass + part * h.step + (part * h.busy + h.drain) * parts * tiles / pairs;
    if (cycles < best.cycles) best = {h.bn, parts, cycles};
  }
  return best;
}

ExactKernel kernel_for(const ExactPlan& how, int fin) {
  return how.parts > 1 ? exact_kernel<2, true>(fin) : how.bn > 192 ? exact_kernel<4, false>(fin) : how.bn > 128 ? exact_kernel<3, false>(fin) : exact_kernel<2, false>(fin);
}

}  // namespace

int64_t exact_cycles(const Plan& plan, const PlanKernel& k) {
  const kb200_kernel_desc& d = k.desc;
  int bias_slot, res_slot;
  if (!k.has_chain || k.batch != 1 || k.M <= 128 || k.N < 128 || k.N % 4 || finish_of(k, &bias_slot, &res_slot) < 0) return -1;
  for (int i : {0, 1, 2, 3, 4, 6})
    if (d.cfg[i] != 0) return -1;                      // a tile, stage or split was asked for
  if (((k.M + 255) / 256) * ((k.N + 127) / 128) >= (int64_t(1) << 20) || k.K >= (int64_t(1) << 24)) return -1;
  const DevOperand& O = k.ops[k.chain.out_slot];
  if (O.stride[2] != 1 || O.stride[1] % 4 || O.stride[1] < k.N || !aligned16(O.ptr)) return -1;
  return plan_exact(plan, k.M, k.N, k.K, k.planes_expected).cycles;
}

int exact_runs(const Plan& plan, const PlanKernel& k, bool* runs) {
  int bias_slot, res_slot;
  cudaFuncAttributes attributes;
  KB200_CUDA(cudaFuncGetAttributes(&attributes, kernel_for(plan_exact(plan, k.M, k.N, k.K, k.planes_expected), finish_of(k, &bias_slot, &res_slot))));
  *runs = attributes.numRegs == 168;
  return KB200_OK;
}

int exact_bind(Plan& plan, PlanKernel& k, int kernel_index, const ExactOperands& ops, void** state) {
  *state = nullptr;
  const kb200_kernel_desc& d = k.desc;
  ExactState* st = new ExactState();
  ExactParams& p = st->params;
  const ExactPlan how = plan_exact(plan, k.M, k.N, k.K, k.planes_expected);
  const int fin = finish_of(k, &st->bias_slot, &st->res_slot);
  p.bn = how.bn;
  p.half_bn = how.bn / 2;
  st->parts = p.parts = how.parts;
  p.steps = (int)((k.K + kExactStepK - 1) / kExactStepK);
  p.sums = 512 / how.bn < kExactMaxSums ? 512 / how.bn : kExactMaxSums;
  const int stage_bytes = 2 * (kExactABytes + p.half_bn * 128), rest = kExactWarps * kExactSlot;
  p.stages = (kExactSmem - rest) / stage_bytes < kExactMaxStages ? (kExactSmem - rest) / stage_bytes : kExactMaxStages;
  st->smem = (size_t)p.stages * stage_bytes + rest;
  // D = F32, A and B = F16, both K-major, N = bn, M = 256 over the pair
  p.idesc = (1u << 4) | ((uint32_t)(p.bn >> 3) << 17) | ((256u >> 4) << 24);
  p.tiles_n = (int)((k.N + p.bn - 1) / p.bn);
  p.num_tiles = (int)((k.M + 255) / 256) * p.tiles_n;
  p.magic_tn = ((uint64_t(1) << 40) + p.tiles_n - 1) / p.tiles_n;
  p.kernel_index = kernel_index;
  p.status = plan.d_status;
  p.M = (int)k.M;
  p.N = (int)k.N;
  p.a_scale = ops.a_scale;
  p.b_scale = ops.b_scale;
  p.a_marks = ops.a_marks;
  p.bias = st->bias_slot >= 0 ? k.ops[st->bias_slot].ptr : nullptr;
  p.res = st->res_slot >= 0 ? k.ops[st->res_slot].ptr : nullptr;
  p.res_row = st->res_slot >= 0 ? k.ops[st->res_slot].stride[1] : 0;
  p.a = k.ops[d.a_slot].ptr;
  p.a_row = k.ops[d.a_slot].stride[1];
  p.b = k.ops[d.b_slot].ptr;
  p.b_k = k.ops[d.b_slot].stride[1];
  p.b_n = k.ops[d.b_slot].stride[2];
  p.K = k.K;
  p.stream_out = streams_out(plan, k, k.chain.out_slot, k.M * k.N) ? 1 : 0;
  const DevOperand& O = k.ops[k.chain.out_slot];
  p.with_tail = k.tail_out != nullptr ? 1 : 0;
  p.pair_scale = nullptr;
  p.store32 = 1;
  // Persistent pairs, up to this plan's share of the GPU with several in flight.
  const int pairs = plan.sm_count / 2, share = plan.concurrency > 1 && pairs / plan.concurrency > 0 ? pairs / plan.concurrency : pairs;
  const int rounds = (p.num_tiles + share - 1) / share;
  st->grid = (unsigned)(st->parts > 1 ? 2 * st->parts * p.num_tiles : 2 * ((p.num_tiles + rounds - 1) / rounds));
  bool ok = encode_map(&st->map_a, true, ops.a, k.K, k.M, 2 * kLevels, ops.pitch, k.M * ops.pitch, kExactStepK, 128, false, 2) &&
            encode_map(&st->map_b, true, ops.b, k.K, k.N, 2, ops.pitch, k.N * ops.pitch, kExactStepK, p.half_bn, false, 2) &&
            encode_map_store(&st->map_out, false, O.ptr, k.N, k.M, 1, O.stride[1], 0);
  st->map_res = st->map_tail = st->map_out;
  if (ok && p.res) ok = encode_map_store(&st->map_res, false, p.res, k.N, k.M, 1, p.res_row, 0);
  if (ok && p.with_tail) ok = set_map_address(&st->map_tail, k.tail_out);
  if (!ok) { delete st; return KB200_OK; }
  st->kernel = kernel_for(how, fin);
  const cudaError_t e = cudaFuncSetAttribute(st->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kExactSmem);
  if (e != cudaSuccess) { delete st; return cuda_fail(e, "cudaFuncSetAttribute(mm_exact_kernel)"); }
  *state = st;
  return KB200_OK;
}

int exact_launch(const Plan& plan, const void* state, cudaStream_t s) {
  const ExactState* st = static_cast<const ExactState*>(state);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(st->grid, 1, 1);
  cfg.blockDim = dim3(kExactThreads, 1, 1);
  cfg.dynamicSmemBytes = st->smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * st->parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = plan.pdl ? 2 : 1;
  KB200_CUDA(cudaLaunchKernelEx(&cfg, st->kernel, st->map_a, st->map_b, st->map_out, st->map_res, st->map_tail, st->params));
  return KB200_OK;
}

bool exact_repoint(const PlanKernel& k, void* state) {
  ExactState* st = static_cast<ExactState*>(state);
  st->params.a = k.ops[k.desc.a_slot].ptr;
  if (st->bias_slot >= 0) st->params.bias = k.ops[st->bias_slot].ptr;
  if (st->res_slot >= 0) st->params.res = k.ops[st->res_slot].ptr;
  return set_map_address(&st->map_out, k.ops[k.chain.out_slot].ptr) && (st->res_slot < 0 || set_map_address(&st->map_res, k.ops[st->res_slot].ptr));
}

std::string exact_detail(const void* state) {
  const ExactState* st = static_cast<const ExactState*>(state);
  return "mm_exact " + std::to_string(st->params.bn) + " columns" + (st->parts > 1 ? ", " + std::to_string(st->parts) + " splits" : "");
}

bool exact_write_pairs(const PlanKernel& k, void* state, const PlanKernel::Planes& to, const float* scale, bool store32) {
  ExactState* st = static_cast<ExactState*>(state);
  if (st->params.with_tail || st->res_slot >= 0 ||
      !encode_map_store(&st->map_tail, true, to.heads, k.N, k.M, 2, to.pitch, to.plane))
    return false;
  st->params.pair_scale = scale;
  st->params.store32 = store32 ? 1 : 0;
  return true;
}

bool exact_writes_tails(const void* state) { return static_cast<const ExactState*>(state)->params.with_tail != 0; }

void exact_destroy(void* state) { delete static_cast<ExactState*>(state); }

}  // namespace kb200
