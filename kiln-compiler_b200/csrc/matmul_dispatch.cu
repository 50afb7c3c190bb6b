// Which matmul kernel runs a descriptor: exact-FP32 SIMT tiles, the decode GEMV, or tcgen05 tiles.
#include "kb200_internal.h"
#include "matmul.h"

namespace kb200 {

bool tc_eligible(const PlanKernel& k);
int tc_bind(Plan& plan, PlanKernel& k, int kernel_index);
int tc_launch(const Plan& plan, const PlanKernel& k, cudaStream_t s);
void tc_destroy(PlanKernel& k);
bool tc_repoint(PlanKernel& k);
std::string tc_detail(const PlanKernel& k);
bool tc_writes_tails(const PlanKernel& k);
bool tc_takes_planes(const PlanKernel& k, PlanKernel::Planes* planes);
void tc_planes_come_ready(PlanKernel& k);
bool tc_write_pairs(PlanKernel& k, const PlanKernel::Planes& to, const float* scale, bool store32);

int choose_matmul(Plan& plan, PlanKernel& k) {
  (void)plan;
  const kb200_kernel_desc& d = k.desc;
  k.has_chain = extract_chain(d, &k.chain) && k.chain.first_slot == -1;
  k.impl = IMPL_MM_SIMT;
  k.launches = 1;
  const DevOperand& B = k.ops[d.b_slot];
  const int forced = d.cfg[5];   // 0 auto, 1 simt, 2 tc, 3 gemv
  if ((forced == 0 || forced == 3) && k.M == 1 && B.stride[2] == 1) {
    // (single floats, a warp along a row of B: rows may begin anywhere; 1 x 2355 x 152 took 13.2 us in the SIMT tiles, 7.7 here)
    k.impl = IMPL_MM_GEMV;
    return KB200_OK;
  }
  if ((forced == 0 || forced == 2) && tc_eligible(k)) k.impl = IMPL_MM_TC;
  if (forced == 2 && k.impl != IMPL_MM_TC)
    return fail(KB200_ERR_UNSUPPORTED, "matmul %s: the tensor-core kernel cannot take these operands", d.name);
  return KB200_OK;
}

int bind_matmul(Plan& plan, PlanKernel& k) {
  if (k.impl != IMPL_MM_TC) return KB200_OK;
  return tc_bind(plan, k, (int)(&k - plan.kernels.data()));
}

int launch_matmul(const Plan& plan, const PlanKernel& k, cudaStream_t s) {
  if (k.impl == IMPL_MM_TC) return tc_launch(plan, k, s);
  return launch_matmul_simt(plan, k, s);
}

bool repoint_matmul(PlanKernel& k) { return tc_repoint(k); }

std::string matmul_detail(const PlanKernel& k) { return tc_detail(k); }

bool matmul_takes_planes(const PlanKernel& k, PlanKernel::Planes* planes) { return k.impl == IMPL_MM_TC && tc_takes_planes(k, planes); }
void matmul_planes_come_ready(PlanKernel& k) { tc_planes_come_ready(k); }
bool matmul_write_pairs(PlanKernel& k, const PlanKernel::Planes& to, const float* scale, bool store32) {
  return k.impl == IMPL_MM_TC && tc_write_pairs(k, to, scale, store32);
}
bool matmul_writes_tails(const PlanKernel& k) { return k.impl == IMPL_MM_TC && tc_writes_tails(k); }

void destroy_matmul(PlanKernel& k) { tc_destroy(k); }

}  // namespace kb200
