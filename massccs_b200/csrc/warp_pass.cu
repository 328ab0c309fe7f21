// warp_pass.cu -- the warp-pass kernels of one precision and gas shape
// (single-ion and batched launches), compiled like lane_pass.cu.
#include <cuda_runtime.h>

#include "engine_ctx.h"

using namespace ccs;

namespace {
template <typename T, int GAS, bool HASQ> ccs_internal::KernelFn warp_nt(int nt, bool batch) {
  if (batch) return resume_kernel<T, GAS, HASQ, RBLOCK, true>;
  return nt == 32 ? resume_kernel<T, GAS, HASQ, 32, false>
                  : nt == 64 ? resume_kernel<T, GAS, HASQ, 64, false> : resume_kernel<T, GAS, HASQ, 128, false>;
}
}  // namespace

template <>
ccs_internal::KernelFn ccs_internal::warp_kernel<CCS_PASS_T, CCS_PASS_GAS>(bool hasq, int nt, bool batch) {
  return hasq ? warp_nt<CCS_PASS_T, CCS_PASS_GAS, true>(nt, batch) : warp_nt<CCS_PASS_T, CCS_PASS_GAS, false>(nt, batch);
}
