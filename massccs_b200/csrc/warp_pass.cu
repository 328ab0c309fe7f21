// warp_pass.cu -- the warp-pass kernels of one precision and gas shape
// (single-ion and batched launches), compiled like lane_pass.cu.
#include <cuda_runtime.h>

#include "engine_ctx.h"
#include "warp_pass.cuh"

using namespace ccs;

namespace {
template <typename T, int GAS, bool HASQ, int NT, bool BATCH> ccs_internal::WarpKernel warp_k() {
  return {warp_pass_kernel<T, GAS, HASQ, NT, BATCH>, WarpShape<T, GAS, HASQ, NT>::THREADS};
}
template <typename T, int GAS, bool HASQ> ccs_internal::WarpKernel warp_nt(int nt, bool batch) {
  if (batch) return warp_k<T, GAS, HASQ, RBLOCK, true>();
  return nt == 32 ? warp_k<T, GAS, HASQ, 32, false>()
                  : nt == 64 ? warp_k<T, GAS, HASQ, 64, false>() : warp_k<T, GAS, HASQ, 128, false>();
}
}  // namespace

template <>
ccs_internal::WarpKernel ccs_internal::warp_kernel<CCS_PASS_T, CCS_PASS_GAS>(bool hasq, int nt, bool batch) {
  return hasq ? warp_nt<CCS_PASS_T, CCS_PASS_GAS, true>(nt, batch) : warp_nt<CCS_PASS_T, CCS_PASS_GAS, false>(nt, batch);
}
