// lane_pass.cu -- the lane-pass kernels of one precision and gas shape
// (single-ion and batched launches).  The build compiles it once per
// CCS_PASS_T (float, double) and CCS_PASS_GAS (0 atom, 1 N2, 2 CO2), in
// parallel; the kernels themselves are in ccs_device.cuh.
#include <cuda_runtime.h>

#include "engine_ctx.h"

using namespace ccs;

namespace {
template <typename T, int GAS, bool HASQ> ccs_internal::KernelFn lane_g(int G) {
  switch (G) {
    case 1: return traj_kernel<T, 1, GAS, HASQ, false>;
    case 4: return traj_kernel<T, 4, GAS, HASQ, false>;
    case 8: return traj_kernel<T, 8, GAS, HASQ, false>;
    case 16: return traj_kernel<T, 16, GAS, HASQ, false>;
    default: return traj_kernel<T, 32, GAS, HASQ, false>;
  }
}
template <typename T, int GAS, bool HASQ> ccs_internal::KernelFn lane_batch_g(int G) {
  return G <= 8 ? traj_kernel<T, 8, GAS, HASQ, true>
                : G == 16 ? traj_kernel<T, 16, GAS, HASQ, true> : traj_kernel<T, 32, GAS, HASQ, true>;
}
}  // namespace

template <>
ccs_internal::KernelFn ccs_internal::lane_kernel<CCS_PASS_T, CCS_PASS_GAS>(bool hasq, int G, bool batch) {
  if (batch) return hasq ? lane_batch_g<CCS_PASS_T, CCS_PASS_GAS, true>(G) : lane_batch_g<CCS_PASS_T, CCS_PASS_GAS, false>(G);
  return hasq ? lane_g<CCS_PASS_T, CCS_PASS_GAS, true>(G) : lane_g<CCS_PASS_T, CCS_PASS_GAS, false>(G);
}
