// Counts the floats with bit patterns lo..hi whose sqrt_mid (warp_pass.cuh)
// is not the rounded square root, and reports the first of them.
#include "warp_pass.cuh"

__global__ void compare(unsigned lo, unsigned hi, unsigned long long *bad, unsigned *first) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = lo + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i <= hi; i += stride) {
    const float x = __uint_as_float((unsigned)i);
    if (__float_as_uint(ccs::sqrt_mid(x)) != __float_as_uint(__fsqrt_rn(x))) {
      atomicAdd(bad, 1ull);
      atomicMin(first, (unsigned)i);
    }
  }
}

extern "C" int sqrt_mid_mismatches(float lo, float hi, unsigned long long *count, float *first) {
  unsigned long long *bad = nullptr;
  unsigned *at = nullptr, ulo, uhi, hat = 0;
  if (cudaMalloc(&bad, sizeof *bad) || cudaMalloc(&at, sizeof *at)) return 1;
  memcpy(&ulo, &lo, 4);
  memcpy(&uhi, &hi, 4);
  if (cudaMemset(bad, 0, sizeof *bad) || cudaMemset(at, 0xff, sizeof *at)) return 2;
  compare<<<1024, 256>>>(ulo, uhi, bad, at);
  if (cudaGetLastError() || cudaMemcpy(count, bad, sizeof *bad, cudaMemcpyDeviceToHost) ||
      cudaMemcpy(&hat, at, sizeof hat, cudaMemcpyDeviceToHost))
    return 3;
  memcpy(first, &hat, 4);
  cudaFree(bad);
  cudaFree(at);
  return 0;
}
