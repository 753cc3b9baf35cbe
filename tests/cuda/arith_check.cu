// Test kernels: sph::sqrt_rn and sph::rcp_rn against CUDA's IEEE operations
// over every float in [lo, hi], and sph::div_rn over pairs (a, b) whose
// mantissas run over all of a's for a set of b's.
#include "sph_kernels.cuh"

__global__ void k_unary(uint32_t u0, uint32_t u1, unsigned long long* bad) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long s = 0, r = 0;
  for (uint64_t u = u0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= u1; u += stride) {
    const float x = __uint_as_float((uint32_t)u);
    s += __float_as_uint(sph::sqrt_rn(x)) != __float_as_uint(__fsqrt_rn(x));
    r += __float_as_uint(sph::rcp_rn(x)) != __float_as_uint(__frcp_rn(x));
  }
  atomicAdd(&bad[0], s);
  atomicAdd(&bad[1], r);
}

__global__ void k_div(const float* b, int nb, float scale, unsigned long long* bad) {
  const uint32_t stride = gridDim.x * blockDim.x;
  unsigned long long s = 0;
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 23); m += stride) {
    const float a = __uint_as_float(0x3f800000u | m) * scale;
    for (int j = 0; j < nb; ++j)
      s += __float_as_uint(sph::div_rn(a, b[j])) != __float_as_uint(__fdiv_rn(a, b[j]));
  }
  atomicAdd(&bad[2], s);
}

// mismatches[0..2]: square roots and reciprocals over [lo, hi], quotients over b[nb] and dividends scale * [1, 2)
extern "C" int arith_check(float lo, float hi, const float* b, int nb, float scale, unsigned long long* mismatches) {
  unsigned long long* d_bad = nullptr;
  float* d_b = nullptr;
  if (cudaMalloc(&d_bad, 3 * sizeof(*d_bad)) != cudaSuccess) return 1;
  if (cudaMalloc(&d_b, (nb > 0 ? nb : 1) * sizeof(float)) != cudaSuccess) return 1;
  cudaMemset(d_bad, 0, 3 * sizeof(*d_bad));
  cudaMemcpy(d_b, b, nb * sizeof(float), cudaMemcpyHostToDevice);
  uint32_t u0, u1;
  memcpy(&u0, &lo, 4);
  memcpy(&u1, &hi, 4);
  k_unary<<<148 * 8, 256>>>(u0, u1, d_bad);
  k_div<<<148 * 8, 256>>>(d_b, nb, scale, d_bad);
  cudaError_t e = cudaDeviceSynchronize();
  cudaMemcpy(mismatches, d_bad, 3 * sizeof(*d_bad), cudaMemcpyDeviceToHost);
  cudaFree(d_bad);
  cudaFree(d_b);
  return e == cudaSuccess ? 0 : 2;
}
