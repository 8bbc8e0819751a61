// Every mantissa vlog can meet: the quotient its refined reciprocal gives
// against the rounded division.  Prints the number that differ.
#include <cstdio>

#include "vcr_math.cuh"

__global__ void count(unsigned long long* bad) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (1u << 23); i += gridDim.x * blockDim.x) {
    float m = vcr::u2f(i | 0x3F800000u);
    if (m > 1.41421356f) m = m * 0.5f;
    const float a = m - 1.0f, b = m + 1.0f;
    if (vcr::f2u(vcr::vlog_div(a, b)) != vcr::f2u(__fdiv_rn(a, b))) atomicAdd(bad, 1ull);
  }
}

int main() {
  unsigned long long *d = nullptr, h = 1;
  if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 1;
  count<<<512, 256>>>(d);
  if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  printf("%llu\n", h);
  return 0;
}
