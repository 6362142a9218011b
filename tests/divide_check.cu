// Counts the operands for which csrc/rrtmg_divide.cuh differs from IEEE division.
#include <cuda_runtime.h>

#include <cstdint>

#include "rrtmg_divide.cuh"

namespace {

__device__ unsigned long long g_bad[2];

__device__ __forceinline__ float binary32(int exponent, unsigned significand) {
  return __uint_as_float((static_cast<unsigned>(exponent + 127) << 23) | significand);
}

// every significand at the exponents [e0, e1)
__global__ void reciprocals(int e0, int e1) {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= (1u << 23)) return;
  unsigned bad = 0;
  for (int e = e0; e < e1; ++e) {
    const float b = binary32(e, m);
    bad += __float_as_uint(rrtmg::recip_in_range(b)) != __float_as_uint(__frcp_rn(b));
    bad += __float_as_uint(rrtmg::recip_in_range(-b)) != __float_as_uint(__frcp_rn(-b));
  }
  if (bad) atomicAdd(&g_bad[0], static_cast<unsigned long long>(bad));
}

__device__ __forceinline__ uint64_t next(uint64_t &s) {  // xorshift64
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}

// random operands over the whole ranges of rrtmg_divide.cuh, of either sign,
// among them significands near 2 and near 1, quotients next to the midpoint of
// two neighbours, and numerators, divisors and quotients at the ranges' ends
__global__ void quotients(int n, uint64_t seed) {
  uint64_t s = seed + (blockIdx.x * blockDim.x + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull;
  unsigned bad = 0;
  for (int i = 0; i < n; ++i) {
    const uint64_t r = next(s) >> 8, x = next(s) >> 16;
    unsigned ma = static_cast<unsigned>(r >> 23) & 0x7fffffu, mb = static_cast<unsigned>(r) & 0x7fffffu;
    if ((i & 3) == 1) mb |= 0x7fff00u;
    if ((i & 3) == 2) ma &= 0xffu;
    int eb = static_cast<int>(x % 200) - 100, ea = static_cast<int>(x / 200 % 200) - 100;
    if ((i & 28) == 4) eb = i & 32 ? 99 : -100;
    if ((i & 28) == 8) ea = i & 32 ? 99 : -100;
    if ((i & 28) == 12) eb = ea + 119;  // the smallest quotients
    if ((i & 28) == 16) eb = ea - 117;  // the largest
    if (eb < -100 || eb > 99 || ea - eb < -119 || ea - eb > 117) continue;
    const float b = x >> 40 & 1u ? -binary32(eb, mb) : binary32(eb, mb);
    float a = x >> 41 & 1u ? -binary32(ea, ma) : binary32(ea, ma);
    if ((i & 3) == 3) a = static_cast<float>(static_cast<double>(__fdiv_rn(a, b)) * (1.0 + 0x1p-24) * b);
    if (fabsf(a) < 0x1p-100f) continue;
    if (i == 0) a = 0.0f;
    bad += __float_as_uint(rrtmg::quotient_in_range(a, b)) != __float_as_uint(__fdiv_rn(a, b));
  }
  if (bad) atomicAdd(&g_bad[1], static_cast<unsigned long long>(bad));
}

}  // namespace

extern "C" int divide_check(int e0, int e1, int quotients_per_thread, unsigned long long *bad) {
  const unsigned long long zero[2] = {0, 0};
  cudaError_t e = cudaMemcpyToSymbol(g_bad, zero, sizeof(zero));
  if (e != cudaSuccess) return static_cast<int>(e);
  reciprocals<<<(1 << 23) / 256, 256>>>(e0, e1);
  quotients<<<148 * 16, 256>>>(quotients_per_thread, 77);
  e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(bad, g_bad, sizeof(zero));
  return static_cast<int>(e);
}
