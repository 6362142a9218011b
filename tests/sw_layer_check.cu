// Counts the operands for which the shortwave layer optics of csrc/rrtmg_sw.cu
// with checked divisions differ from their general form.
#include <cstdint>
#include <vector>

#include "rrtmg_sw.cu"

namespace rrtmg {
namespace {

__device__ unsigned long long g_bad[2];  // clear sky, cloudy

__device__ __forceinline__ uint64_t next(uint64_t &s) {  // xorshift64
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}

__device__ __forceinline__ float uniform(uint64_t &s) { return static_cast<float>(next(s) >> 40) * 0x1p-24f; }

// 2^e (1 + f), e drawn from [lo, hi]
__device__ __forceinline__ float spread(uint64_t &s, int lo, int hi) {
  const int e = lo + static_cast<int>((next(s) >> 33) % static_cast<unsigned>(hi - lo + 1));
  return ldexpf(1.0f + uniform(s), e);
}

__device__ __forceinline__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a == 0.0f && b == 0.0f) || (a != a && b != b);
}

__device__ __forceinline__ bool same(const SwOptics &a, const SwOptics &b) {
  return same(a.rt.ref, b.rt.ref) && same(a.rt.refd, b.rt.refd) && same(a.rt.tra, b.rt.tra) &&
         same(a.rt.trad, b.rt.trad) && same(a.dbt, b.dbt) && same(a.dbt_nd, b.dbt_nd);
}

// ends: operands up to and beyond the ends of the ranges that the checked form accepts
__global__ void layers(const __grid_constant__ Tables T, int n, int ends, uint64_t seed) {
  uint64_t s = seed + (blockIdx.x * blockDim.x + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull;
  unsigned bad_clear = 0, bad_cloudy = 0;
  for (int i = 0; i < n; ++i) {
    float tr = spread(s, -20, 0), tg = spread(s, -30, 12), mu = 1.0e-10f + uniform(s);
    float4 cld = make_float4(spread(s, -20, 8), 1.0f - spread(s, -24, -2), 0.99f * uniform(s), 0.0f);
    if (ends) {
      const float zero_inf[2] = {0.0f, __int_as_float(0x7f800000)};
      const unsigned pick = static_cast<unsigned>(next(s) >> 20);
      tr = spread(s, -100, 62);
      tg = pick & 1u ? spread(s, -110, 70) : tg;
      mu = pick & 2u ? spread(s, -33, 100) : mu;
      cld.x = pick & 4u ? spread(s, -100, 62) : cld.x;
      cld.y = pick & 8u ? spread(s, -40, 0) : cld.y;
      cld.z = pick & 16u ? spread(s, -100, 0) : cld.z;
      if ((pick & 0x1e0u) == 0u) tr = zero_inf[pick >> 9 & 1u];
      if ((pick & 0x3c00u) == 0u) tg = zero_inf[pick >> 14 & 1u];
      if ((pick & 0x78000u) == 0u) mu = zero_inf[1];
      if ((pick & 0x780000u) == 0u) cld.x = zero_inf[pick >> 23 & 1u];
      if ((pick & 0xf000000u) == 0u) cld.z = zero_inf[0];
    }
    cld.w = cld.x * (1.0f + 10.0f * uniform(s));
    const float y_mu = recip_in_range(mu);
    SwClear c, c_any;
    const SwOptics clear = sw_clear<false>(T, tg, tr, mu, y_mu, c), clear_any = sw_clear_any<false>(T, tg, tr, mu, c_any);
    bad_clear += !same(clear, clear_any);
    bad_cloudy += !same(sw_cloudy<false>(T, c, clear, cld, mu, y_mu), sw_cloudy_any<false>(T, c_any, clear_any, cld, mu));
  }
  if (bad_clear) atomicAdd(&g_bad[0], static_cast<unsigned long long>(bad_clear));
  if (bad_cloudy) atomicAdd(&g_bad[1], static_cast<unsigned long long>(bad_cloudy));
}

}  // namespace
}  // namespace rrtmg

extern "C" int sw_layer_check(int ntbl, const float *exp_tbl, float bpade, int per_thread, int ends,
                              unsigned long long *bad) {
  using namespace rrtmg;
  std::vector<float2> pairs(ntbl + 1);
  for (int i = 0; i <= ntbl; ++i) pairs[i] = make_float2(exp_tbl[i], 1.0f / exp_tbl[i]);
  float *table = nullptr;
  float2 *pade = nullptr;
  const unsigned long long zero[2] = {0, 0};
  cudaError_t e = cudaMalloc(&table, sizeof(float) * (ntbl + 1));
  if (e == cudaSuccess) e = cudaMalloc(&pade, sizeof(float2) * (ntbl + 1));
  if (e == cudaSuccess) e = cudaMemcpy(table, exp_tbl, sizeof(float) * (ntbl + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(pade, pairs.data(), sizeof(float2) * (ntbl + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_bad, zero, sizeof(zero));
  if (e == cudaSuccess) {
    Tables T{};
    T.sw_pade_exp = table;
    T.sw_pade = pade;
    T.sw_bpade = bpade;
    T.sw_ntbl = ntbl;
    layers<<<148 * 4, 256>>>(T, per_thread, ends, 55);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(bad, g_bad, sizeof(zero));
  cudaFree(table);
  cudaFree(pade);
  return static_cast<int>(e);
}
