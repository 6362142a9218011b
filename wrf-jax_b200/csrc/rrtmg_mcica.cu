// McICA stochastic cloud masks on the GPU.
//
// Reference: generate_stochastic_clouds_overlap2 and the KISS stream
// (src/wrf_jax/physics/module_ra_rrtmg_common.py:964-1153).  The stream of one
// column is seeded from the fractional digits of its four lowest layer
// pressures and consumed in (subcolumn, layer) order after `skip` discarded
// draws (150 for LW, 1 for SW).  Here one thread owns one (column, subcolumn):
// it jumps the four KISS recurrences straight to draw skip + g*nlay with a
// host-computed jump (integer arithmetic, identical to sequential stepping),
// runs the maximum-random overlap chain up the column, and each warp ballots
// its 32 cloudy bits per layer into one mask word.  Layers above the column's
// highest cloud draw no random numbers (their bits are zero whatever is drawn),
// and a cloudless layer below it only steps the generators: its threshold for
// the layer above is 1, which no draw exceeds.
//
// Mask layout: mask[(l * words + w) * ncol + c], bit (g % 32) of word g / 32.
#include "rrtmg_device.cuh"
#include "rrtmg_kernels.h"

namespace rrtmg {

// Bound by integer issue.  425 x 425 x 50, clouds in the lowest 20 of 63 (LW)
// or 51 (SW) layers: LW 3.1 -> 1.0 ms, SW 2.2 -> 0.6 ms against drawing for
// every layer of every column from jump records of one subcolumn each (loads
// 152 bytes apart) with 64-bit remainders; a column cloudy to its top keeps the
// faster jump.
__global__ void __launch_bounds__(256) mcica_mask_kernel(McicaArgs a) {
  const int warps_per_col = a.words;
  const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int col = gwarp / warps_per_col;
  const int w = gwarp - col * warps_per_col;
  if (col >= a.ncol || dead_column(a.live, col)) return;  // whole warp exits together
  if (a.coszr && !(ld(a.coszr + col) > 0.0f)) return;       // a night column: nobody reads its mask
  const int i = col / a.ny, j = col - i * a.ny;
  const int nk = a.nk;

  // the column's cloud fractions, layer 32 q + lane in cld[q], and its highest cloud
  float cld[kMaxLay / 32];
  int top = -1;
#pragma unroll
  for (int q = 0; q < kMaxLay / 32; ++q) {
    const int l = 32 * q + lane;
    cld[q] = 0.0f;
    if (l < nk && a.enabled) cld[q] = ld(a.cldfra + (static_cast<size_t>(i) * nk + l) * a.ny + j);
    if (cld[q] < 1.0e-20f) cld[q] = 0.0f;
    const unsigned cloudy = __ballot_sync(0xffffffffu, cld[q] != 0.0f);
    if (cloudy) top = 32 * q + 31 - __clz(cloudy);
  }
  uint32_t *const mask = a.mask + static_cast<size_t>(w) * a.ncol + col;
  const size_t mstride = static_cast<size_t>(warps_per_col) * a.ncol;
  for (int l = top + 1 + lane; l < a.nlay; l += 32) mask[l * mstride] = 0u;
  if (top < 0) return;

  // seeds from pmid = play * 100 of the four lowest layers (common:1000-1004)
  Kiss s;
  {
    float pm[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float play = pa_to_hpa(ld(a.p3d + (static_cast<size_t>(i) * nk + k) * a.ny + j));
      pm[k] = play * 100.0f;
    }
    s.s1 = kiss_seed(pm[0]);
    s.s2 = kiss_seed(pm[1]);
    s.s3 = kiss_seed(pm[2]);
    s.s4 = kiss_seed(pm[3]);
  }
  const int g = w * 32 + lane;
  const bool active = g < a.nsub;
  s = kiss_jump(s, a.jumps, a.nsub, active ? g : 0);

  float cdf_prev = 0.0f, thr_prev = 1.0f;
#pragma unroll
  for (int q = 0; q < kMaxLay / 32; ++q) {
    if (32 * q > top) break;
    const int count = top - 32 * q < 31 ? top - 32 * q + 1 : 32;
    uint32_t mine = 0u;  // the word of layer 32 q + lane
    for (int e = 0; e < count; ++e) {
      const float c = __shfl_sync(0xffffffffu, cld[q], e);
      if (c == 0.0f) {
        s.step();
        cdf_prev = 0.0f;
        thr_prev = 1.0f;
        continue;
      }
      const float ran = s.next();
      const float cdf = (cdf_prev > thr_prev) ? cdf_prev : ran * thr_prev;
      thr_prev = 1.0f - c;
      cdf_prev = cdf;
      const unsigned word = __ballot_sync(0xffffffffu, active && cdf >= thr_prev);
      if (lane == e) mine = word;
    }
    if (lane < count) mask[static_cast<size_t>(32 * q + lane) * mstride] = mine;
  }
}

cudaError_t launch_mcica(const McicaArgs &a, cudaStream_t stream) {
  const int threads = 256;
  const long long total = static_cast<long long>(a.ncol) * a.words * 32;
  const int blocks = static_cast<int>((total + threads - 1) / threads);
  mcica_mask_kernel<<<blocks, threads, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace rrtmg
