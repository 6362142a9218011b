// RRTMG longwave, fused schedule: one thread per column, every step from the
// WRF adapter to the theta tendencies, no scratch but the McICA masks.  Used
// by rrtmg_lwrad_static_scratch only; every other call runs the sweep schedule
// of rrtmg_lw.cu, whose operations and order these are.
//
// Each thread sweeps its column layer by layer: the downward sweep visits
// layers top to bottom and, per layer, evaluates the band gas optics for all
// 140 g-points, advances their radiances and forms the level flux as the
// reference's ordered g-point/band sum; the upward sweep re-derives the layer
// optics bottom to top.  The 2 x 140 radiances, the downward level fluxes and
// the buffer-layer profile live in thread-local memory.
#include "rrtmg_lw_common.cuh"

namespace rrtmg {
namespace {

// One band of one layer in a sweep.  kDown: downward sweep (radiances radA =
// radld, radB = radclrd); otherwise upward (radA = radlu, radB = radclru).
// Returns the band's g-ordered radiance sums of the new level.
template <int B, bool kDown>
__device__ __forceinline__ void band_sums(const Tables &T, const Layer &L, const uint32_t *mask, bool cloudy_layer,
                                          int iceflag, float secdiff, float *radA, float *radB, bool sep_clear,
                                          float &bandsum, float &bandsumc) {
  constexpr int ngc = kNgc[B];
  constexpr int gofs = kGofs[B];
  const float blay = planck(T, L.indlay, L.tlayfrac, B);
  const float dplankup = planck(T, L.indlev1, L.tlev1frac, B) - blay;
  const float dplankdn = planck(T, L.indlev0, L.tlev0frac, B) - blay;
  float tauc = 0.0f, abscld = 0.0f;
  bool active = false;
  if (cloudy_layer) {
    tauc = cloud_tau(T, L, B, iceflag, active);
  }
  bandsum = 0.0f;
  bandsumc = 0.0f;
  auto gpoint = [&](int g, float tau, float fracs_g) {
    if (g >= ngc) return;
    const int G = gofs + g;
    const bool cld = (mask[G >> 5] >> (G & 31)) & 1u;
    float odepth = secdiff * tau;
    if (odepth < 0.0f) odepth = 0.0f;
    float odcld = 0.0f, efcl = 0.0f;
    if (cld) {
      const float t = active ? tauc : 0.0f;
      const float odcld_raw = secdiff * t;
      abscld = 1.0f - glibc_expf(T, -odcld_raw);
      odcld = odcld_raw;
      efcl = abscld * 1.0f;
    }
    const Terms tm = layer_terms(T, cloudy_layer, odepth, odcld, fracs_g, blay, dplankdn, dplankup);
    const float cf = cld ? 1.0f : 0.0f;
    float r = radA[G], rc = radB[G];
    if constexpr (kDown) {
      float rn;
      if (cloudy_layer) {
        rn = r - r * (tm.a + efcl * (1.0f - tm.a)) + tm.gassrc + cf * (tm.bbdtot * tm.atot - tm.gassrc);
      } else {
        rn = r + (tm.bbdgas - r) * tm.a;
      }
      const float rcn = sep_clear ? rc + (tm.bbdgas - rc) * tm.a : rn;
      radA[G] = rn;
      radB[G] = rcn;
      bandsum = bandsum + rn;
      bandsumc = bandsumc + rcn;
    } else {
      float rn;
      if (cloudy_layer) {
        const float gas = tm.bbugas * tm.a;
        rn = r - r * (tm.a + efcl * (1.0f - tm.a)) + gas + cf * (tm.bbutot * tm.atot - gas);
      } else {
        rn = r + (tm.bbugas - r) * tm.a;
      }
      const float rcn = sep_clear ? rc + (tm.bbugas - rc) * tm.a : rn;
      radA[G] = rn;
      radB[G] = rcn;
      bandsum = bandsum + rn;
      bandsumc = bandsumc + rcn;
    }
  };
  gas_quads<B>(T, L, [&](int q, float4 tau, float4 frac) {
    gpoint(4 * q, tau.x, frac.x);
    gpoint(4 * q + 1, tau.y, frac.y);
    gpoint(4 * q + 2, tau.z, frac.z);
    gpoint(4 * q + 3, tau.w, frac.w);
  });
}

template <int B, bool kDown>
__device__ __forceinline__ void band_step(const Tables &T, const Layer &L, const uint32_t *mask, bool cloudy_layer,
                                          int iceflag, float secdiff, float *radA, float *radB, bool sep_clear,
                                          float &total, float &totalc) {
  float bandsum, bandsumc;
  band_sums<B, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff, radA, radB, sep_clear, bandsum, bandsumc);
  total = total + (bandsum * 0.5f) * kDelwave[B];
  totalc = totalc + (bandsumc * 0.5f) * kDelwave[B];
}

template <bool kDown>
__device__ __forceinline__ void all_bands(const Tables &T, const Layer &L, const uint32_t *mask, bool cloudy_layer,
                                          int iceflag, const float *secdiff, float *radA, float *radB, bool sep,
                                          float &total, float &totalc) {
  band_step<0, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[0], radA, radB, sep, total, totalc);
  band_step<1, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[1], radA, radB, sep, total, totalc);
  band_step<2, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[2], radA, radB, sep, total, totalc);
  band_step<3, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[3], radA, radB, sep, total, totalc);
  band_step<4, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[4], radA, radB, sep, total, totalc);
  band_step<5, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[5], radA, radB, sep, total, totalc);
  band_step<6, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[6], radA, radB, sep, total, totalc);
  band_step<7, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[7], radA, radB, sep, total, totalc);
  band_step<8, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[8], radA, radB, sep, total, totalc);
  band_step<9, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[9], radA, radB, sep, total, totalc);
  band_step<10, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[10], radA, radB, sep, total, totalc);
  band_step<11, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[11], radA, radB, sep, total, totalc);
  band_step<12, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[12], radA, radB, sep, total, totalc);
  band_step<13, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[13], radA, radB, sep, total, totalc);
  band_step<14, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[14], radA, radB, sep, total, totalc);
  band_step<15, kDown>(T, L, mask, cloudy_layer, iceflag, secdiff[15], radA, radB, sep, total, totalc);
}

// Surface: rad0 = fracs(layer 0) * plankbnd, reflected downward radiance
// (lw:5648-5655); returns the level-0 upward flux sums.
template <int B>
__device__ __forceinline__ void surface_sums(const Tables &T, const Layer &L0, float plankbnd, float reflect,
                                             float *radA, float *radB, float &bandsum, float &bandsumc) {
  constexpr int ngc = kNgc[B];
  constexpr int gofs = kGofs[B];
  bandsum = 0.0f;
  bandsumc = 0.0f;
  auto gpoint = [&](int g, float fracs_g) {
    if (g >= ngc) return;
    const int G = gofs + g;
    const float rad0 = fracs_g * plankbnd;
    const float lu = rad0 + reflect * radA[G];
    const float lc = rad0 + reflect * radB[G];
    radA[G] = lu;
    radB[G] = lc;
    bandsum = bandsum + lu;
    bandsumc = bandsumc + lc;
  };
  gas_quads<B>(T, L0, [&](int q, float4, float4 frac) {
    gpoint(4 * q, frac.x);
    gpoint(4 * q + 1, frac.y);
    gpoint(4 * q + 2, frac.z);
    gpoint(4 * q + 3, frac.w);
  });
}

template <int B>
__device__ __forceinline__ void surface_band(const Tables &T, const Layer &L0, float plankbnd, float reflect,
                                             float *radA, float *radB, float &total, float &totalc) {
  float bandsum, bandsumc;
  surface_sums<B>(T, L0, plankbnd, reflect, radA, radB, bandsum, bandsumc);
  total = total + (bandsum * 0.5f) * kDelwave[B];
  totalc = totalc + (bandsumc * 0.5f) * kDelwave[B];
}

__device__ __forceinline__ void column_core(const Tables &T, const LwArgs &a, int col, Col &C) {
  column_head(a, col, C);
  column_setup(T, a, C);
  const int nlay = C.nlay;
  // column integrals: laytrop and pwvcm, summed in layer order
  int laytrop = 0;
  float amttl = 0.0f, wvttl = 0.0f;
  for (int l = 0; l < nlay; ++l) {
    bool trop;
    float coldry, wk0;
    column_layer(T, a, C, l, trop, coldry, wk0);
    laytrop += trop;
    amttl = (amttl + coldry) + wk0;
    wvttl = wvttl + wk0;
  }
  C.laytrop = laytrop;
  C.pwvcm = column_pwvcm(a, C, amttl, wvttl);
}

__device__ __forceinline__ void column_prologue(const Tables &T, const LwArgs &a, int col, Col &C, float *secdiff,
                                                bool &has_cloud) {
  column_core(T, a, col, C);
  const int nlay = C.nlay;
  column_secdiff(T, C, secdiff);

  // cloudy layers and whether any layer is cloudy (lw:5566-5567, 5656)
  has_cloud = false;
  for (int l = 0; l < nlay; ++l) {
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < kLwMaskWords; ++w) any |= a.mask[(static_cast<size_t>(l) * kLwMaskWords + w) * a.ncol + col];
    has_cloud |= any != 0u;
  }
}

__global__ void __launch_bounds__(128) lw_kernel(Tables T, LwArgs a) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= a.ncol) return;
  Col C;
  float secdiff[kLwBands];
  bool has_cloud;
  column_prologue(T, a, col, C, secdiff, has_cloud);
  const int nlay = C.nlay;

  float radA[kLwGpts], radB[kLwGpts];
  float dfl[kMaxLay + 1], dflc[kMaxLay + 1];
#pragma unroll 4
  for (int g = 0; g < kLwGpts; ++g) { radA[g] = 0.0f; radB[g] = 0.0f; }
  const float pi = 3.1415926535897932384626433832795f;
  const float fluxfac = pi * 2.0e4f;
  const float heatfac = (9.8066f * 8.6400e4f) / (1004.5f * 1.0e2f);
  dfl[nlay] = 0.0f * fluxfac;
  dflc[nlay] = 0.0f * fluxfac;

  // downward sweep, top to bottom
  bool iclddn = false;
  for (int l = nlay - 1; l >= 0; --l) {
    uint32_t mask[kLwMaskWords];
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < kLwMaskWords; ++w) {
      mask[w] = a.mask[(static_cast<size_t>(l) * kLwMaskWords + w) * a.ncol + col];
      any |= mask[w];
    }
    const bool cloudy = any != 0u;
    iclddn = iclddn || cloudy;
    const Layer L = make_layer(T, a, C, l);
    float total = 0.0f, totalc = 0.0f;
    all_bands<true>(T, L, mask, cloudy, C.iceflg, secdiff, radA, radB, iclddn, total, totalc);
    dfl[l] = total * fluxfac;
    dflc[l] = totalc * fluxfac;
  }
  // surface emission and reflection
  float ufl_prev, uflc_prev;
  {
    const Layer L0 = make_layer(T, a, C, 0);
    const float bt = C.tsfc - 159.0f;
    const int indbound = clampi(static_cast<int>(bt), 1, 180);
    const float tbndfrac = bt - static_cast<float>(indbound);
    const float reflect = 1.0f - C.semiss;
    float total = 0.0f, totalc = 0.0f;
#define SURF(B) surface_band<B>(T, L0, C.semiss * planck(T, indbound, tbndfrac, B), reflect, radA, radB, total, totalc)
    SURF(0); SURF(1); SURF(2); SURF(3); SURF(4); SURF(5); SURF(6); SURF(7);
    SURF(8); SURF(9); SURF(10); SURF(11); SURF(12); SURF(13); SURF(14); SURF(15);
#undef SURF
    ufl_prev = total * fluxfac;
    uflc_prev = totalc * fluxfac;
  }
  const float upb = ufl_prev, upbc = uflc_prev;
  // upward sweep, bottom to top, with the heating rate of each layer
  const size_t rbase = static_cast<size_t>(C.i) * C.nk * C.ny + C.j;
  for (int l = 0; l < nlay; ++l) {
    uint32_t mask[kLwMaskWords];
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < kLwMaskWords; ++w) {
      mask[w] = a.mask[(static_cast<size_t>(l) * kLwMaskWords + w) * a.ncol + col];
      any |= mask[w];
    }
    const bool cloudy = any != 0u;
    const Layer L = make_layer(T, a, C, l);
    float total = 0.0f, totalc = 0.0f;
    all_bands<false>(T, L, mask, cloudy, C.iceflg, secdiff, radA, radB, has_cloud, total, totalc);
    const float ufl = total * fluxfac, uflc = totalc * fluxfac;
    if (l < C.nk) {
      const float fnet0 = ufl_prev - dfl[l], fnet1 = ufl - dfl[l + 1];
      const float fnetc0 = uflc_prev - dflc[l], fnetc1 = uflc - dflc[l + 1];
      const float dp = L.plev0 - L.plev1;
      float htr = heatfac * (fnet0 - fnet1) / dp;
      float htrc = heatfac * (fnetc0 - fnetc1) / dp;
      if (l >= a.fp64_from) {
        htr = heating64(heatfac, ufl_prev, dfl[l], ufl, dfl[l + 1], L.plev0, L.plev1);
        htrc = heating64(heatfac, uflc_prev, dflc[l], uflc, dflc[l + 1], L.plev0, L.plev1);
      }
      const float pi3d = ld(a.in.pi3d + rbase + static_cast<size_t>(l) * C.ny);
      a.rthraten[rbase + static_cast<size_t>(l) * C.ny] = (htr / 86400.0f) / pi3d;
      a.rthratenc[rbase + static_cast<size_t>(l) * C.ny] = (htrc / 86400.0f) / pi3d;
    }
    ufl_prev = ufl;
    uflc_prev = uflc;
  }
  // 2-D outputs (lw:7059-7077)
  a.upt[col] = ufl_prev;
  a.uptc[col] = uflc_prev;
  a.dnt[col] = dfl[nlay];
  a.dntc[col] = dflc[nlay];
  a.upb[col] = upb;
  a.upbc[col] = upbc;
  a.dnb[col] = dfl[0];
  a.dnbc[col] = dflc[0];
  a.glw[col] = dfl[0];
  a.olr[col] = ufl_prev;
  a.lwcf[col] = uflc_prev - ufl_prev;
#pragma unroll
  for (int q = 0; q < 4; ++q) a.zero2[q][col] = 0.0f;
}

}  // namespace

cudaError_t launch_lw(const Tables &T, const LwArgs &a, cudaStream_t stream) {
  const int threads = 128;
  const int blocks = (a.ncol + threads - 1) / threads;
  lw_kernel<<<blocks, threads, 0, stream>>>(T, a);
  return cudaGetLastError();
}

}  // namespace rrtmg
