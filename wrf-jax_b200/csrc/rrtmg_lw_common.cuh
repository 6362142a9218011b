// Longwave pieces shared by the sweep schedule (rrtmg_lw.cu) and the fused
// one-thread-per-column schedule (rrtmg_lw_fused.cu): the column context and
// set-up, the layer set-up, cloud optics, Planck terms and layer transfer.
#pragma once

#include "rrtmg_device.cuh"
#include "rrtmg_kernels.h"
#include "rrtmg_lw_gas.cuh"

namespace rrtmg {
namespace {

// lwdatinit delwave (module_ra_rrtmg_common.py:736-738)
__constant__ float kDelwave[kLwBands] = {340.0f, 150.0f, 130.0f, 70.0f, 120.0f, 160.0f, 100.0f, 100.0f,
                                      210.0f, 90.0f, 320.0f, 280.0f, 170.0f, 130.0f, 220.0f, 650.0f};
// diffusivity fit (lw:5520-5531)
__constant__ float kA0[kLwBands] = {1.66f, 1.55f, 1.58f, 1.66f, 1.54f, 1.454f, 1.89f, 1.33f,
                                 1.668f, 1.66f, 1.66f, 1.66f, 1.66f, 1.66f, 1.66f, 1.66f};
__constant__ float kA1[kLwBands] = {0.0f, 0.25f, 0.22f, 0.0f, 0.13f, 0.446f, -0.10f, 0.40f,
                                 -0.006f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
__constant__ float kA2[kLwBands] = {0.0f, -12.0f, -11.7f, 0.0f, -0.72f, -0.243f, 0.19f, -0.062f,
                                 0.414f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};

// ---------------------------------------------------------------------------
// per-column context
// ---------------------------------------------------------------------------
struct Col {
  int i, j, nk, nlay, ny, nbuf;
  int laytrop;
  float tsfc, semiss, pwvcm;
  float co2, n2o, ch4, cfc11, cfc12;
  int inflg, iceflg, has_reqc, has_reqi, has_reqs, icloud;
  float plev_b[kMaxBuf + 1];   // levels nk .. nlay
  float play_b[kMaxBuf];       // layers nk .. nlay-1
  float tlev_b[kMaxBuf + 1];   // levels nk .. nlay
  float tlay_b[kMaxBuf + 1];   // layers nk-1 .. nlay-1
  float o3_b[kMaxBuf];         // layers nk .. nlay-1
};

__device__ __forceinline__ float in3(const float *p, const Col &C, int k) {
  return ld(p + (static_cast<size_t>(C.i) * C.nk + k) * C.ny + C.j);
}
__device__ __forceinline__ float in3w(const float *p, const Col &C, int k) {
  return ld(p + (static_cast<size_t>(C.i) * (C.nk + 1) + k) * C.ny + C.j);
}

__device__ __forceinline__ float plev_at(const LwArgs &a, const Col &C, int l) {
  return l < C.nk ? pa_to_hpa(in3w(a.in.p8w, C, l)) : C.plev_b[l - C.nk];
}
__device__ __forceinline__ float play_at(const LwArgs &a, const Col &C, int l) {
  return l < C.nk ? pa_to_hpa(in3(a.in.p3d, C, l)) : C.play_b[l - C.nk];
}
__device__ __forceinline__ float tlev_at(const LwArgs &a, const Col &C, int l) {
  return l < C.nk ? in3w(a.in.t8w, C, l) : C.tlev_b[l - C.nk];
}
__device__ __forceinline__ float tlay_at(const LwArgs &a, const Col &C, int l) {
  return l < C.nk - 1 ? in3(a.in.t3d, C, l) : C.tlay_b[l - (C.nk - 1)];
}
__device__ __forceinline__ float h2o_at(const LwArgs &a, const Col &C, int l) {
  const int k = l < C.nk ? l : C.nk - 1;
  return fmaxf(in3(a.in.qv, C, k), 1.0e-12f) * 1.607793f;
}
__device__ __forceinline__ float o3_at(const LwArgs &a, const Col &C, int l) {
  return l < C.nk ? in3(a.in.o3, C, l) : C.o3_b[l - C.nk];
}

// o3data (common:357-404) for one layer bounded by pressures pa > pb
__device__ float o3data_layer(const Tables &T, float pa, float pb) {
  float total = 0.0f;
#pragma unroll 4
  for (int b = 0; b < 31; ++b) {
    const float pb1 = fmaxf(pa - T.ppwrkh[b], 0.0f);
    const float pb2 = fmaxf(pa - T.ppwrkh[b + 1], 0.0f);
    const float pt1 = fmaxf(pb - T.ppwrkh[b], 0.0f);
    const float pt2 = fmaxf(pb - T.ppwrkh[b + 1], 0.0f);
    const float overlap = ((pb2 - pb1) - pt2) + pt1;
    total = total + overlap * T.o3wrk[b];
  }
  return total / (pa - pb);
}

__device__ float retab_interp(const Tables &T, float temp, int hi) {
  const int tint = static_cast<int>(temp);
  const int index = clampi(static_cast<int>(temp - 179.0f), 1, hi);
  const float corr = temp - static_cast<float>(tint);
  return ld(T.retab + index - 1) * (1.0f - corr) + ld(T.retab + index) * corr;
}

// Interface temperature of the standard profile at pressure p, between the last
// entry not below p (count entries are) and the next.
__device__ __forceinline__ float profile_between(const Tables &T, int count, float p) {
  const int idx = clampi(count - 1, 0, T.nprof - 1);
  const int idx1 = idx + 1 < T.nprof - 1 ? idx + 1 : T.nprof - 1;
  const float p0 = ld(T.pprof + idx), p1 = ld(T.pprof + idx1);
  const float t0 = ld(T.tprof + idx), t1 = ld(T.tprof + idx1);
  const float w = (idx == T.nprof - 1) ? 0.0f : (p - p0) / (p1 - p0);
  return w * (t1 - t0) + t0;
}

// Pressures of the levels above the model top.
__device__ __forceinline__ void column_levels(const LwArgs &a, Col &C) {
  C.plev_b[0] = pa_to_hpa(in3w(a.in.p8w, C, C.nk));
  for (int m = 1; m <= C.nbuf; ++m) C.plev_b[m] = C.plev_b[m - 1] - 4.0f;
  C.plev_b[C.nbuf] = 0.0f;
}

// Column set-up: buffer layers above the model top (lw:6633-6786).
__device__ void column_setup(const Tables &T, const LwArgs &a, Col &C) {
  const int nk = C.nk, nbuf = C.nbuf;
  column_levels(a, C);
  for (int m = 0; m < nbuf; ++m) C.play_b[m] = 0.5f * (C.plev_b[m] + C.plev_b[m + 1]);
  // interface temperatures from the standard profile plus the model-top offset
  auto varint = [&](float p) {
    int count = 0;
    for (int q = 0; q < T.nprof; ++q) count += (ld(T.pprof + q) >= p);
    return profile_between(T, count, p);
  };
  const float offset = in3w(a.in.t8w, C, nk - 1) - varint(pa_to_hpa(in3w(a.in.p8w, C, nk - 1)));
  for (int m = 0; m <= nbuf; ++m) C.tlev_b[m] = varint(C.plev_b[m]) + offset;
  // ozone above the model top (lw:6766-6786)
  const float amdo = 0.603461f;
  const float o3base = in3(a.in.o3, C, nk - 1) -
                       o3data_layer(T, pa_to_hpa(in3w(a.in.p8w, C, nk - 1)), C.plev_b[0]) * amdo;
  for (int m = 0; m < nbuf; ++m) {
    const float mmr = o3data_layer(T, C.plev_b[m], C.plev_b[m + 1]) * amdo;
    float top = o3base + mmr;
    if (top <= 0.0f) top = mmr;
    C.o3_b[m] = top;
  }
  // tlay[lev-1] = (tlev[lev] + tlev[lev-1]) / 2 for lev = nk .. nlay
  C.tlay_b[0] = 0.5f * (C.tlev_b[0] + in3w(a.in.t8w, C, nk - 1));
  for (int m = 1; m <= nbuf; ++m) C.tlay_b[m] = 0.5f * (C.tlev_b[m] + C.tlev_b[m - 1]);
}

// The same by the 32 lanes of a warp for one column, C in shared memory: a
// lane takes every 32nd level or layer, with the model-top values (the offset's
// profile temperature, the ozone base) as one more; s_tlev holds kMaxBuf + 2
// values, s_o3 kMaxBuf + 1.
__device__ void column_setup_warp(const Tables &T, const LwArgs &a, Col &C, int lane, float *s_tlev, float *s_o3) {
  const int nk = C.nk, nbuf = C.nbuf;
  column_levels(a, C);  // every lane, the same values
  __syncwarp();
  for (int m = lane; m < nbuf; m += 32) C.play_b[m] = 0.5f * (C.plev_b[m] + C.plev_b[m + 1]);
  const float top_p = pa_to_hpa(in3w(a.in.p8w, C, nk - 1)), top_t = in3w(a.in.t8w, C, nk - 1);
  for (int m0 = 0; m0 < nbuf + 2; m0 += 32) {
    const int m = m0 + lane;
    const float p = m <= nbuf ? C.plev_b[m] : top_p;
    int count = 0;
    for (int q0 = 0; q0 < T.nprof; q0 += 32) {
      const float v = q0 + lane < T.nprof ? ld(T.pprof + q0 + lane) : 0.0f;
      const int end = T.nprof - q0 < 32 ? T.nprof - q0 : 32;
      for (int q = 0; q < end; ++q) count += __shfl_sync(0xffffffffu, v, q) >= p;
    }
    if (m < nbuf + 2) s_tlev[m] = profile_between(T, count, p);
  }
  const float amdo = 0.603461f;
  for (int m = lane; m <= nbuf; m += 32)
    s_o3[m] = (m < nbuf ? o3data_layer(T, C.plev_b[m], C.plev_b[m + 1]) : o3data_layer(T, top_p, C.plev_b[0])) * amdo;
  __syncwarp();
  const float offset = top_t - s_tlev[nbuf + 1];
  const float o3base = in3(a.in.o3, C, nk - 1) - s_o3[nbuf];
  for (int m = lane; m <= nbuf; m += 32) C.tlev_b[m] = s_tlev[m] + offset;
  for (int m = lane; m < nbuf; m += 32) {
    const float mmr = s_o3[m];
    float top = o3base + mmr;
    if (top <= 0.0f) top = mmr;
    C.o3_b[m] = top;
  }
  __syncwarp();
  for (int m = lane; m <= nbuf; m += 32) C.tlay_b[m] = 0.5f * (C.tlev_b[m] + (m == 0 ? top_t : C.tlev_b[m - 1]));
  __syncwarp();
}

// Layer coefficients: inatm (lw:953-1035), cloud paths, setcoef (lw:1175-1441).
__device__ __forceinline__ Layer make_layer(const Tables &T, const LwArgs &a, const Col &C, int l) {
  Layer L;
  L.pavel = play_at(a, C, l);
  L.tavel = tlay_at(a, C, l);
  L.plev0 = plev_at(a, C, l);
  L.plev1 = plev_at(a, C, l + 1);
  const float h2o = h2o_at(a, C, l);
  const float o3 = o3_at(a, C, l);
  const float amd = 28.9660f, amw = 18.0160f, avogad = 6.02214199e23f, grav = 9.8066f;
  const float amm = (1.0f - h2o) * amd + h2o * amw;
  const float pm = ((L.plev0 - L.plev1) * 1.0e3f) * avogad;
  float md = 1.0e2f * grav;
  md = md * amm;
  md = md * (1.0f + h2o);
  const float coldry = pm / md;
  L.coldry = coldry;
  const float o2 = 0.209488f;
  float summol = 0.0f;
  summol = summol + C.co2;
  summol = summol + o3;
  summol = summol + C.n2o;
  summol = summol + 0.0f;
  summol = summol + C.ch4;
  summol = summol + o2;
  const float wbrodl = coldry * (1.0f - summol);
  const float wk0 = h2o * coldry, wk1 = C.co2 * coldry, wk2 = o3 * coldry, wk3 = C.n2o * coldry;
  const float wk4 = 0.0f * coldry, wk5 = C.ch4 * coldry, wk6 = o2 * coldry;
  L.wx0 = (0.093e-9f * coldry) * 1.0e-20f;
  L.wx1 = (C.cfc11 * coldry) * 1.0e-20f;
  L.wx2 = (C.cfc12 * coldry) * 1.0e-20f;
  L.wx3 = (0.169e-9f * coldry) * 1.0e-20f;

  // Planck indices
  {
    const float tl = L.tavel - 159.0f;
    L.indlay = clampi(static_cast<int>(tl), 1, 180);
    L.tlayfrac = tl - static_cast<float>(L.indlay);
    const float t0 = tlev_at(a, C, l) - 159.0f;
    L.indlev0 = clampi(static_cast<int>(t0), 1, 180);
    L.tlev0frac = t0 - static_cast<float>(L.indlev0);
    const float t1 = tlev_at(a, C, l + 1) - 159.0f;
    L.indlev1 = clampi(static_cast<int>(t1), 1, 180);
    L.tlev1frac = t1 - static_cast<float>(L.indlev1);
  }
  const float stpfac = 296.0f / 1013.0f;
  const float plog = glibc_logf(T, L.pavel);
  const int jp = clampi(static_cast<int>(36.0f - 5.0f * (plog + 0.04f)), 1, 58);
  const float fp = 5.0f * (ld(T.lw_preflog + jp - 1) - plog);
  const float tf = (L.tavel - ld(T.lw_tref + jp - 1)) / 15.0f;
  const int jt = clampi(static_cast<int>(3.0f + tf), 1, 4);
  const float ft = tf - static_cast<float>(jt - 3);
  const float tf1 = (L.tavel - ld(T.lw_tref + jp)) / 15.0f;
  const int jt1 = clampi(static_cast<int>(3.0f + tf1), 1, 4);
  const float ft1 = tf1 - static_cast<float>(jt1 - 3);
  const float water = wk0 / coldry;
  const float scalefac = (L.pavel * stpfac) / L.tavel;
  const int trop = plog > 4.56f;
  L.trop = l < C.laytrop;
  const float forfac_base = scalefac / (1.0f + water);
  const float ftf = (332.0f - L.tavel) / 36.0f;
  const int indfor_t = clampi(static_cast<int>(ftf), 1, 2);
  const float forfrac_t = ftf - static_cast<float>(indfor_t);
  const float fsf = (L.tavel - 188.0f) / 36.0f;
  L.indfor = trop ? indfor_t : 3;
  L.forfrac = trop ? forfrac_t : fsf - 1.0f;
  const float fself = (L.tavel - 188.0f) / 7.2f;
  const int indself_t = clampi(static_cast<int>(fself) - 7, 1, 9);
  const float selffrac_t = fself - static_cast<float>(indself_t + 7);
  L.indself = trop ? indself_t : 0;
  L.selffrac = trop ? selffrac_t : 0.0f;
  L.scaleminor = L.pavel / L.tavel;
  L.scaleminorn2 = L.scaleminor * (wbrodl / (coldry + wk0));
  const float fminor = (L.tavel - 180.8f) / 7.2f;
  L.indminor = clampi(static_cast<int>(fminor), 1, 18);
  L.minorfrac = fminor - static_cast<float>(L.indminor);
  const float tiny = 1.0e-20f;
  const float fallback = 1.0e-32f * coldry;
  L.colh2o = tiny * wk0;
  L.colco2 = tiny * wk1;
  L.colo3 = tiny * wk2;
  L.coln2o = tiny * wk3;
  L.colco = tiny * wk4;
  L.colch4 = tiny * wk5;
  L.colo2 = tiny * wk6;
  if (L.colco2 == 0.0f) L.colco2 = fallback;
  if (L.colo3 == 0.0f) L.colo3 = fallback;
  if (L.coln2o == 0.0f) L.coln2o = fallback;
  if (L.colco == 0.0f) L.colco = fallback;
  if (L.colch4 == 0.0f) L.colch4 = fallback;
  L.colbrd = tiny * wbrodl;
  const float *chi = T.chi_mls;
  const int j0 = jp - 1, j1 = jp;
  auto CHI = [&](int gas, int lev) { return ld(chi + gas * 59 + lev); };
  L.rat_h2oco2 = CHI(0, j0) / CHI(1, j0);
  L.rat_h2oco2_1 = CHI(0, j1) / CHI(1, j1);
  L.rat_h2oo3 = trop ? CHI(0, j0) / CHI(2, j0) : 0.0f;
  L.rat_h2oo3_1 = trop ? CHI(0, j1) / CHI(2, j1) : 0.0f;
  L.rat_h2on2o = trop ? CHI(0, j0) / CHI(3, j0) : 0.0f;
  L.rat_h2on2o_1 = trop ? CHI(0, j1) / CHI(3, j1) : 0.0f;
  L.rat_h2och4 = trop ? CHI(0, j0) / CHI(5, j0) : 0.0f;
  L.rat_h2och4_1 = trop ? CHI(0, j1) / CHI(5, j1) : 0.0f;
  L.rat_n2oco2 = trop ? CHI(3, j0) / CHI(1, j0) : 0.0f;
  L.rat_n2oco2_1 = trop ? CHI(3, j1) / CHI(1, j1) : 0.0f;
  L.rat_o3co2 = trop ? 0.0f : CHI(2, j0) / CHI(1, j0);
  L.rat_o3co2_1 = trop ? 0.0f : CHI(2, j1) / CHI(1, j1);
  const float compfp = 1.0f - fp;
  L.fac10 = compfp * ft;
  L.fac00 = compfp * (1.0f - ft);
  L.fac11 = fp * ft1;
  L.fac01 = fp * (1.0f - ft1);
  L.selffac = L.colh2o * (water * forfac_base);
  L.forfac = L.colh2o * forfac_base;
  L.jp = jp;
  L.jt = jt;
  L.jt1 = jt1;

  // cloud radii and in-cloud paths (common:801-961); zero above the model top
  L.cldfrac = 0.0f; L.clwp = 0.0f; L.ciwp = 0.0f; L.cswp = 0.0f;
  L.rel = 10.0f; L.rei = 10.0f; L.res = 10.0f;
  if (l < C.nk) {
    const float t = in3(a.in.t3d, C, l);
    const float cldfra = in3(a.in.cldfra, C, l);
    float qc = fmaxf(in3(a.in.qc, C, l), 0.0f), qi = fmaxf(in3(a.in.qi, C, l), 0.0f);
    float qs = fmaxf(in3(a.in.qs, C, l), 0.0f);
    const float xland = ld(a.in.xland + C.i * C.ny + C.j);
    float recloud = 5.0f, reice = 10.0f, resnow = 10.0f;
    if (C.icloud != 0) {
      if (C.has_reqc) {
        recloud = fmaxf(2.5f, in3(a.in.re_cloud, C, l) * 1.0e6f);
        const int cloudy_min = (recloud <= 2.5f) && (cldfra > 0.0f);
        if (cloudy_min && (xland - 1.5f > 0.0f)) recloud = 10.5f;
        if (cloudy_min && (xland - 1.5f < 0.0f)) recloud = 7.5f;
      }
      if (C.has_reqi) {
        reice = fmaxf(5.0f, in3(a.in.re_ice, C, l) * 1.0e6f);
        if ((reice <= 5.0f) && (cldfra > 0.0f)) reice = fmaxf(retab_interp(T, t, 75), 5.0f);
      }
      if (C.has_reqs) resnow = fmaxf(10.0f, in3(a.in.re_snow, C, l) * 1.0e6f);
      if (!C.has_reqs && C.has_reqi && C.has_reqc) {
        resnow = fmaxf(10.0f, in3(a.in.re_ice, C, l) * 1.0e6f);
        qs = qi;
        qi = 0.0f;
        reice = 10.0f;
      }
    }
    const float temp = L.tavel;
    const float dp = L.plev0 - L.plev1;
    const float denom = fmaxf(0.01f, cldfra);
    float gicewp = (qi + qs) * dp * 100.0f / grav * 1000.0f;
    const float gliqwp = qc * dp * 100.0f / grav * 1000.0f;
    float cicewp = gicewp / denom;
    const float cliqwp = gliqwp / denom;
    if (C.iceflg >= 4) {
      gicewp = qi * dp * 100.0f / grav * 1000.0f;
      cicewp = gicewp / denom;
    }
    float csnowp = 0.0f, res_adj = resnow;
    if (C.iceflg == 5) {
      float smf = 0.99f;
      if (res_adj > 130.0f) {
        const float lim = (130.0f / res_adj) * (130.0f / res_adj);
        smf = fminf(0.99f, lim);
        res_adj = 130.0f;
      }
      const float gsnowp = qs * smf * dp * 100.0f / grav * 1000.0f;
      csnowp = gsnowp / denom;
    }
    const float xice = ld(a.in.xice + C.i * C.ny + C.j), snow = ld(a.in.snow + C.i * C.ny + C.j);
    const float landm = 2.0f - xland, snowh = 0.001f * snow;
    const float rocean = 14.0f, rland = 8.0f, rice = 14.0f;
    float rel = rland + (rocean - rland) * fminf(1.0f, fmaxf(0.0f, (273.16f - temp) * 0.05f));
    rel = rel + (rocean - rel) * fminf(1.0f, fmaxf(0.0f, snowh * 10.0f));
    rel = rel + (rocean - rel) * fminf(1.0f, fmaxf(0.0f, 1.0f - landm));
    rel = rel + (rice - rel) * fminf(1.0f, fmaxf(0.0f, xice));
    float rei = retab_interp(T, temp, 94);
    if (C.inflg >= 3) rel = recloud;
    if (C.iceflg >= 4) rei = reice;
    if (C.iceflg == 3) rei = fminf(140.0f, rei * 1.0315f);
    L.cldfrac = cldfra;
    L.clwp = cliqwp;
    L.ciwp = cicewp;
    L.cswp = (C.inflg == 5) ? csnowp : 0.0f;
    L.rel = rel;
    L.rei = rei;
    L.res = (C.inflg == 5) ? res_adj : 10.0f;
  }
  return L;
}

// ---------------------------------------------------------------------------
// Cloud optical depth of band B for a cloudy g-point of a layer
// (cldprmc, lw:5725-5830; ice options >= 3, liquid option 1)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float cloud_tau(const Tables &T, const Layer &L, int band, int iceflag, bool &active) {
  const float ciwp = L.ciwp, clwp = L.clwp, cswp = L.cswp;
  const float cwp = (ciwp + clwp) + cswp;
  active = cwp >= 1.0e-20f;
  const float factor = (L.rei - 2.0f) / 3.0f;
  int index = static_cast<int>(factor);
  if (index == 46) index = 45;
  const float fint = factor - static_cast<float>(index);
  float abscoice = interpf(ld(T.absice3 + jrow(index - 1, 46) * 16 + band), ld(T.absice3 + jrow(index, 46) * 16 + band), fint);
  float abscosno = 0.0f;
  if ((ciwp + cswp) == 0.0f) abscoice = 0.0f;
  if (iceflag == 5 && cswp > 0.0f) {
    const float fs = (L.res - 2.0f) / 3.0f;
    int is = static_cast<int>(fs);
    if (is == 46) is = 45;
    const float fints = fs - static_cast<float>(is);
    abscosno = interpf(ld(T.absice3 + jrow(is - 1, 46) * 16 + band), ld(T.absice3 + jrow(is, 46) * 16 + band), fints);
  }
  int il = static_cast<int>(L.rel - 1.5f);
  if (il == 0) il = 1;
  if (il == 58) il = 57;
  const float fl = (L.rel - 1.5f) - static_cast<float>(il);
  const float abscoliq = clwp == 0.0f ? 0.0f
      : interpf(ld(T.absliq1 + jrow(il - 1, 58) * 16 + band), ld(T.absliq1 + jrow(il, 58) * 16 + band), fl);
  return (ciwp * abscoice + clwp * abscoliq) + cswp * abscosno;
}

// cloud_tau and planck of bands 4 b4 .. 4 b4 + 3 (table rows of 16 bands).
__device__ __forceinline__ float4 cloud_tau4(const Tables &T, const Layer &L, int b4, int iceflag, bool &active) {
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float ciwp = L.ciwp, clwp = L.clwp, cswp = L.cswp;
  const float cwp = (ciwp + clwp) + cswp;
  active = cwp >= 1.0e-20f;
  // rows `index - 1` and `index` of a size with spacing 3, as cldprmc does
  auto ice = [&](float size) {
    const float factor = (size - 2.0f) / 3.0f;
    int index = static_cast<int>(factor);
    if (index == 46) index = 45;
    return interp4(row4<16>(T.absice3, jrow(index - 1, 46), b4), row4<16>(T.absice3, jrow(index, 46), b4),
                   factor - static_cast<float>(index));
  };
  const float4 abscoice = (ciwp + cswp) == 0.0f ? zero : ice(L.rei);
  const float4 abscosno = iceflag == 5 && cswp > 0.0f ? ice(L.res) : zero;
  float4 abscoliq = zero;
  if (clwp != 0.0f) {
    int il = static_cast<int>(L.rel - 1.5f);
    if (il == 0) il = 1;
    if (il == 58) il = 57;
    const float fl = (L.rel - 1.5f) - static_cast<float>(il);
    abscoliq = interp4(row4<16>(T.absliq1, jrow(il - 1, 58), b4), row4<16>(T.absliq1, jrow(il, 58), b4), fl);
  }
  return add4(add4(mul4(ciwp, abscoice), mul4(clwp, abscoliq)), mul4(cswp, abscosno));
}

__device__ __forceinline__ float4 planck4(const Tables &T, int ind, float frac, int b4) {
  return interp4(row4<16>(T.totplnk, ind - 1, b4), row4<16>(T.totplnk, ind, b4), frac);
}

__device__ __forceinline__ int pade_index(const Tables &T, float od) {
  const float tblind = od / (T.lw_bpade + od);
  const float pos = static_cast<float>(T.lw_ntbl) * tblind + 0.5f;
  return clampi(static_cast<int>(pos), 0, T.lw_ntbl);
}

// Layer transfer terms of one g-point (_rtrnmc_clear_terms/_rtrnmc_cloudy_terms,
// lw:5157-5262).
struct Terms {
  float a, gassrc, atot, bbdtot, bbdgas, bbugas, bbutot;
};

__device__ __forceinline__ Terms layer_terms(const Tables &T, bool cloudy_layer, float odepth, float odcld,
                                             float plfrac, float blay, float dplankdn, float dplankup) {
  const float rec_6 = 0.166667f;
  Terms t;
  t.atot = 0.0f;
  t.bbutot = 0.0f;
  t.bbdtot = 0.0f;
  t.gassrc = 0.0f;
  if (cloudy_layer) {
    const float odtot = odepth + odcld;
    if (odtot < 0.06f) {
      const float odepth_rec = rec_6 * odepth, odtot_rec = rec_6 * odtot;
      t.a = odepth - 0.5f * odepth * odepth;
      t.gassrc = plfrac * (blay + dplankdn * odepth_rec) * t.a;
      t.atot = odtot - 0.5f * odtot * odtot;
      t.bbdtot = plfrac * (blay + dplankdn * odtot_rec);
      t.bbdgas = plfrac * (blay + dplankdn * odepth_rec);
      t.bbugas = plfrac * (blay + dplankup * odepth_rec);
      t.bbutot = plfrac * (blay + dplankup * odtot_rec);
    } else if (odepth <= 0.06f) {
      const float odepth_rec = rec_6 * odepth;
      t.a = odepth - 0.5f * odepth * odepth;
      t.gassrc = plfrac * (blay + dplankdn * odepth_rec) * t.a;
      const int it = pade_index(T, odtot);
      const float tfactot = ld(T.lw_pade_tfn + it);
      t.atot = 1.0f - ld(T.lw_pade_exp + it);
      t.bbdtot = plfrac * (blay + tfactot * dplankdn);
      t.bbdgas = plfrac * (blay + dplankdn * odepth_rec);
      t.bbugas = plfrac * (blay + dplankup * odepth_rec);
      t.bbutot = plfrac * (blay + tfactot * dplankup);
    } else {
      const int ig = pade_index(T, odepth);
      const float odtbl = ld(T.lw_pade_tau + ig);
      t.a = 1.0f - ld(T.lw_pade_exp + ig);
      const float tfacgas = ld(T.lw_pade_tfn + ig);
      t.gassrc = t.a * plfrac * (blay + tfacgas * dplankdn);
      const float odtot3 = odtbl + odcld;
      const int it = pade_index(T, odtot3);
      const float tfactot = ld(T.lw_pade_tfn + it);
      t.atot = 1.0f - ld(T.lw_pade_exp + it);
      t.bbdtot = plfrac * (blay + tfactot * dplankdn);
      t.bbdgas = plfrac * (blay + tfacgas * dplankdn);
      t.bbugas = plfrac * (blay + tfacgas * dplankup);
      t.bbutot = plfrac * (blay + tfactot * dplankup);
    }
  } else {
    if (odepth <= 0.06f) {
      const float odepth_rec = rec_6 * odepth;
      t.a = odepth - (0.5f * odepth) * odepth;
      t.bbdgas = plfrac * (blay + dplankdn * odepth_rec);
      t.bbugas = plfrac * (blay + dplankup * odepth_rec);
    } else {
      const int it = pade_index(T, odepth);
      t.a = 1.0f - ld(T.lw_pade_exp + it);
      const float tausfac = ld(T.lw_pade_tfn + it);
      t.bbdgas = plfrac * (blay + tausfac * dplankdn);
      t.bbugas = plfrac * (blay + tausfac * dplankup);
    }
  }
  return t;
}

__device__ __forceinline__ float planck(const Tables &T, int ind, float frac, int band) {
  return interpf(ld(T.totplnk + (ind - 1) * 16 + band), ld(T.totplnk + ind * 16 + band), frac);
}

// Fields of the column context taken from the call and the 2-D inputs.
__device__ __forceinline__ void column_head(const LwArgs &a, int col, Col &C) {
  C.i = col / a.ny;
  C.j = col - C.i * a.ny;
  C.nk = a.nk;
  C.ny = a.ny;
  C.nlay = a.nlay;
  C.nbuf = a.nlay - a.nk;
  C.co2 = a.co2; C.n2o = a.n2o; C.ch4 = a.ch4; C.cfc11 = a.cfc11; C.cfc12 = a.cfc12;
  C.inflg = a.inflg; C.iceflg = a.iceflg;
  C.has_reqc = a.has_reqc; C.has_reqi = a.has_reqi; C.has_reqs = a.has_reqs; C.icloud = a.icloud;
  C.tsfc = ld(a.in.tsk + col);
  C.semiss = ld(a.in.emiss + col);
}

constexpr float kAmd = 28.9660f, kAmw = 18.0160f, kAvogad = 6.02214199e23f, kGrav = 9.8066f;

// Layer l's share of the column integrals: whether it is below the
// tropopause test pressure, its dry-air column and its water column
// (lw:1037-1064, 1263-1264).
__device__ __forceinline__ void column_layer(const Tables &T, const LwArgs &a, const Col &C, int l, bool &trop,
                                             float &coldry, float &wk0) {
  const float pavel = play_at(a, C, l);
  trop = glibc_logf(T, pavel) > 4.56f;
  const float h2o = h2o_at(a, C, l);
  const float amm = (1.0f - h2o) * kAmd + h2o * kAmw;
  const float pm = ((plev_at(a, C, l) - plev_at(a, C, l + 1)) * 1.0e3f) * kAvogad;
  float md = 1.0e2f * kGrav;
  md = md * amm;
  md = md * (1.0f + h2o);
  coldry = pm / md;
  wk0 = h2o * coldry;
}

__device__ __forceinline__ float column_pwvcm(const LwArgs &a, const Col &C, float amttl, float wvttl) {
  const float wvsh = (kAmw * wvttl) / (kAmd * amttl);
  return (wvsh * (1.0e3f * plev_at(a, C, 0))) / (1.0e2f * kGrav);
}

// Band diffusivities from the column water (lw:5520-5539).
__device__ __forceinline__ float band_secdiff(const Tables &T, const Col &C, int b) {
  const bool variable = !(b == 0 || b == 3 || b >= 9);
  if (!variable) return 1.66f;
  const float e = glibc_expf(T, kA2[b] * C.pwvcm);
  const float v = kA0[b] + kA1[b] * e;
  return v < 1.50f ? 1.50f : (v > 1.80f ? 1.80f : v);
}

__device__ __forceinline__ void column_secdiff(const Tables &T, const Col &C, float *secdiff) {
#pragma unroll
  for (int b = 0; b < kLwBands; ++b) secdiff[b] = band_secdiff(T, C, b);
}

}  // namespace
}  // namespace rrtmg
