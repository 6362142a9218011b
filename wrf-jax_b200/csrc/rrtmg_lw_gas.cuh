// Longwave gas optics (taugb1..taugb16, module_ra_rrtmg_lw.py:1597-4684) of one
// layer, four g-points at a time.
//
// Every table is read through the padded layout that the context builds once
// (rows of a multiple of four g-points, absorption tables with their edge rows
// repeated kPadRows times on both sides; see rrtmg_capi.cu), so that one
// 16-byte load serves four g-points and a row index needs one clamp instead
// of one per row.  A band's set-up (species ratios, interpolation weights,
// row offsets) is evaluated once and its g-point quads run as a loop that is
// not unrolled: fully unrolled over the g-points, the 16 bands' code did not
// fit the instruction caches (7 of 26 stall cycles per instruction were
// instruction fetch) and took one 4-byte load per g-point and row.
#pragma once

#include "rrtmg_device.cuh"

namespace rrtmg {
namespace {

constexpr int kNgc[kLwBands] = {10, 12, 16, 14, 16, 8, 12, 8, 12, 6, 8, 8, 4, 2, 2, 2};
constexpr int kGofs[kLwBands] = {0, 10, 22, 38, 52, 68, 76, 88, 96, 108, 114, 122, 130, 134, 136, 138};
constexpr float kOneMinus = 1.0f - 1.0e-6f;

struct Layer {
  float pavel, tavel, plev0, plev1, coldry;
  float wx0, wx1, wx2, wx3;
  int jp, jt, jt1, indself, indfor, indminor;
  int trop;  // l < laytrop
  float colh2o, colco2, colo3, coln2o, colco, colch4, colo2, colbrd;
  float fac00, fac01, fac10, fac11;
  float rat_h2oco2, rat_h2oco2_1, rat_h2oo3, rat_h2oo3_1, rat_h2on2o, rat_h2on2o_1;
  float rat_h2och4, rat_h2och4_1, rat_n2oco2, rat_n2oco2_1, rat_o3co2, rat_o3co2_1;
  float selffac, selffrac, forfac, forfrac, minorfrac, scaleminor, scaleminorn2;
  // Planck interpolation (lw:1210-1233): layer, lower and upper level
  int indlay, indlev0, indlev1;
  float tlayfrac, tlev0frac, tlev1frac;
  // cloud path inputs of the layer (common:877-961), zero above the model top
  float cldfrac, clwp, ciwp, cswp, rel, rei, res;
};

struct Spec {
  float sc, sp, fs;
  int js;
};

__device__ __forceinline__ Spec specint(float primary, float ratio, float secondary, float scale) {
  Spec s;
  s.sc = primary + ratio * secondary;
  const float q = primary / s.sc;
  s.sp = q > kOneMinus ? kOneMinus : q;
  const float sm = scale * s.sp;
  s.js = 1 + static_cast<int>(sm);
  s.fs = sm - floorf(sm);
  return s;
}

// Weights of the nine-species interpolation (lw:1444-1594) in the order that
// the reference adds their rows: rows r, r + 1, r + 2, r + 9, r + 10, r + 11.
// Away from the ends of the species range the third of each three is unused
// (six false, weight 0).
struct Edge {
  float w[6];
  int row;
  bool six;
};

// base: the reference's row; rows: the table's.  The padded table repeats its
// edge rows kPadRows = 12 times, so one clamp of the first row stands for the
// reference's clamp of each.
__device__ __forceinline__ Edge edge_rows(const Spec &s, int base, int rows, float fa, float fb) {
  Edge e;
  const bool low = s.sp < 0.125f;
  e.six = low || s.sp > 0.875f;
  float f0, f1, f2;
  if (e.six) {
    const float p = low ? s.fs - 1.0f : 0.0f - s.fs;
    const float p2 = p * p, p4 = p2 * p2;
    const float fk0 = p4, fk1 = (1.0f - p) - 2.0f * p4, fk2 = p + p4;
    f0 = low ? fk0 : fk2;
    f1 = fk1;
    f2 = low ? fk2 : fk0;
  } else {
    f0 = 1.0f - s.fs;
    f1 = s.fs;
    f2 = 0.0f;
  }
  e.w[0] = f0 * fa; e.w[1] = f1 * fa; e.w[2] = f2 * fa;
  e.w[3] = f0 * fb; e.w[4] = f1 * fb; e.w[5] = f2 * fb;
  e.row = clampi(e.six && !low ? base - 1 : base, -kPadRows, rows);
  return e;
}

template <int PAD>
__device__ __forceinline__ float4 edge_sum(const float *tab, const Edge &e, bool six, int q) {
  float4 s = mul4(e.w[0], row4<PAD>(tab, e.row, q));
  s = add4(s, mul4(e.w[1], row4<PAD>(tab, e.row + 1, q)));
  if (six) s = add4(s, mul4(e.w[2], row4<PAD>(tab, e.row + 2, q)));
  s = add4(s, mul4(e.w[3], row4<PAD>(tab, e.row + 9, q)));
  s = add4(s, mul4(e.w[4], row4<PAD>(tab, e.row + 10, q)));
  if (six) s = add4(s, mul4(e.w[5], row4<PAD>(tab, e.row + 11, q)));
  return s;
}

template <int PAD>
__device__ __forceinline__ float4 major4(const float *tab, int i0, int i1, int q, const Layer &L) {
  float4 s = mul4(L.fac00, row4<PAD>(tab, i0, q));
  s = add4(s, mul4(L.fac10, row4<PAD>(tab, i0 + 1, q)));
  s = add4(s, mul4(L.fac01, row4<PAD>(tab, i1, q)));
  s = add4(s, mul4(L.fac11, row4<PAD>(tab, i1 + 1, q)));
  return s;
}

// Five-species stratospheric interpolation: rows r, r + 1, r + 5, r + 6.
struct Strat {
  float w[4];
  int row;
};

__device__ __forceinline__ Strat strat_rows(float fs, int ind, int rows, float fa, float fb) {
  Strat s;
  const float comp = 1.0f - fs;
  s.w[0] = comp * fa; s.w[1] = fs * fa; s.w[2] = comp * fb; s.w[3] = fs * fb;
  s.row = clampi(ind, -kPadRows, rows);
  return s;
}

template <int PAD>
__device__ __forceinline__ float4 strat_sum(const float *tab, const Strat &e, int q) {
  float4 s = mul4(e.w[0], row4<PAD>(tab, e.row, q));
  s = add4(s, mul4(e.w[1], row4<PAD>(tab, e.row + 1, q)));
  s = add4(s, mul4(e.w[2], row4<PAD>(tab, e.row + 5, q)));
  s = add4(s, mul4(e.w[3], row4<PAD>(tab, e.row + 6, q)));
  return s;
}

__device__ __forceinline__ int ind5(int v, int rows) { return clampi(v, 0, rows - 2); }

template <int PAD>
__device__ __forceinline__ float4 lin_minor(const float *tab, int m0, float frac, int q) {
  return interp4(row4<PAD>(tab, m0, q), row4<PAD>(tab, m0 + 1, q), frac);
}

// r0 = j0 * 19 + m0
template <int PAD>
__device__ __forceinline__ float4 spec_minor(const float *tab, int r0, float fm, float frac, int q) {
  const float4 a = interp4(row4<PAD>(tab, r0, q), row4<PAD>(tab, r0 + 19, q), fm);
  const float4 b = interp4(row4<PAD>(tab, r0 + 1, q), row4<PAD>(tab, r0 + 20, q), fm);
  return interp4(a, b, frac);
}

__device__ __forceinline__ int spec_row(const Spec &s, int nspec, int m0) { return clampi(s.js - 1, 0, nspec - 2) * 19 + m0; }

template <int PAD>
__device__ __forceinline__ float4 self_tau(const LwBand &B, const Layer &L, int i0, int q) {
  return mul4(L.selffac, interp4(row4<PAD>(B.selfref, i0, q), row4<PAD>(B.selfref, i0 + 1, q), L.selffrac));
}

template <int PAD>
__device__ __forceinline__ float4 for_tau(const LwBand &B, const Layer &L, int i0, int q) {
  return mul4(L.forfac, interp4(row4<PAD>(B.forref, i0, q), row4<PAD>(B.forref, i0 + 1, q), L.forfrac));
}

__device__ __forceinline__ float chi(const Tables &T, int gas, int lev) { return ld(T.chi_mls + gas * 59 + lev); }

// Minor-gas column scaled where the gas exceeds its reference ratio by more
// than `above` (lw:134 and the bands' own constants).
template <class Adjust>
__device__ __forceinline__ float adjusted(float col, float coldry, float chi_ref, float above, Adjust adjfac) {
  const float chi_col = col / coldry;
  const float ratio = (1.0e20f * chi_col) / chi_ref;
  return ratio > above ? ((adjfac(ratio) * chi_ref) * coldry) * 1.0e-20f : col;
}

// Per-g-point corrections of bands 4 and 7 in the stratosphere, padded.
__constant__ float4 kCorr4[4] = {{1.0f, 1.0f, 1.0f, 1.0f},
                                 {1.0f, 1.0f, 1.0f, 0.92f},
                                 {0.88f, 1.07f, 1.1f, 0.99f},
                                 {0.88f, 0.943f, 1.0f, 1.0f}};
__constant__ float4 kCorr7[3] = {{1.0f, 1.0f, 1.0f, 1.0f}, {1.0f, 0.92f, 0.88f, 1.07f}, {1.1f, 0.99f, 0.855f, 1.0f}};

// ---------------------------------------------------------------------------
// Gas optics of band B at one layer: emit(q, tau, frac) with the optical
// depths and Planck fractions of g-points 4 q .. 4 q + 3 (padding g-points
// beyond the band's last get whatever the zero padding gives).
// ---------------------------------------------------------------------------
template <int B, class Emit>
__device__ __forceinline__ void gas_quads(const Tables &T, const Layer &L, Emit emit) {
  constexpr int PAD = lw_pad(B), Q = PAD / 4;
  const LwBand &K = T.lw[B];
  const int jp = L.jp, jt = L.jt, jt1 = L.jt1;
  const bool trop = L.trop;
  const int m0 = clampi(L.indminor - 1, 0, 17);
  const int is = clampi(L.indself - 1, 0, 8), ifo = clampi(L.indfor - 1, 0, 2);
  const float mf = L.minorfrac;
  if constexpr (B == 0 || B == 1 || B == 9 || B == 10 || B == 13) {
    // single-species bands 1, 2, 10, 11, 14
    const int i0 = trop ? ind5((jp - 1) * 5 + (jt - 1), K.ka_rows) : ind5((jp - 13) * 5 + (jt - 1), K.kb_rows);
    const int i1 = trop ? ind5(jp * 5 + (jt1 - 1), K.ka_rows) : ind5((jp - 12) * 5 + (jt1 - 1), K.kb_rows);
    const float *tab = trop ? K.ka : K.kb;
    const float *frac = trop ? K.fracrefa : K.fracrefb;
    float corr = 1.0f, scalen2 = 0.0f, scaleo2 = 0.0f;
    if constexpr (B == 0) {
      corr = trop ? (L.pavel < 250.0f ? 1.0f - ((0.15f * (250.0f - L.pavel)) / 154.4f) : 1.0f)
                  : 1.0f - 0.15f * (L.pavel / 95.6f);
      scalen2 = L.colbrd * L.scaleminorn2;
    }
    if constexpr (B == 1) corr = 1.0f - ((0.05f * (L.pavel - 100.0f)) / 900.0f);
    if constexpr (B == 10) scaleo2 = L.colo2 * L.scaleminor;
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const float4 major = major4<PAD>(tab, i0, i1, q, L);
      float4 tau;
      if constexpr (B == 13) {
        tau = mul4(L.colco2, major);
        if (trop) tau = add4(add4(tau, self_tau<PAD>(K, L, is, q)), for_tau<PAD>(K, L, ifo, q));
      } else {
        tau = mul4(L.colh2o, major);
        if (trop) tau = add4(tau, self_tau<PAD>(K, L, is, q));
        tau = add4(tau, for_tau<PAD>(K, L, ifo, q));
        if constexpr (B == 0) {
          const float4 taun2 = mul4(scalen2, lin_minor<PAD>(trop ? K.ka_mn2 : K.kb_mn2, m0, mf, q));
          tau = mul4(corr, add4(tau, taun2));
        }
        if constexpr (B == 1) {
          if (trop) tau = mul4(corr, tau);
        }
        if constexpr (B == 10)
          tau = add4(tau, mul4(scaleo2, lin_minor<PAD>(trop ? K.ka_mo2 : K.kb_mo2, m0, mf, q)));
      }
      emit(q, tau, row4<PAD>(frac, 0, q));
    }
  } else if constexpr (B == 5 || B == 7) {
    // bands 6 and 8: halocarbons, single species
    const float adjco2 = adjusted(L.colco2, L.coldry, chi(T, 1, clampi(jp, 0, 58)), 3.0f, [](float r) {
      return 2.0f + powf(fmaxf(r - 2.0f, 0.0f), B == 5 ? 0.77f : 0.65f);
    });
    const int i0 = trop || B == 5 ? ind5((jp - 1) * 5 + (jt - 1), K.ka_rows) : ind5((jp - 13) * 5 + (jt - 1), K.kb_rows);
    const int i1 = trop || B == 5 ? ind5(jp * 5 + (jt1 - 1), K.ka_rows) : ind5((jp - 12) * 5 + (jt1 - 1), K.kb_rows);
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const float4 x0 = mul4(B == 5 ? L.wx1 : L.wx2, row4<PAD>(B == 5 ? K.cfc11adj : K.cfc12, 0, q));
      const float4 x1 = mul4(B == 5 ? L.wx2 : L.wx3, row4<PAD>(B == 5 ? K.cfc12 : K.cfc22adj, 0, q));
      float4 tau, frac = row4<PAD>(K.fracrefa, 0, q);
      if (trop) {
        tau = mul4(L.colh2o, major4<PAD>(K.ka, i0, i1, q, L));
        tau = add4(add4(tau, self_tau<PAD>(K, L, is, q)), for_tau<PAD>(K, L, ifo, q));
        tau = add4(tau, mul4(adjco2, lin_minor<PAD>(K.ka_mco2, m0, mf, q)));
        if constexpr (B == 7) {
          tau = add4(tau, mul4(L.colo3, lin_minor<PAD>(K.ka_mo3, m0, mf, q)));
          tau = add4(tau, mul4(L.coln2o, lin_minor<PAD>(K.ka_mn2o, m0, mf, q)));
        }
        tau = add4(add4(tau, x0), x1);
      } else if constexpr (B == 5) {
        tau = add4(x0, x1);
      } else {
        tau = mul4(L.colo3, major4<PAD>(K.kb, i0, i1, q, L));
        tau = add4(tau, mul4(adjco2, lin_minor<PAD>(K.kb_mco2, m0, mf, q)));
        tau = add4(tau, mul4(L.coln2o, lin_minor<PAD>(K.kb_mn2o, m0, mf, q)));
        tau = add4(add4(tau, x0), x1);
        frac = row4<PAD>(K.fracrefb, 0, q);
      }
      emit(q, tau, frac);
    }
  } else if (trop) {
    // binary species in the troposphere: bands 3, 4, 5, 7, 9, 12, 13, 15, 16
    float prim = L.colh2o, sec, ra0, ra1, rfrac, rminor = 0.0f;
    if constexpr (B == 2 || B == 3 || B == 4 || B == 11) {
      sec = L.colco2; ra0 = L.rat_h2oco2; ra1 = L.rat_h2oco2_1;
      constexpr int lev = B == 2 ? 8 : B == 3 ? 10 : B == 4 ? 4 : 9;
      rfrac = chi(T, 0, lev) / chi(T, 1, lev);
      if constexpr (B == 2) rminor = chi(T, 0, 2) / chi(T, 1, 2);
      if constexpr (B == 4) rminor = chi(T, 0, 6) / chi(T, 1, 6);
    } else if constexpr (B == 6) {
      sec = L.colo3; ra0 = L.rat_h2oo3; ra1 = L.rat_h2oo3_1;
      rfrac = chi(T, 0, 2) / chi(T, 2, 2);
      rminor = rfrac;
    } else if constexpr (B == 8 || B == 15) {
      sec = L.colch4; ra0 = L.rat_h2och4; ra1 = L.rat_h2och4_1;
      constexpr int lev = B == 8 ? 8 : 5;
      rfrac = chi(T, 0, lev) / chi(T, 5, lev);
      if constexpr (B == 8) rminor = chi(T, 0, 2) / chi(T, 5, 2);
    } else if constexpr (B == 12) {
      sec = L.coln2o; ra0 = L.rat_h2on2o; ra1 = L.rat_h2on2o_1;
      rfrac = chi(T, 0, 4) / chi(T, 3, 4);
      rminor = chi(T, 0, 0) / chi(T, 3, 0);
    } else {
      prim = L.coln2o; sec = L.colco2; ra0 = L.rat_n2oco2; ra1 = L.rat_n2oco2_1;
      rfrac = chi(T, 3, 0) / chi(T, 1, 0);
      rminor = rfrac;
    }
    const Spec s0 = specint(prim, ra0, sec, 8.0f);
    const Spec s1 = specint(prim, ra1, sec, 8.0f);
    const Spec sp = specint(prim, rfrac, sec, 8.0f);
    const Edge e0 = edge_rows(s0, (jp - 1) * 45 + (jt - 1) * 9 + (s0.js - 1), K.ka_rows, L.fac00, L.fac10);
    const Edge e1 = edge_rows(s1, jp * 45 + (jt1 - 1) * 9 + (s1.js - 1), K.ka_rows, L.fac01, L.fac11);
    // minor species: its column and its row of the (species, temperature) table
    float minor = 0.0f, fm = 0.0f, fm3 = 0.0f;
    int rm = 0, rm3 = 0;
    if constexpr (B == 2 || B == 4 || B == 6 || B == 8 || B == 12 || B == 14) {
      const Spec sm = specint(prim, rminor, sec, 8.0f);
      rm = spec_row(sm, 9, m0);
      fm = sm.fs;
    }
    if constexpr (B == 2 || B == 8)
      minor = adjusted(L.coln2o, L.coldry, chi(T, 3, clampi(jp, 0, 58)), 1.5f,
                       [](float r) { return 0.5f + powf(r - 0.5f, 0.65f); });
    if constexpr (B == 6)
      minor = adjusted(L.colco2, L.coldry, chi(T, 1, clampi(jp, 0, 58)), 3.0f,
                       [](float r) { return 3.0f + powf(r - 3.0f, 0.79f); });
    if constexpr (B == 12) {
      minor = adjusted(L.colco2, L.coldry, 3.55e-4f, 3.0f, [](float r) { return 2.0f + powf(r - 2.0f, 0.68f); });
      const Spec s3 = specint(prim, chi(T, 0, 2) / chi(T, 3, 2), sec, 8.0f);
      rm3 = spec_row(s3, 9, m0);
      fm3 = s3.fs;
    }
    if constexpr (B == 14) minor = L.colbrd * L.scaleminor;
    const int rf = clampi(sp.js - 1, 0, 7);
    const bool six = __any_sync(__activemask(), e0.six || e1.six);
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const float4 tm0 = mul4(s0.sc, edge_sum<PAD>(K.ka, e0, six, q));
      const float4 tm1 = mul4(s1.sc, edge_sum<PAD>(K.ka, e1, six, q));
      float4 tau = add4(add4(add4(tm0, tm1), self_tau<PAD>(K, L, is, q)), for_tau<PAD>(K, L, ifo, q));
      if constexpr (B == 2 || B == 8) tau = add4(tau, mul4(minor, spec_minor<PAD>(K.ka_mn2o, rm, fm, mf, q)));
      if constexpr (B == 4) {
        tau = add4(tau, mul4(L.colo3, spec_minor<PAD>(K.ka_mo3, rm, fm, mf, q)));
        tau = add4(tau, mul4(L.wx0, row4<PAD>(K.ccl4, 0, q)));
      }
      if constexpr (B == 6 || B == 12) tau = add4(tau, mul4(minor, spec_minor<PAD>(K.ka_mco2, rm, fm, mf, q)));
      if constexpr (B == 12) tau = add4(tau, mul4(L.colco, spec_minor<PAD>(K.ka_mco, rm3, fm3, mf, q)));
      if constexpr (B == 14) tau = add4(tau, mul4(minor, spec_minor<PAD>(K.ka_mn2, rm, fm, mf, q)));
      emit(q, tau, interp4(row4<PAD>(K.fracrefa, rf, q), row4<PAD>(K.fracrefa, rf + 1, q), sp.fs));
    }
  } else if constexpr (B == 2 || B == 3 || B == 4) {
    // binary species in the stratosphere: bands 3, 4, 5
    float prim, r0, r1, rfrac;
    if constexpr (B == 2) {
      prim = L.colh2o; r0 = L.rat_h2oco2; r1 = L.rat_h2oco2_1;
      rfrac = chi(T, 0, 12) / chi(T, 1, 12);
    } else {
      prim = L.colo3; r0 = L.rat_o3co2; r1 = L.rat_o3co2_1;
      rfrac = B == 3 ? chi(T, 2, 12) / chi(T, 1, 12) : chi(T, 2, 42) / chi(T, 1, 42);
    }
    const Spec s0 = specint(prim, r0, L.colco2, 4.0f);
    const Spec s1 = specint(prim, r1, L.colco2, 4.0f);
    const Spec sp = specint(prim, rfrac, L.colco2, 4.0f);
    const Strat e0 = strat_rows(s0.fs, (jp - 13) * 25 + (jt - 1) * 5 + (s0.js - 1), K.kb_rows, L.fac00, L.fac10);
    const Strat e1 = strat_rows(s1.fs, (jp - 12) * 25 + (jt1 - 1) * 5 + (s1.js - 1), K.kb_rows, L.fac01, L.fac11);
    float minor = 0.0f;
    if constexpr (B == 2)
      minor = adjusted(L.coln2o, L.coldry, chi(T, 3, clampi(jp, 0, 58)), 1.5f,
                       [](float r) { return 0.5f + powf(r - 0.5f, 0.65f); });
    const int rm = spec_row(sp, 5, m0);  // band 3: the minor species' ratio is the fractions'
    const int rf = clampi(sp.js - 1, 0, 3);
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const float4 tm0 = mul4(s0.sc, strat_sum<PAD>(K.kb, e0, q));
      const float4 tm1 = mul4(s1.sc, strat_sum<PAD>(K.kb, e1, q));
      float4 tau = add4(tm0, tm1);
      if constexpr (B == 2)
        tau = add4(add4(tau, for_tau<PAD>(K, L, ifo, q)), mul4(minor, spec_minor<PAD>(K.kb_mn2o, rm, sp.fs, mf, q)));
      if constexpr (B == 3) tau = mul4(tau, kCorr4[q]);
      if constexpr (B == 4) tau = add4(tau, mul4(L.wx0, row4<PAD>(K.ccl4, 0, q)));
      emit(q, tau, interp4(row4<PAD>(K.fracrefb, rf, q), row4<PAD>(K.fracrefb, rf + 1, q), sp.fs));
    }
  } else if constexpr (B == 6 || B == 8) {
    // bands 7 and 9 in the stratosphere: one species and a minor one
    float minor;
    if constexpr (B == 6)
      minor = adjusted(L.colco2, L.coldry, chi(T, 1, clampi(jp, 0, 58)), 3.0f,
                       [](float r) { return 2.0f + powf(r - 2.0f, 0.79f); });
    else
      minor = adjusted(L.coln2o, L.coldry, chi(T, 3, clampi(jp, 0, 58)), 1.5f,
                       [](float r) { return 0.5f + powf(r - 0.5f, 0.65f); });
    const int i0 = ind5((jp - 13) * 5 + (jt - 1), K.kb_rows), i1 = ind5((jp - 12) * 5 + (jt1 - 1), K.kb_rows);
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const float4 major = mul4(B == 6 ? L.colo3 : L.colch4, major4<PAD>(K.kb, i0, i1, q, L));
      float4 tau = add4(major, mul4(minor, lin_minor<PAD>(B == 6 ? K.kb_mco2 : K.kb_mn2o, m0, mf, q)));
      if constexpr (B == 6) tau = mul4(tau, kCorr7[q]);
      emit(q, tau, row4<PAD>(K.fracrefb, 0, q));
    }
  } else {
    // bands 12, 13, 15, 16 in the stratosphere
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      float4 tau = make_float4(0.0f, 0.0f, 0.0f, 0.0f), frac = tau;
      if constexpr (B == 12) tau = mul4(L.colo3, lin_minor<PAD>(K.kb_mo3, m0, mf, q));
      // nspb(16) = 0: both base rows collapse to 0 (lw:4660-4663)
      if constexpr (B == 15) tau = mul4(L.colch4, major4<PAD>(K.kb, 0, 0, q, L));
      if constexpr (B == 12 || B == 15) frac = row4<PAD>(K.fracrefb, 0, q);
      emit(q, tau, frac);
    }
  }
}

}  // namespace
}  // namespace rrtmg
