// RRTMG shortwave on the GPU: the sweep schedule, from the WRF adapter to the
// theta tendencies and the 2-D surface/TOA fields.
//
// Reference call: rrtmg_swrad_wrf_columns (src/wrf_jax/physics/module_ra_rrtmg_sw.py:2386)
// and below it: inatm_sw (sw:1250), cldprmc_sw (sw:1409), setcoef_sw (sw:7101),
// taumol16..29 (sw:4043-6675), spcvmc (sw:6788-7094) with reftra (sw:3490-3601)
// and vrtqdr (sw:3604-3720), heating (sw:2285-2301), day mask (sw:2667-2719).
// The adapter passes rounding_token=None, so every statement is one binary32
// operation in the order written.
//
// Night columns (coszr <= 0) get zeros: the reference masks every output of such
// columns.  Day columns are listed and taken in chunks; per chunk the column and
// layer set-up, then every band's gas and cloud optics into layer records, then
// per g-point a top-down pass (delta-Eddington layer reflectance and
// transmittance, direct beam, downward adding recurrence) and a bottom-up pass
// (upward adding recurrence, level fluxes) whose spectral sums are taken in
// g-point order (see "Sweep schedule" below).
#include "rrtmg_device.cuh"
#include "rrtmg_divide.cuh"
#include "rrtmg_kernels.h"

namespace rrtmg {
namespace {

constexpr int kNgc[kSwBands] = {6, 12, 8, 8, 10, 10, 2, 10, 8, 6, 6, 8, 6, 12};
constexpr int kGofs[kSwBands] = {0, 6, 18, 26, 34, 44, 54, 56, 66, 74, 80, 86, 94, 100};
constexpr int kMaxLev = kMaxLay + 1;
constexpr float kOneMinus = 1.0f - 1.0e-6f;

struct Col {
  int i, j, nk, nlay, ny;
  float o3top, adjflux, mu, coszen, albedo;
  int laytrop;
  int inflg, iceflg, has_reqc, has_reqi, has_reqs, icloud;
  float co2, n2o, ch4;
};

struct SLayer {
  float pavel, tavel, pdp;
  int jp, jt, jt1, indself, indfor, trop;
  float fac00, fac01, fac10, fac11;
  float colh2o, colco2, colo3, colch4, colo2, colmol;
  float selffac, selffrac, forfac, forfrac;
  float cldfrac, clwp, ciwp, cswp, rel, rei, res;
};

// The fields of SLayer, as the sweep schedule's layer kernel stores them
// (one array per field, (layer, chunk slot) with slots fastest) for the
// band-parallel optics kernel.
#define RRTMG_SW_LAYER_FLOATS(X)                                                                           \
  X(pavel) X(tavel) X(pdp) X(fac00) X(fac01) X(fac10) X(fac11) X(colh2o) X(colco2) X(colo3) X(colch4)      \
  X(colo2) X(colmol) X(selffac) X(selffrac) X(forfac) X(forfrac) X(cldfrac) X(clwp) X(ciwp) X(cswp) X(rel) \
  X(rei) X(res)
#define RRTMG_SW_LAYER_INTS(X) X(jp) X(jt) X(jt1) X(indself) X(indfor) X(trop)
#define RRTMG_SW_COUNT(name) +1
constexpr int kSwLayerFields = 1 RRTMG_SW_LAYER_FLOATS(RRTMG_SW_COUNT) RRTMG_SW_LAYER_INTS(RRTMG_SW_COUNT);  // + cloud-water flag
#undef RRTMG_SW_COUNT
#define RRTMG_SW_INDEX(name) kSwField_##name,
enum SwField { RRTMG_SW_LAYER_FLOATS(RRTMG_SW_INDEX) RRTMG_SW_LAYER_INTS(RRTMG_SW_INDEX) kSwField_cloud_water };
#undef RRTMG_SW_INDEX
static_assert(kSwField_cloud_water + 1 == kSwLayerFields, "layer fields");

__device__ __forceinline__ float in3(const float *p, const Col &C, int k) {
  return ld(p + (static_cast<size_t>(C.i) * C.nk + k) * C.ny + C.j);
}
__device__ __forceinline__ float in3w(const float *p, const Col &C, int k) {
  return ld(p + (static_cast<size_t>(C.i) * (C.nk + 1) + k) * C.ny + C.j);
}

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

// Layer quantities: adapter extension, inatm_sw, cloud paths, setcoef_sw.
__device__ SLayer make_layer(const Tables &T, const SwArgs &a, const Col &C, int l) {
  SLayer L;
  const int nk = C.nk;
  const float plev0 = pa_to_hpa(in3w(a.in.p8w, C, l));
  const float plev1 = l + 1 <= nk ? pa_to_hpa(in3w(a.in.p8w, C, l + 1)) : 1.0e-5f;
  L.pavel = l < nk ? pa_to_hpa(in3(a.in.p3d, C, l)) : 0.5f * pa_to_hpa(in3w(a.in.p8w, C, nk));
  L.tavel = l < nk ? in3(a.in.t3d, C, l) : in3w(a.in.t8w, C, nk);
  const int kq = l < nk ? l : nk - 1;
  const float h2o = fmaxf(in3(a.in.qv, C, kq), 1.0e-12f) * 1.607793f;
  const float o3 = l < nk ? in3(a.in.o3, C, l) : C.o3top;
  // inatm_sw (sw:1286-1320)
  const float amd = 28.9660f, amw = 18.0160f, avogad = 6.02214199e23f, grav = 9.8066f;
  L.pdp = plev0 - plev1;
  const float amm = (1.0f - h2o) * amd + h2o * amw;
  const float num = (L.pdp * 1.0e3f) * avogad;
  const float den = ((1.0e2f * grav) * amm) * (1.0f + h2o);
  const float coldry = num / den;
  const float wk0 = h2o * coldry, wk1 = C.co2 * coldry, wk2 = o3 * coldry, wk3 = C.n2o * coldry;
  const float wk5 = C.ch4 * coldry, wk6 = 0.209488f * coldry;
  // setcoef_sw (sw:7101-7306)
  const float stpfac = 296.0f / 1013.0f;
  const float plog = glibc_logf(T, L.pavel);
  const int jp = clampi(static_cast<int>(36.0f - 5.0f * (plog + 0.04f)), 1, 58);
  const float fp = 5.0f * (ld(T.sw_preflog + jp - 1) - plog);
  const float tf = (L.tavel - ld(T.sw_tref + jp - 1)) / 15.0f;
  const int jt = clampi(static_cast<int>(3.0f + tf), 1, 4);
  const float ft = tf - static_cast<float>(jt - 3);
  const float tf1 = (L.tavel - ld(T.sw_tref + jp)) / 15.0f;
  const int jt1 = clampi(static_cast<int>(3.0f + tf1), 1, 4);
  const float ft1 = tf1 - static_cast<float>(jt1 - 3);
  const float water = wk0 / coldry;
  const float scalefac = (L.pavel * stpfac) / L.tavel;
  const int trop = plog > 4.56f;
  L.trop = l < C.laytrop;
  const float forfac = scalefac / (1.0f + water);
  const float ftf = (332.0f - L.tavel) / 36.0f;
  const int indfor_t = clampi(static_cast<int>(ftf), 1, 2);
  const float forfrac_t = ftf - static_cast<float>(indfor_t);
  const float fsf = (L.tavel - 188.0f) / 36.0f;
  L.indfor = trop ? indfor_t : 3;
  L.forfrac = trop ? forfrac_t : fsf - 1.0f;
  const float selffac_t = water * forfac;
  const float fself = (L.tavel - 188.0f) / 7.2f;
  const int indself_t = clampi(static_cast<int>(fself) - 7, 1, 9);
  const float selffrac_t = fself - static_cast<float>(indself_t + 7);
  L.indself = trop ? indself_t : 0;
  L.selffac = trop ? selffac_t : 0.0f;
  L.selffrac = trop ? selffrac_t : 0.0f;
  L.forfac = forfac;
  const float cs = 1.0e-20f;
  L.colh2o = cs * wk0;
  L.colco2 = cs * wk1;
  L.colo3 = cs * wk2;
  const float coln2o0 = cs * wk3;
  L.colch4 = cs * wk5;
  L.colo2 = cs * wk6;
  L.colmol = cs * coldry + L.colh2o;
  const float fallback = 1.0e-32f * coldry;
  if (L.colco2 == 0.0f) L.colco2 = fallback;
  (void)coln2o0;
  if (L.colch4 == 0.0f) L.colch4 = fallback;
  if (L.colo2 == 0.0f) L.colo2 = fallback;
  const float compfp = 1.0f - fp;
  L.fac10 = compfp * ft;
  L.fac00 = compfp * (1.0f - ft);
  L.fac11 = fp * ft1;
  L.fac01 = fp * (1.0f - ft1);
  L.jp = jp;
  L.jt = jt;
  L.jt1 = jt1;
  // cloud radii and paths (common:801-961); zero in the extra top layer
  L.cldfrac = 0.0f; L.clwp = 0.0f; L.ciwp = 0.0f; L.cswp = 0.0f;
  L.rel = 10.0f; L.rei = 10.0f; L.res = 10.0f;
  if (l < nk) {
    const float t = L.tavel;
    const float cldfra = in3(a.in.cldfra, C, l);
    float qc = fmaxf(in3(a.in.qc, C, l), 0.0f), qi = fmaxf(in3(a.in.qi, C, l), 0.0f);
    float qs = fmaxf(in3(a.in.qs, C, l), 0.0f);
    const int c2 = C.i * C.ny + C.j;
    const float xland = ld(a.in.xland + c2);
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
    const float dp = L.pdp;
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
    const float xice = ld(a.in.xice + c2), snow = ld(a.in.snow + c2);
    const float landm = 2.0f - xland, snowh = 0.001f * snow;
    const float rocean = 14.0f, rland = 8.0f, rice = 14.0f;
    float rel = rland + (rocean - rland) * fminf(1.0f, fmaxf(0.0f, (273.16f - t) * 0.05f));
    rel = rel + (rocean - rel) * fminf(1.0f, fmaxf(0.0f, snowh * 10.0f));
    rel = rel + (rocean - rel) * fminf(1.0f, fmaxf(0.0f, 1.0f - landm));
    rel = rel + (rice - rel) * fminf(1.0f, fmaxf(0.0f, xice));
    float rei = retab_interp(T, t, 94);
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
// taumol16..29 (sw:4043-6675), four g-points at a time from the padded tables
// (rrtmg_device.cuh): the set-up of a band once, its quads in a loop that is
// not unrolled (unrolled over single g-points the 14 bands' code overran the
// instruction caches: 10 of 26 stall cycles per instruction).
// ---------------------------------------------------------------------------
struct SwSpec {
  float sc, fs;
  int js0;
};

__device__ __forceinline__ SwSpec sw_species(float primary, float ratio_secondary, float scale, int cap) {
  SwSpec s;
  s.sc = primary + ratio_secondary;
  const float q = primary / s.sc;
  const float sp = q > kOneMinus ? kOneMinus : q;
  const float sm = scale * sp;
  const int js = 1 + static_cast<int>(sm);
  s.fs = sm - floorf(sm);
  s.js0 = clampi(js - 1, 0, cap);
  return s;
}

// The species ratio of band B (0 = band 16); its eight-interval form below
// laytrop (kLow) or the four-interval one of the bands that have two there.
template <int B, bool kLow, class Field>
__device__ __forceinline__ SwSpec sw_band_species(const SwBand &K, Field field) {
  constexpr int bn = B + 16;
  constexpr float scale = kLow ? 8.0f : 4.0f;
  constexpr int cap = kLow ? 7 : 3;
  if constexpr (bn == 16) return sw_species(field(kSwField_colh2o), K.strrat1 * field(kSwField_colch4), scale, cap);
  if constexpr (bn == 17 || bn == 19 || bn == 21)
    return sw_species(field(kSwField_colh2o), K.strrat * field(kSwField_colco2), scale, cap);
  if constexpr (bn == 18) return sw_species(field(kSwField_colh2o), K.strrat * field(kSwField_colch4), scale, cap);
  if constexpr (bn == 22)
    return sw_species(field(kSwField_colh2o), (1.6f * K.strrat) * field(kSwField_colo2), scale, cap);
  if constexpr (bn == 24) return sw_species(field(kSwField_colh2o), K.strrat * field(kSwField_colo2), scale, cap);
  if constexpr (bn == 28) return sw_species(field(kSwField_colo3), K.strrat * field(kSwField_colo2), scale, cap);
  return SwSpec{0.0f, 0.0f, 0};
}

// Two-species interpolation over pressure, temperature and species ratio:
// rows r0, r0 + 1, r0 + NS, r0 + NS + 1 and the same from r1, in this order.
struct SwRows8 {
  float f[8];
  int r0, r1;
};

template <int NS>
__device__ __forceinline__ SwRows8 sw_rows8(const SwSpec &s, const SLayer &L, int jt0, int jt10, int jp0, int jp1) {
  SwRows8 k;
  const float comp = 1.0f - s.fs;
  k.f[0] = comp * L.fac00;
  k.f[1] = s.fs * L.fac00;
  k.f[2] = comp * L.fac10;
  k.f[3] = s.fs * L.fac10;
  k.f[4] = comp * L.fac01;
  k.f[5] = s.fs * L.fac01;
  k.f[6] = comp * L.fac11;
  k.f[7] = s.fs * L.fac11;
  k.r0 = (jp0 * 5 + jt0) * NS + s.js0;
  k.r1 = (jp1 * 5 + jt10) * NS + s.js0;
  return k;
}

template <int PAD, int NS>
__device__ __forceinline__ float4 sum8(const float *tab, const SwRows8 &k, int q) {
  float4 s = mul4(k.f[0], row4<PAD>(tab, k.r0, q));
  s = add4(s, mul4(k.f[1], row4<PAD>(tab, k.r0 + 1, q)));
  s = add4(s, mul4(k.f[2], row4<PAD>(tab, k.r0 + NS, q)));
  s = add4(s, mul4(k.f[3], row4<PAD>(tab, k.r0 + NS + 1, q)));
  s = add4(s, mul4(k.f[4], row4<PAD>(tab, k.r1, q)));
  s = add4(s, mul4(k.f[5], row4<PAD>(tab, k.r1 + 1, q)));
  s = add4(s, mul4(k.f[6], row4<PAD>(tab, k.r1 + NS, q)));
  s = add4(s, mul4(k.f[7], row4<PAD>(tab, k.r1 + NS + 1, q)));
  return s;
}

// One-species interpolation, rows (pressure * 5 + temperature).
template <int PAD>
__device__ __forceinline__ float4 sum4(const float *tab, int r0, int r1, const SLayer &L, int q) {
  float4 s = mul4(L.fac00, row4<PAD>(tab, r0, q));
  s = add4(s, mul4(L.fac10, row4<PAD>(tab, r0 + 1, q)));
  s = add4(s, mul4(L.fac01, row4<PAD>(tab, r1, q)));
  s = add4(s, mul4(L.fac11, row4<PAD>(tab, r1 + 1, q)));
  return s;
}

// Gas and Rayleigh optical depths of band B (0 = band 16) at one layer:
// emit(q, taug, taur) for g-points 4 q .. 4 q + 3.  field: the layer fields.
template <int B, class Field, class Emit>
__device__ __forceinline__ void sw_quads(const Tables &T, const SLayer &L, Field field, Emit emit) {
  constexpr int PAD = sw_pad(B), Q = PAD / 4, bn = B + 16;
  const SwBand &K = T.sw[B];
  const bool trop = L.trop;
  const int jp = L.jp;
  const int jt0 = clampi(L.jt - 1, 0, 3), jt10 = clampi(L.jt1 - 1, 0, 3);
  const int jp0 = clampi(jp - 1, 0, 11), jp1 = jp0 + 1;
  const int kjp0 = clampi(jp - 13, 0, 45), kjp1 = clampi(jp - 12, 0, 46);
  const float colh2o = L.colh2o, colmol = L.colmol;
  // bands with two species below laytrop, and those with two above it too
  constexpr bool two = bn == 16 || bn == 17 || bn == 18 || bn == 19 || bn == 21 || bn == 22 || bn == 24 || bn == 28;
  constexpr bool two_above = bn == 17 || bn == 21 || bn == 28;
  SwSpec sp8{0.0f, 0.0f, 0};
  if constexpr (two) sp8 = sw_band_species<B, true>(K, field);
  SwRows8 k8{};
  if constexpr (two) {
    if (trop) {
      k8 = sw_rows8<9>(sp8, L, jt0, jt10, jp0, jp1);
    } else if constexpr (two_above) {
      k8 = sw_rows8<5>(sw_band_species<B, false>(K, field), L, jt0, jt10, kjp0, kjp1);
    }
  }
  const int r0 = trop ? jp0 * 5 + jt0 : kjp0 * 5 + jt0, r1 = trop ? jp1 * 5 + jt10 : kjp1 * 5 + jt10;
  const int is = clampi(L.indself - 1, 0, 8);
  constexpr int fcap = bn == 16 || bn == 23 || bn == 24 ? 1 : 2;
  const int if0 = clampi(L.indfor - 1, 0, fcap), if1 = jrow(if0 + 1, K.forref_rows);
  const float selffrac = L.selffrac, forfrac = L.forfrac, selffac = L.selffac, forfac = L.forfac;
  auto self = [&](int q) {
    return mul4(selffac, interp4(row4<PAD>(K.selfref, is, q), row4<PAD>(K.selfref, is + 1, q), selffrac));
  };
  auto foreign_raw = [&](int q) {
    return interp4(row4<PAD>(K.forref, if0, q), row4<PAD>(K.forref, if1, q), forfrac);
  };
  auto foreign = [&](int q) { return mul4(forfac, foreign_raw(q)); };
  const float o2cont = bn == 22 ? (4.35e-4f * L.colo2) / (350.0f * 2.0f) : 0.0f;
  const float ray = colmol * K.rayl;
#pragma unroll 1
  for (int q = 0; q < Q; ++q) {
    float4 tg = make_float4(0.0f, 0.0f, 0.0f, 0.0f), tr = make_float4(ray, ray, ray, ray);
    if constexpr (bn == 16 || bn == 17 || bn == 18 || bn == 19 || bn == 21 || bn == 22) {
      if (trop) {
        const float4 cont = mul4(colh2o, add4(self(q), foreign(q)));
        tg = add4(mul4(sp8.sc, sum8<PAD, 9>(K.ka, k8, q)), cont);
        if constexpr (bn == 22) tg = add4(tg, make_float4(o2cont, o2cont, o2cont, o2cont));
      } else if constexpr (bn == 17 || bn == 21) {
        const float4 cont = mul4(colh2o * forfac, foreign_raw(q));
        tg = add4(mul4(sp8.sc, sum8<PAD, 5>(K.kb, k8, q)), cont);
      } else if constexpr (bn == 22) {
        tg = add4(mul4(L.colo2 * 1.6f, sum4<PAD>(K.kb, r0, r1, L, q)), make_float4(o2cont, o2cont, o2cont, o2cont));
      } else {
        tg = mul4(bn == 19 ? L.colco2 : L.colch4, sum4<PAD>(K.kb, r0, r1, L, q));
      }
    } else if constexpr (bn == 20) {
      float4 inner = sum4<PAD>(trop ? K.ka : K.kb, r0, r1, L, q);
      if (trop) inner = add4(inner, self(q));
      inner = add4(inner, foreign(q));
      tg = add4(mul4(colh2o, inner), mul4(L.colch4, row4<PAD>(K.absch4, 0, q)));
    } else if constexpr (bn == 23) {
      if (trop)
        tg = mul4(colh2o, add4(add4(mul4(K.givfac, sum4<PAD>(K.ka, r0, r1, L, q)), self(q)), foreign(q)));
      tr = mul4(colmol, row4<PAD>(K.rayl_g, 0, q));
    } else if constexpr (bn == 24) {
      if (trop) {
        const float4 cont = mul4(colh2o, add4(self(q), foreign(q)));
        tg = add4(add4(mul4(sp8.sc, sum8<PAD, 9>(K.ka, k8, q)), mul4(L.colo3, row4<PAD>(K.abso3a, 0, q))), cont);
        tr = mul4(colmol, interp4(row4<PAD>(K.rayla, sp8.js0, q), row4<PAD>(K.rayla, sp8.js0 + 1, q), sp8.fs));
      } else {
        tg = add4(mul4(L.colo2, sum4<PAD>(K.kb, r0, r1, L, q)), mul4(L.colo3, row4<PAD>(K.abso3b, 0, q)));
        tr = mul4(colmol, row4<PAD>(K.raylb, 0, q));
      }
    } else if constexpr (bn == 25) {
      if (trop)
        tg = add4(mul4(colh2o, sum4<PAD>(K.ka, r0, r1, L, q)), mul4(L.colo3, row4<PAD>(K.abso3a, 0, q)));
      else
        tg = mul4(L.colo3, row4<PAD>(K.abso3b, 0, q));
      tr = mul4(colmol, row4<PAD>(K.rayl_g, 0, q));
    } else if constexpr (bn == 26) {
      tr = mul4(colmol, row4<PAD>(K.rayl_g, 0, q));
    } else if constexpr (bn == 27) {
      tg = mul4(L.colo3, sum4<PAD>(trop ? K.ka : K.kb, r0, r1, L, q));
      tr = mul4(colmol, row4<PAD>(K.rayl_g, 0, q));
    } else if constexpr (bn == 28) {
      tg = mul4(sp8.sc, trop ? sum8<PAD, 9>(K.ka, k8, q) : sum8<PAD, 5>(K.kb, k8, q));
    } else {  // 29
      const float4 k = sum4<PAD>(trop ? K.ka : K.kb, r0, r1, L, q);
      if (trop)
        tg = add4(mul4(colh2o, add4(add4(k, self(q)), foreign(q))), mul4(L.colco2, row4<PAD>(K.absco2, 0, q)));
      else
        tg = add4(mul4(L.colco2, k), mul4(colh2o, row4<PAD>(K.absh2o, 0, q)));
    }
    emit(q, tg, tr);
  }
}

// cldprmc_sw for one cloudy (band, layer) (sw:1409-1626; ice >= 3, liquid 1)
struct CloudOpt {
  float tau, ssa, asm_, taor;
  bool active;
};

__device__ CloudOpt sw_cloud(const Tables &T, const SLayer &L, int band, int iceflag) {
  CloudOpt o;
  const float cldmin = 1.0e-20f;
  const float ciwp = L.ciwp, clwp = L.clwp, cswp = iceflag == 5 ? L.cswp : 0.0f;
  const float cwp = (ciwp + clwp) + cswp;
  o.active = cwp >= cldmin;
  const float radice = L.rei, radliq = L.rel, radsno = iceflag == 5 ? L.res : 0.0f;
  const float factor = (radice - 2.0f) / 3.0f;
  int index = static_cast<int>(factor);
  if (index == 46) index = 45;
  const float fint = factor - static_cast<float>(index);
  const int r0 = jrow(index - 1, 46), r1 = jrow(index, 46);
  float extice = interpf(ld(T.extice3 + r0 * 14 + band), ld(T.extice3 + r1 * 14 + band), fint);
  float ssaice = interpf(ld(T.ssaice3 + r0 * 14 + band), ld(T.ssaice3 + r1 * 14 + band), fint);
  float gice = interpf(ld(T.asyice3 + r0 * 14 + band), ld(T.asyice3 + r1 * 14 + band), fint);
  const float fdelta = interpf(ld(T.fdlice3 + r0 * 14 + band), ld(T.fdlice3 + r1 * 14 + band), fint);
  const float fw = fdelta + 0.5f / ssaice;
  float forwice = fw > gice ? gice : fw;
  if ((ciwp + cswp) == 0.0f) { extice = 0.0f; ssaice = 0.0f; gice = 0.0f; forwice = 0.0f; }
  float extsno = 0.0f, ssasno = 0.0f, gsno = 0.0f, forwsno = 0.0f;
  if (iceflag == 5 && cswp > 0.0f) {
    const float fs = (radsno - 2.0f) / 3.0f;
    int is = static_cast<int>(fs);
    if (is == 46) is = 45;
    const float fints = fs - static_cast<float>(is);
    const int s0 = jrow(is - 1, 46), s1 = jrow(is, 46);
    extsno = interpf(ld(T.extice3 + s0 * 14 + band), ld(T.extice3 + s1 * 14 + band), fints);
    ssasno = interpf(ld(T.ssaice3 + s0 * 14 + band), ld(T.ssaice3 + s1 * 14 + band), fints);
    gsno = interpf(ld(T.asyice3 + s0 * 14 + band), ld(T.asyice3 + s1 * 14 + band), fints);
    const float fds = interpf(ld(T.fdlice3 + s0 * 14 + band), ld(T.fdlice3 + s1 * 14 + band), fints);
    const float fw2 = fds + 0.5f / ssasno;
    forwsno = fw2 > gsno ? gsno : fw2;
  }
  int il = static_cast<int>(radliq - 1.5f);
  if (il == 0) il = 1;
  if (il == 58) il = 57;
  const float fint_liq = (radliq - 1.5f) - static_cast<float>(il);
  const int q0 = jrow(il - 1, 58), q1 = jrow(il, 58);
  float extliq = interpf(ld(T.extliq1 + q0 * 14 + band), ld(T.extliq1 + q1 * 14 + band), fint_liq);
  float ssaliq = interpf(ld(T.ssaliq1 + q0 * 14 + band), ld(T.ssaliq1 + q1 * 14 + band), fint_liq);
  if (fint_liq < 0.0f && ssaliq > 1.0f) ssaliq = ld(T.ssaliq1 + q0 * 14 + band);
  float gliq = interpf(ld(T.asyliq1 + q0 * 14 + band), ld(T.asyliq1 + q1 * 14 + band), fint_liq);
  if (clwp == 0.0f) { extliq = 0.0f; ssaliq = 0.0f; gliq = 0.0f; }
  const float forwliq = gliq * gliq;
  const float tauliqorig = clwp * extliq;
  const float tauiceorig = ciwp * extice;
  const float ssaliq_d = ssaliq * (1.0f - forwliq) / (1.0f - forwliq * ssaliq);
  const float tauliq = (1.0f - forwliq * ssaliq) * tauliqorig;
  const float ssaice_d = ssaice * (1.0f - forwice) / (1.0f - forwice * ssaice);
  const float tauice = (1.0f - forwice * ssaice) * tauiceorig;
  const float scatliq = ssaliq_d * tauliq;
  float scatice = ssaice_d * tauice;
  float tau_new, taor_new, scatsno = 0.0f;
  if (iceflag == 5) {
    const float tausnoorig = cswp * extsno;
    const float ssasno_d = ssasno * (1.0f - forwsno) / (1.0f - forwsno * ssasno);
    const float tausno = (1.0f - forwsno * ssasno) * tausnoorig;
    scatsno = ssasno_d * tausno;
    tau_new = (tauliq + tauice) + tausno;
    taor_new = (tauliqorig + tauiceorig) + tausnoorig;
  } else {
    tau_new = tauliq + tauice;
    taor_new = tauliqorig + tauiceorig;
  }
  if (tau_new == 0.0f) tau_new = cldmin;
  if (scatice == 0.0f) scatice = cldmin;
  if (scatsno == 0.0f) scatsno = cldmin;
  if (iceflag == 5) {
    const float ssum = (scatliq + scatice) + scatsno;
    o.ssa = ssum / tau_new;
    const float num = (scatliq * (gliq - forwliq) / (1.0f - forwliq) + scatice * (gice - forwice) / (1.0f - forwice)) +
                      scatsno * (gsno - forwsno) / (1.0f - forwsno);
    o.asm_ = num / ssum;
  } else {
    const float ssum = scatliq + scatice;
    o.ssa = ssum / tau_new;
    const float num = scatliq * (gliq - forwliq) / (1.0f - forwliq) + scatice * (gice - forwice) / (1.0f - forwice);
    o.asm_ = num / ssum;
  }
  o.tau = tau_new;
  o.taor = taor_new;
  if (!o.active) { o.tau = 0.0f; o.ssa = 1.0f; o.asm_ = 0.0f; o.taor = 0.0f; }
  return o;
}

__device__ __forceinline__ float exp_lookup(const Tables &T, float v) {
  if (v <= 0.06f) return (1.0f - v) + (0.5f * v) * v;
  const float tblind = v / (T.sw_bpade + v);
  const int it = clampi(static_cast<int>(static_cast<float>(T.sw_ntbl) * tblind + 0.5f), 0, T.sw_ntbl);
  return ld(T.sw_pade_exp + it);
}

struct RT4 {
  float ref, refd, tra, trad;
};

// exp_lookup of min(v, 500) given ex_v = exp_lookup(v) (reftra's clamp of
// its exponent arguments, sw:3530-3545)
__device__ __forceinline__ float lookup_clamped(const Tables &T, float v, float ex_v) {
  return v > 500.0f ? exp_lookup(T, 500.0f) : ex_v;
}

// x / d, or x itself when d is exactly 1 (then the quotient is x exactly).
__device__ __forceinline__ float div_or_same(float x, float d) { return d == 1.0f ? x : x / d; }

// 0 / x as IEEE binary32 division computes it: a zero with the sign of x, or
// the canonical NaN when x is zero or NaN.
__device__ __forceinline__ float zero_over(float x) {
  if (x == 0.0f || x != x) return __int_as_float(0x7fffffff);
  return __int_as_float(__float_as_int(x) & static_cast<int>(0x80000000u));
}

// FP64 mode: the Pade lookup of exp(-v) (sw:2722-2760) with binary64
// arithmetic; the table is the same binary32 data.
__device__ __forceinline__ double exp_lookup64(const Tables &T, double v) {
  if (v <= 0.06) return (1.0 - v) + (0.5 * v) * v;
  const double tblind = v / (static_cast<double>(T.sw_bpade) + v);
  const int it = clampi(static_cast<int>(static_cast<double>(T.sw_ntbl) * tblind + 0.5), 0, T.sw_ntbl);
  return static_cast<double>(ld(T.sw_pade_exp + it));
}

// FP64 mode's reftra (sw:3490-3601) for a layer whose delta-scaled
// single-scattering albedo zwo is >= 0.999 or whose optical depth zto1 is
// below 0.1: both branches in binary64 on the binary32 inputs, the four
// results rounded once.  Near zwo = 1 the general branch's g1 * g1 - g2 * g2
// cancels (its binary32 relative error grows as 1 / (1 - zw)); for a thin
// layer the O(1) terms of the reflectance and transmittance numerators cancel
// to O(zto1), and in binary32 a layer of optical depth 5e-4 can come out with
// a negative reflectance and 70% transmittance instead of 99.96%.
__device__ __noinline__ RT4 reftra64(const Tables &T, float zg_in, float mu_in, float zto1_in, float zw_in) {
  const double zg = zg_in, mu = mu_in, zto1 = zto1_in, zw = zw_in;
  const double eps = 1.0e-8, zwcrit = 0.9999995;
  double ref, refd, tra, trad;
  const double zg3 = 3.0 * zg;
  const double g1 = (8.0 - zw * (5.0 + zg3)) * 0.25;
  const double g2 = 3.0 * (zw * (1.0 - zg)) * 0.25;
  const double g3 = (2.0 - zg3 * mu) * 0.25;
  const double g4 = 1.0 - g3;
  const double sr = zg != 1.0 ? zg / (1.0 - zg) : 0.0;
  const double denom = zg != 1.0 ? 1.0 - (1.0 - zw) * sr * sr : 1.0;
  const double zwo = (zw > 0.0 && denom != 0.0) ? zw / denom : 0.0;
  double ze2 = zto1 / mu;
  if (ze2 > 500.0) ze2 = 500.0;
  const double zem2 = exp_lookup64(T, ze2);
  if (zwo >= zwcrit) {
    const double za = g1 * mu;
    const double za1 = za - g3;
    const double zgt = g1 * zto1;
    ref = (zgt - za1 * (1.0 - zem2)) / (1.0 + zgt);
    tra = 1.0 - ref;
    refd = zgt / (1.0 + zgt);
    trad = 1.0 - refd;
    if (zem2 == 1.0) { ref = 0.0; tra = 1.0; refd = 0.0; trad = 1.0; }
  } else {
    const double za1 = g1 * g4 + g2 * g3;
    const double za2 = g1 * g3 + g2 * g4;
    const double rad = g1 * g1 - g2 * g2;
    const double zrk = sqrt(rad > 0.0 ? rad : 0.0);
    const double zrp = zrk * mu;
    const double zrp1 = 1.0 + zrp, zrm1 = 1.0 - zrp, zrk2 = 2.0 * zrk;
    const double zrpp = 1.0 - zrp * zrp;
    const double zrkg = zrk + g1;
    const double zr1 = zrm1 * (za2 + zrk * g3);
    const double zr2 = zrp1 * (za2 - zrk * g3);
    const double zr3 = zrk2 * (g3 - za2 * mu);
    const double zr4 = zrpp * zrkg;
    const double zr5 = zrpp * (zrk - g1);
    const double zt1 = zrp1 * (za1 + zrk * g4);
    const double zt2 = zrm1 * (za1 - zrk * g4);
    const double zt3 = zrk2 * (g4 + za1 * mu);
    const double zbeta = (g1 - zrk) / zrkg;
    double ze1 = zrk * zto1;
    if (ze1 > 500.0) ze1 = 500.0;
    const double zem1 = exp_lookup64(T, ze1);
    const double zep1 = 1.0 / zem1;
    const double zep2 = 1.0 / zem2;
    const double zdenr = zr4 * zep1 + zr5 * zem1;
    const double zdent = zr4 * zep1 + zr5 * zem1;
    if (zdenr >= -eps && zdenr <= eps) {
      ref = eps;
      tra = zem2;
    } else {
      ref = zw * (zr1 * zep1 - zr2 * zem1 - zr3 * zem2) / zdenr;
      tra = zem2 - zem2 * zw * (zt1 * zep1 - zt2 * zem1 - zt3 * zep2) / zdent;
    }
    const double zemm = zem1 * zem1;
    const double zdend = 1.0 / ((1.0 - zbeta * zemm) * zrkg);
    refd = g2 * (1.0 - zemm) * zdend;
    trad = zrk2 * zem1 * zdend;
  }
  RT4 r;
  r.ref = static_cast<float>(ref);
  r.refd = static_cast<float>(refd);
  r.tra = static_cast<float>(tra);
  r.trad = static_cast<float>(trad);
  return r;
}

// Delta-Eddington layer reflectance/transmittance (reftra_sw_columns,
// sw:3490-3601) of a layer that scatters (the reference's lrt = true).
// zto1_mu = zto1 / mu and ex_zto1_mu = exp_lookup(zto1_mu) come from the
// caller, which needs the same quotient and lookup for its direct beam.
// Divisions whose divisor is exactly 1 are skipped: their quotient is the
// dividend, bit for bit.
// kFp64: the FP64 mode, which hands layers with zwo >= 0.999 or zto1 < 0.1
// to reftra64.
template <bool kFp64>
__device__ __forceinline__ RT4 reftra(const Tables &T, float zg, float mu, float zto1, float zw, float zto1_mu,
                                      float ex_zto1_mu) {
  RT4 r;
  const float eps = 1.0e-8f, zwcrit = 0.9999995f;
  const float zg3 = 3.0f * zg;
  const float g1 = (8.0f - zw * (5.0f + zg3)) * 0.25f;
  const float g2 = 3.0f * (zw * (1.0f - zg)) * 0.25f;
  const float g3 = (2.0f - zg3 * mu) * 0.25f;
  const float g4 = 1.0f - g3;
  const float sr = zg != 1.0f ? div_or_same(zg, 1.0f - zg) : 0.0f;
  const float denom = zg != 1.0f ? 1.0f - (1.0f - zw) * sr * sr : 1.0f;
  const float zwo = (zw > 0.0f && denom != 0.0f) ? div_or_same(zw, denom) : 0.0f;
  if constexpr (kFp64) {
    if (zwo >= 0.999f || zto1 < 0.1f) return reftra64(T, zg, mu, zto1, zw);
  }
  if (zwo >= zwcrit) {
    const float za = g1 * mu;
    const float za1 = za - g3;
    const float zgt = g1 * zto1;
    const float ex = lookup_clamped(T, zto1_mu, ex_zto1_mu);
    r.ref = (zgt - za1 * (1.0f - ex)) / (1.0f + zgt);
    r.tra = 1.0f - r.ref;
    r.refd = zgt / (1.0f + zgt);
    r.trad = 1.0f - r.refd;
    if (ex == 1.0f) { r.ref = 0.0f; r.tra = 1.0f; r.refd = 0.0f; r.trad = 1.0f; }
    return r;
  }
  const float za1 = g1 * g4 + g2 * g3;
  const float za2 = g1 * g3 + g2 * g4;
  const float rad = g1 * g1 - g2 * g2;
  const float zrk = sqrtf(rad > 0.0f ? rad : 0.0f);
  const float zrp = zrk * mu;
  const float zrp1 = 1.0f + zrp, zrm1 = 1.0f - zrp, zrk2 = 2.0f * zrk;
  const float zrpp = 1.0f - zrp * zrp;
  const float zrkg = zrk + g1;
  const float zr1 = zrm1 * (za2 + zrk * g3);
  const float zr2 = zrp1 * (za2 - zrk * g3);
  const float zr3 = zrk2 * (g3 - za2 * mu);
  const float zr4 = zrpp * zrkg;
  const float zr5 = zrpp * (zrk - g1);
  const float zt1 = zrp1 * (za1 + zrk * g4);
  const float zt2 = zrm1 * (za1 - zrk * g4);
  const float zt3 = zrk2 * (g4 + za1 * mu);
  const float zbeta = (g1 - zrk) / zrkg;
  float ze1 = zrk * zto1;
  if (ze1 > 500.0f) ze1 = 500.0f;
  const float zem1 = exp_lookup(T, ze1);
  const float zep1 = 1.0f / zem1;
  const float zem2 = lookup_clamped(T, zto1_mu, ex_zto1_mu);
  const float zep2 = 1.0f / zem2;
  const float zdenr = zr4 * zep1 + zr5 * zem1;
  const float zdent = zr4 * zep1 + zr5 * zem1;
  if ((zdenr >= -eps) && (zdenr <= eps)) {
    r.ref = eps;
    r.tra = zem2;
  } else {
    r.ref = zw * (zr1 * zep1 - zr2 * zem1 - zr3 * zem2) / zdenr;
    r.tra = zem2 - zem2 * zw * (zt1 * zep1 - zt2 * zem1 - zt3 * zep2) / zdent;
  }
  const float zemm = zem1 * zem1;
  const float zdend = 1.0f / ((1.0f - zbeta * zemm) * zrkg);
  r.refd = g2 * (1.0f - zemm) * zdend;
  r.trad = zrk2 * zem1 * zdend;
  return r;
}

// ---------------------------------------------------------------------------
// Layer optics of one g-point for the sweep: delta-Eddington results and the
// direct beam's transmittances with and without delta scaling.
// ---------------------------------------------------------------------------
struct SwOptics {
  RT4 rt;
  float dbt, dbt_nd;
};

// The clear-sky layer's inputs that the cloudy one builds on, and whether the
// checked form below served it.
struct SwClear {
  float ztau, ztauc, zomcc, zgcc;
  bool checked;
};

// Clear sky, any operands: gas + Rayleigh, no aerosol (sw:6923-6927).  Divisions
// whose divisor is exactly 1 are skipped: their quotient is the dividend.
template <bool kFp64>
__device__ __forceinline__ SwOptics sw_clear_any(const Tables &T, float tg, float tr, float mu, SwClear &c) {
  SwOptics o;
  c.checked = false;
  c.ztau = (tr + tg) + 0.0f;
  const float zom0 = tr + 0.0f * 1.0f;
  const float zgr = zero_over(zom0);  // 0 * 1 * 0 / zom
  const float zom = zom0 / c.ztau;
  const float v_nd = c.ztau / mu;
  o.dbt_nd = exp_lookup(T, v_nd);
  const float zf = zgr * zgr;
  const float zwf = zom * zf;
  const float d_w = 1.0f - zwf;
  c.ztauc = d_w * c.ztau;
  c.zomcc = div_or_same(zom - zwf, d_w);
  c.zgcc = div_or_same(zgr - zf, 1.0f - zf);
  // ztauc is ztau exactly when d_w == 1
  const float v_c = d_w == 1.0f ? v_nd : c.ztauc / mu;
  o.dbt = d_w == 1.0f ? o.dbt_nd : exp_lookup(T, v_c);
  o.rt = reftra<kFp64>(T, c.zgcc, mu, c.ztauc, c.zomcc, v_c, o.dbt);
  return o;
}

// A cloudy g-point layer, any operands (sw:6935-7010): cld = the band's cloud
// (tau, ssa, asm, unscaled tau).  The reference's mix clear * c + cloud * o has
// clear = 0, cloud = 1 here.
template <bool kFp64>
__device__ __forceinline__ SwOptics sw_cloudy_any(const Tables &T, const SwClear &c, const SwOptics &oc, float4 cld,
                                                  float mu) {
  const float clear = 0.0f, cloud = 1.0f;
  const float tcld = cld.x, wcld = cld.y, gcld = cld.z, taor = cld.w;
  const float dbtmo_nd = exp_lookup(T, (c.ztau + taor) / mu);
  const float ztauo = c.ztauc + tcld;
  float zomco = c.ztauc * c.zomcc + tcld * wcld;
  const float zgco = (tcld * wcld * gcld + c.ztauc * c.zomcc * c.zgcc) / zomco;
  zomco = zomco / ztauo;
  const float v_o = ztauo / mu;
  const float dbtmo = exp_lookup(T, v_o);
  const RT4 o = reftra<kFp64>(T, zgco, mu, ztauo, zomco, v_o, dbtmo);
  SwOptics t;
  t.dbt_nd = clear * oc.dbt_nd + cloud * dbtmo_nd;
  t.rt.ref = clear * oc.rt.ref + cloud * o.ref;
  t.rt.refd = clear * oc.rt.refd + cloud * o.refd;
  t.rt.tra = clear * oc.rt.tra + cloud * o.tra;
  t.rt.trad = clear * oc.rt.trad + cloud * o.trad;
  t.dbt = clear * oc.dbt + cloud * dbtmo;
  return t;
}

// ---------------------------------------------------------------------------
// The same layers with their operands checked once: every division is then
// within the ranges of rrtmg_divide.cuh, quotients by mu and by equal divisors
// share a reciprocal, and the reciprocals of table exponentials come from the
// table.  `ok` turns false where an operand is outside (the caller then takes
// the *_any form); inside, the results are the same bits.  (Where a zero
// differs only in its sign it stays a zero in every flux.)
// ---------------------------------------------------------------------------
constexpr float kSafeLow = 0x1p-90f, kSafeHigh = 0x1p60f;

struct SwExp {
  float e, r;  // exp(-v) by the table or the series, and its reciprocal
};

__device__ __forceinline__ SwExp exp_pair(const Tables &T, float v) {
  SwExp x;
  if (v <= 0.06f) {
    x.e = (1.0f - v) + (0.5f * v) * v;
    x.r = recip_in_range(x.e);
  } else {
    const float tblind = quotient_in_range(v, T.sw_bpade + v);
    const int it = clampi(static_cast<int>(static_cast<float>(T.sw_ntbl) * tblind + 0.5f), 0, T.sw_ntbl);
    const float2 p = __ldg(T.sw_pade + it);
    x.e = p.x;
    x.r = p.y;
  }
  return x;
}

__device__ __forceinline__ bool safe_size(float a) { return fabsf(a) >= kSafeLow && fabsf(a) <= kSafeHigh; }

// reftra's general and conservative branches.  kIso: zg = 0 (no cloud), where
// g3 = g4 = 1/2 and za1, za2 are one value.  zw in (0, 1], zto1 in
// [kSafeLow, kSafeHigh].
template <bool kIso>
__device__ __forceinline__ RT4 reftra_safe(const Tables &T, float zg, float mu, float zto1, float zw, float zto1_mu,
                                           SwExp ex2, bool conservative, bool &ok) {
  RT4 r;
  const float eps = 1.0e-8f;
  const float zg3 = 3.0f * zg;
  const float g1 = kIso ? (8.0f - zw * 5.0f) * 0.25f : (8.0f - zw * (5.0f + zg3)) * 0.25f;
  const float g2 = kIso ? 3.0f * zw * 0.25f : 3.0f * (zw * (1.0f - zg)) * 0.25f;
  const float g3 = kIso ? 0.5f : (2.0f - zg3 * mu) * 0.25f;
  const float g4 = kIso ? 0.5f : 1.0f - g3;
  if (zto1_mu > 500.0f) ex2 = exp_pair(T, 500.0f);
  if (conservative) {
    const float za = g1 * mu;
    const float za1 = za - g3;
    const float zgt = g1 * zto1;
    const float num = zgt - za1 * (1.0f - ex2.e), den = 1.0f + zgt, y = recip_in_range(den);
    ok = ok && safe_size(num);
    r.ref = quotient_by(num, den, y);
    r.tra = 1.0f - r.ref;
    r.refd = quotient_by(zgt, den, y);
    r.trad = 1.0f - r.refd;
    if (ex2.e == 1.0f) { r.ref = 0.0f; r.tra = 1.0f; r.refd = 0.0f; r.trad = 1.0f; }
    return r;
  }
  const float za1 = g1 * g4 + g2 * g3;
  const float za2 = kIso ? za1 : g1 * g3 + g2 * g4;
  const float rad = g1 * g1 - g2 * g2;
  const float zrk = sqrtf(rad > 0.0f ? rad : 0.0f);
  const float zrp = zrk * mu;
  const float zrp1 = 1.0f + zrp, zrm1 = 1.0f - zrp, zrk2 = 2.0f * zrk;
  const float zrpp = 1.0f - zrp * zrp;
  const float zrkg = zrk + g1;
  const float s3 = zrk * g3, s4 = zrk * g4;
  const float zr1 = zrm1 * (za2 + s3);
  const float zr2 = zrp1 * (za2 - s3);
  const float zr3 = zrk2 * (g3 - za2 * mu);
  const float zr4 = zrpp * zrkg;
  const float zr5 = zrpp * (zrk - g1);
  const float zt1 = zrp1 * (za1 + s4);
  const float zt2 = zrm1 * (za1 - s4);
  const float zt3 = zrk2 * (g4 + za1 * mu);
  const float zbeta = quotient_in_range(g1 - zrk, zrkg);
  float ze1 = zrk * zto1;
  if (ze1 > 500.0f) ze1 = 500.0f;
  const SwExp ex1 = exp_pair(T, ze1);
  const float zden = zr4 * ex1.r + zr5 * ex1.e;
  if ((zden >= -eps) && (zden <= eps)) {
    r.ref = eps;
    r.tra = ex2.e;
  } else {
    const float y = recip_in_range(zden);
    const float nr = zw * (zr1 * ex1.r - zr2 * ex1.e - zr3 * ex2.e);
    const float nt = ex2.e * zw * (zt1 * ex1.r - zt2 * ex1.e - zt3 * ex2.r);
    const float least = fabsf(zden) * 0x1p-95f;  // of a numerator, for a quotient in range
    ok = ok && fabsf(zden) <= 0x1p90f && fabsf(nr) <= 0x1p90f && fabsf(nt) <= 0x1p90f &&
         fabsf(nr) >= fmaxf(least, kSafeLow) && fabsf(nt) >= fmaxf(least, kSafeLow);
    r.ref = quotient_by(nr, zden, y);
    r.tra = ex2.e - quotient_by(nt, zden, y);
  }
  const float zemm = ex1.e * ex1.e;
  const float dd = (1.0f - zbeta * zemm) * zrkg;
  ok = ok && safe_size(dd);
  const float zdend = recip_in_range(dd);
  r.refd = g2 * (1.0f - zemm) * zdend;
  r.trad = zrk2 * ex1.e * zdend;
  return r;
}

// y_mu = recip_in_range(mu)
__device__ __forceinline__ SwOptics sw_clear_safe(const Tables &T, float tg, float tr, float mu, float y_mu, SwClear &c,
                                                  bool &ok) {
  SwOptics o;
  c.ztau = (tr + tg) + 0.0f;
  const float zom = quotient_in_range(tr, c.ztau);
  ok = tr >= kSafeLow && c.ztau <= kSafeHigh && zom >= 0x1p-30f && zom <= 1.0f && mu >= 0x1p-34f && mu <= 2.0f;
  // zg = 0: no delta scaling (sw:6923-6927 gives zf = 0), scaled = unscaled
  c.ztauc = c.ztau;
  c.zomcc = zom;
  c.zgcc = 0.0f;
  const float v = quotient_by(c.ztau, mu, y_mu);
  const SwExp ex2 = exp_pair(T, v);
  o.dbt = ex2.e;
  o.dbt_nd = ex2.e;
  o.rt = reftra_safe<true>(T, 0.0f, mu, c.ztau, zom, v, ex2, zom >= 0.9999995f, ok);
  return o;
}

__device__ __forceinline__ SwOptics sw_cloudy_safe(const Tables &T, const SwClear &c, float4 cld, float mu, float y_mu,
                                                   bool &ok) {
  SwOptics t;
  const float tcld = cld.x, wcld = cld.y, gcld = cld.z, taor = cld.w;
  t.dbt_nd = exp_pair(T, quotient_by(c.ztau + taor, mu, y_mu)).e;
  const float ztauo = c.ztauc + tcld;
  const float scat = c.ztauc * c.zomcc + tcld * wcld;
  const float scatg = tcld * wcld * gcld + 0.0f;  // the clear sky's share has zgcc = 0
  const float zg = quotient_in_range(scatg, scat);
  const float zw = quotient_in_range(scat, ztauo);
  // (scat is at most ztauo where zw is at most 1: with 2^30 the quotient zg is at least 2^-120)
  ok = ok && tcld >= 0.0f && taor >= 0.0f && taor <= kSafeHigh && ztauo <= 0x1p30f && scat >= kSafeLow &&
       scatg >= kSafeLow && zg <= 0.99f && zw >= 0x1p-30f && zw <= 1.0f;
  // whether zw / (1 - (1 - zw) (zg / (1 - zg))^2) reaches 0.9999995: far below
  // it by an approximate divisor, else by the reference's own quotients
  float sr_approx = __fdividef(zg, 1.0f - zg);
  const float den_approx = 1.0f - (1.0f - zw) * sr_approx * sr_approx;
  bool conservative = false;
  if (!(den_approx > 0.05f && zw < 0.99f * den_approx)) {
    const float sr = div_or_same(zg, 1.0f - zg);
    const float denom = 1.0f - (1.0f - zw) * sr * sr;
    conservative = (denom != 0.0f ? div_or_same(zw, denom) : 0.0f) >= 0.9999995f;
  }
  const float v = quotient_by(ztauo, mu, y_mu);
  const SwExp ex2 = exp_pair(T, v);
  t.dbt = ex2.e;
  t.rt = reftra_safe<false>(T, zg, mu, ztauo, zw, v, ex2, conservative, ok);
  return t;
}

// The *_any forms out of line, for the rare layers with operands out of range.
__device__ __noinline__ SwOptics sw_clear_slow(const Tables &T, float tg, float tr, float mu, SwClear &c) {
  return sw_clear_any<false>(T, tg, tr, mu, c);
}
__device__ __noinline__ SwOptics sw_cloudy_slow(const Tables &T, const SwClear &c, const SwOptics &oc, float4 cld,
                                                float mu) {
  return sw_cloudy_any<false>(T, c, oc, cld, mu);
}

// Solar source of band B (the per-band rules of sw:4430-4450): the source
// layer from the layers' jp (jp(l)), the spectral interpolation of that layer
// from its fields (field(f, l), where the band uses it), and the source of
// each g-point.
template <int B, class JpFn, class FieldFn>
__device__ __forceinline__ void sw_source(const Tables &T, const Col &C, JpFn jp, FieldFn field, float *sflux) {
  constexpr int ngc = kNgc[B];
  constexpr int bn = B + 16;
  const int n = C.nlay;
  const SwBand &K = T.sw[B];
  const int layreffr = K.layreffr;
  int ls = -1;
  bool found = false;
  // The searches read jp in batches of kJpBatch layers so that the record
  // loads overlap; each stops where its condition can no longer hold (below
  // laytrop for the lower-atmosphere bands, from laytrop up for 17 and 28).
  constexpr int kJpBatch = 8;
  if constexpr (bn == 18 || bn == 19 || bn == 21 || bn == 22 || bn == 24) {
    // first troposphere crossing of layreffr, one layer up, capped at laytrop-1
    const int lend = C.laytrop < n ? C.laytrop : n;
    for (int l0 = 0; l0 < lend && !found; l0 += kJpBatch) {
      int jb[kJpBatch + 1];
#pragma unroll
      for (int q = 0; q <= kJpBatch; ++q) jb[q] = l0 + q < n ? jp(l0 + q) : 0;
#pragma unroll
      for (int q = 0; q < kJpBatch; ++q) {
        const int l = l0 + q;
        if (l < lend && !found) {
          const int jl = jb[q];
          const int next = l + 1 < n ? jb[q + 1] : jl;
          if (jl < layreffr && next >= layreffr) {
            found = true;
            ls = (l + 1 < C.laytrop - 1) ? l + 1 : C.laytrop - 1;
          }
        }
      }
    }
    if (!found) ls = C.laytrop - 1;
  }
  if constexpr (bn == 17 || bn == 28) {
    const int lbeg = C.laytrop > 1 ? C.laytrop : 1;
    for (int l0 = lbeg; l0 < n && !found; l0 += kJpBatch) {
      int jb[kJpBatch + 1];  // jp(l0 - 1 + q)
#pragma unroll
      for (int q = 0; q <= kJpBatch; ++q) jb[q] = l0 - 1 + q < n ? jp(l0 - 1 + q) : 0;
#pragma unroll
      for (int q = 0; q < kJpBatch; ++q) {
        const int l = l0 + q;
        if (l < n && !found && jb[q] < layreffr && jb[q + 1] >= layreffr) {
          found = true;
          ls = l;
        }
      }
    }
    if (!found) ls = n - 1;
  }
  bool have = false;
  if constexpr (bn == 17 || bn == 28) have = C.laytrop < n;
  if constexpr (bn == 18 || bn == 19 || bn == 21 || bn == 22 || bn == 24) have = C.laytrop > 0;
  float src_fs = 0.0f;
  int src_js0 = 0;
  if (have && ls >= 0) {
    constexpr bool low = !(bn == 17 || bn == 28);
    const SwSpec sp = sw_band_species<B, low>(K, [&](SwField f) { return field(f, ls); });
    src_js0 = sp.js0;
    src_fs = sp.fs;
  }
#pragma unroll
  for (int g = 0; g < ngc; ++g) {
    float sz = 0.0f;
    if constexpr (bn == 16 || bn == 29) sz = C.laytrop < n ? ld(K.sfluxref + g) : 0.0f;
    if constexpr (bn == 20 || bn == 23 || bn == 25 || bn == 26) sz = C.laytrop > 0 ? ld(K.sfluxref + g) : 0.0f;
    if constexpr (bn == 27) sz = C.laytrop < n ? K.scalekur * ld(K.sfluxref + g) : 0.0f;
    if constexpr (bn == 17 || bn == 28 || bn == 18 || bn == 19 || bn == 21 || bn == 22 || bn == 24) {
      if (have) {
        const int c = K.sflux_cols;
        const float s0 = ld(K.sfluxref + g * c + src_js0), s1 = ld(K.sfluxref + g * c + src_js0 + 1);
        sz = s0 + src_fs * (s1 - s0);
      }
    }
    sflux[g] = sz;
  }
}

// Day-column compaction: a warp ballots its columns' coszr > 0 and appends the
// day columns to a.daylist (one atomic per warp, ascending within a warp); the
// night columns' outputs (sw:2536-2557 masks them to zero) and every column's
// coszr / *cln outputs are written here.
__global__ void __launch_bounds__(256) sw_daylist_kernel(SwArgs a) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool inside = col < a.ncol && !dead_column(a.live, col);
  const float coszen = inside ? ld(a.in.coszr + col) : 0.0f;
  const bool day = coszen > 0.0f;
  const unsigned ballot = __ballot_sync(0xffffffffu, inside && day);
  int base = 0;
  if (lane == 0 && ballot) base = atomicAdd(a.nday, __popc(ballot));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (!inside) return;
  a.coszr_out[col] = coszen;
#pragma unroll
  for (int q = 0; q < 4; ++q) a.zero2[q][col] = 0.0f;
  if (day) {
    a.daylist[base + __popc(ballot & ((1u << lane) - 1u))] = col;
    return;
  }
  const int i = col / a.ny, j = col - i * a.ny;
  const size_t rbase = static_cast<size_t>(i) * a.nk * a.ny + j;
  for (int k = 0; k < a.nk; ++k) {
    a.rthraten[rbase + static_cast<size_t>(k) * a.ny] = 0.0f;
    a.rthratenc[rbase + static_cast<size_t>(k) * a.ny] = 0.0f;
  }
  a.upt[col] = 0.0f; a.uptc[col] = 0.0f; a.dnt[col] = 0.0f; a.dntc[col] = 0.0f;
  a.upb[col] = 0.0f; a.upbc[col] = 0.0f; a.dnb[col] = 0.0f; a.dnbc[col] = 0.0f;
  a.swcf[col] = 0.0f; a.gsw[col] = 0.0f; a.swddir[col] = 0.0f; a.swddni[col] = 0.0f;
  a.swddif[col] = 0.0f; a.swdownc[col] = 0.0f; a.swddnic[col] = 0.0f; a.swddirc[col] = 0.0f;
}

__device__ __forceinline__ float sw_pavel(const SwArgs &a, const Col &C, int l) {
  return l < C.nk ? pa_to_hpa(in3(a.in.p3d, C, l)) : 0.5f * pa_to_hpa(in3w(a.in.p8w, C, C.nk));
}

// Column set-up of a day column without laytrop (buffer ozone; sw:2491-2508).
__device__ __forceinline__ void sw_setup_head(const Tables &T, const SwArgs &a, int col, Col &C) {
  C.i = col / a.ny;
  C.j = col - C.i * a.ny;
  C.nk = a.nk;
  C.ny = a.ny;
  C.nlay = a.nk + 1;
  const int nk = C.nk, n = C.nlay;
  const float coszen = ld(a.in.coszr + col);
  C.coszen = coszen;
  C.mu = fmaxf(coszen, 1.0e-10f);
  C.albedo = ld(a.in.albedo + col);
  C.co2 = a.co2; C.n2o = a.n2o; C.ch4 = a.ch4;
  C.inflg = a.inflg; C.iceflg = a.iceflg;
  C.has_reqc = a.has_reqc; C.has_reqi = a.has_reqi; C.has_reqs = a.has_reqs; C.icloud = a.icloud;
  C.adjflux = 1.0f * (a.solcon / 1.36822e3f);
  // ozone in the extra top layer (sw:2491-2508)
  {
    const float amdo = 0.603461f;
    const float pnk1 = pa_to_hpa(in3w(a.in.p8w, C, nk - 1)), pnk = pa_to_hpa(in3w(a.in.p8w, C, nk));
    const float mmr_k = o3data_layer(T, pnk1, pnk);
    const float mmr_t = o3data_layer(T, pnk, 1.0e-5f);
    float top = (in3(a.in.o3, C, nk - 1) - mmr_k * amdo) + mmr_t * amdo;
    if (top <= 0.0f) top = mmr_t * amdo;
    C.o3top = top;
  }
  (void)n;
}

// Heating rate and theta tendency of layer l of a day column from its level
// sums accs (six arrays of stride `stride`, top-down; sw:2285-2301).
__device__ __forceinline__ void sw_layer_output(const SwArgs &a, const Col &C, int l, const float *accs,
                                                int stride) {
  const int nk = C.nk, n = C.nlay;
  const size_t rbase = static_cast<size_t>(C.i) * nk * C.ny + C.j;
  const float *fu = accs, *fd = accs + stride, *cu = accs + 2 * stride, *cd = accs + 3 * stride;
  const float heatfac = (9.8066f * 8.6400e4f) / (1004.5f * 1.0e2f);
  // bottom-up level l is top-down index n - l
  const float n1 = fd[n - (l + 1)] - fu[n - (l + 1)], n0 = fd[n - l] - fu[n - l];
  const float c1 = cd[n - (l + 1)] - cu[n - (l + 1)], c0 = cd[n - l] - cu[n - l];
  const float plev0 = pa_to_hpa(in3w(a.in.p8w, C, l));
  const float plev1 = pa_to_hpa(in3w(a.in.p8w, C, l + 1));
  const float zdpgcp = heatfac / (plev0 - plev1);
  float hr = (n1 - n0) * zdpgcp;
  float hrc = (c1 - c0) * zdpgcp;
  if (l >= a.fp64_from) {  // FP64 mode
    hr = heating64(heatfac, fu[n - l], fd[n - l], fu[n - (l + 1)], fd[n - (l + 1)], plev0, plev1);
    hrc = heating64(heatfac, cu[n - l], cd[n - l], cu[n - (l + 1)], cd[n - (l + 1)], plev0, plev1);
  }
  const float pi3d = ld(a.in.pi3d + rbase + static_cast<size_t>(l) * C.ny);
  a.rthraten[rbase + static_cast<size_t>(l) * C.ny] = (hr / 86400.0f) / pi3d;
  a.rthratenc[rbase + static_cast<size_t>(l) * C.ny] = (hrc / 86400.0f) / pi3d;
}

// 2-D outputs of a day column from its level sums (sw:2536-2719).
__device__ __forceinline__ void sw_column_outputs(const SwArgs &a, const Col &C, int col, const float *accs,
                                                  int stride) {
  const int n = C.nlay;
  const float coszen = C.coszen;
  const float *fu = accs, *fd = accs + stride, *cu = accs + 2 * stride, *cd = accs + 3 * stride;
  const float *fdir = accs + 4 * stride, *cdir = accs + 5 * stride;
  a.upt[col] = fu[0];
  a.uptc[col] = cu[0];
  a.dnt[col] = fd[0];
  a.dntc[col] = cd[0];
  a.upb[col] = fu[n];
  a.upbc[col] = cu[n];
  a.dnb[col] = fd[n];
  a.dnbc[col] = cd[n];
  a.swcf[col] = (fd[0] - fu[0]) - (cd[0] - cu[0]);
  a.gsw[col] = fd[n] - fu[n];
  a.swddir[col] = fdir[n];
  a.swddni[col] = fdir[n] / coszen;
  a.swddif[col] = fd[n] - fdir[n];
  a.swdownc[col] = cd[n];
  a.swddirc[col] = cdir[n];
  a.swddnic[col] = cdir[n] / coszen;
}

// ---------------------------------------------------------------------------
// Sweep schedule, every domain size.  Day-list slots are processed in chunks;
// per chunk:
//   sw_colprep_kernel  warp = day slot: the column set-up once (laytrop by a
//                      warp vote over the layers);
//   sw_layer_kernel    thread = (day slot, layer): the layer set-up into
//                      layer fields;
//   sw_optics_kernel   thread = (day slot, layer), block = one band: the
//                      band's gas and Rayleigh depths of every g-point and its
//                      cloud optics, into the layer record; some blocks take
//                      the bands' solar sources, thread = (day slot, band);
//   sw_sweep_kernel    block = kSweepCols day slots x 112 g-points, thread =
//                      one g-point: the top-down pass (delta-Eddington layers,
//                      direct beam, downward adding) and the bottom-up pass
//                      (upward adding, level fluxes) of spcvmc, the
//                      per-level spectral sums in g-point order in shared
//                      memory, then heating and the 2-D outputs.
// Records: per chunk slot a column record, then nlay layer records of kSwRec
// floats (1,248 bytes per layer, 64 KB per day column at nk = 50), then the
// kSwLayerFields layer fields (124 bytes per layer).  Each band's g-points
// start on a 16-byte boundary (kPadOfs) so the optics kernel writes whole
// float4s: taug at [0, 128), taur at [128, 256), the cloud optics (tau, ssa,
// asm, unscaled tau) of band B at 256 + 4 B.
constexpr int kSwRec = 312;
constexpr int kSwRecTaur = 128, kSwRecCloud = 256;
constexpr int kPadOfs[kSwBands] = {0, 8, 20, 28, 36, 48, 60, 64, 76, 84, 92, 100, 108, 116};
static_assert(kSwRecCloud + 4 * kSwBands == kSwRec && kSwRec % 8 == 0, "record layout");
static_assert(kPadOfs[kSwBands - 1] + sw_pad(kSwBands - 1) == kSwRecTaur, "padded g-points");
__constant__ int kPadOfsDev[kSwBands] = {0, 8, 20, 28, 36, 48, 60, 64, 76, 84, 92, 100, 108, 116};

struct SwColRec {
  Col C;
  float sflux[kSwGpts];
};
constexpr size_t kSwColRecFloats = (sizeof(SwColRec) + 15) / 16 * 4;

// chunk-relative slot u = t - a.chunk_first
__device__ __forceinline__ SwColRec *sw_colrecs(const SwArgs &a) { return reinterpret_cast<SwColRec *>(a.records); }
__device__ __forceinline__ float *sw_layrecs(const SwArgs &a) {
  return a.records + kSwColRecFloats * static_cast<size_t>(a.chunk_capacity);
}
// the layer fields of the chunk: field f of (layer l, slot u) at
// [(f * (nk + 1) + l) * chunk_capacity + u]
__device__ __forceinline__ float *sw_layfields(const SwArgs &a) {
  return sw_layrecs(a) + static_cast<size_t>(kSwRec) * (a.nk + 1) * a.chunk_capacity;
}

// Day slots of the launched chunk, and whether the small-chunk sweep takes them.
__device__ __forceinline__ int sw_chunk_slots(const SwArgs &a) {
  const int left = *a.nday - a.chunk_first;
  return left < a.chunk_count ? left : a.chunk_count;
}
__device__ __forceinline__ bool sw_small(const SwArgs &a, int slots) {
  return a.chunk_capacity <= kSmallColumns && slots <= kSwSmallColumns;
}

// A warp per day column; the lanes take the layers of the laytrop count.
__global__ void __launch_bounds__(128) sw_colprep_kernel(Tables T, SwArgs a) {
  const int lane = threadIdx.x & 31;
  const int u = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int t = a.chunk_first + u;
  if (u >= a.chunk_count || t >= *a.nday) return;  // whole warps
  Col C;
  sw_setup_head(T, a, a.daylist[t], C);
  int count = 0;
  for (int l = lane; l < C.nlay; l += 32) count += glibc_logf(T, sw_pavel(a, C, l)) > 4.56f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
  C.laytrop = count;
  if (lane == 0) sw_colrecs(a)[u].C = C;
}

// 16-byte pieces of a warp's stage: gas depths, then Rayleigh depths, of 32 rows of up to 3
constexpr int kSwStage = 2 * 32 * 3;

// Band B of the layer records of a warp's 32 (layer, slot) pairs: gas and
// Rayleigh depths of every g-point, and the band's cloud optics (cldprmc_sw
// only where the layer holds cloud water; a layer without any has the
// reference's inactive values 0, 1, 0, 0).  The layer fields are read inside
// the band's own code, so that each band loads only those it uses, and the
// depths go through the warp's shared stage, so that neighbouring lanes write
// neighbouring 16-byte pieces.  record: the lane's layer record, or -1.
template <int B>
__device__ __forceinline__ void sw_band_record(const Tables &T, const SwArgs &a, const float *fld, size_t fstride,
                                               int record, float4 *stage) {
  constexpr int Q = sw_pad(B) / 4, kRow = Q | 1;
  const int lane = threadIdx.x & 31;
  if (record >= 0) {
    auto field = [&](SwField f) { return fld[static_cast<size_t>(f) * fstride]; };
    SLayer L;
#define RRTMG_SW_GET(name) L.name = field(kSwField_##name);
#define RRTMG_SW_GETI(name) L.name = __float_as_int(field(kSwField_##name));
    RRTMG_SW_LAYER_FLOATS(RRTMG_SW_GET)
    RRTMG_SW_LAYER_INTS(RRTMG_SW_GETI)
#undef RRTMG_SW_GET
#undef RRTMG_SW_GETI
    float4 *row = stage + lane * kRow;
    sw_quads<B>(T, L, field, [&](int q, float4 tg, float4 tr) {
      row[q] = tg;
      row[q + kSwStage / 2] = tr;
    });
    float4 cq = make_float4(0.0f, 1.0f, 0.0f, 0.0f);
    if (__float_as_int(field(kSwField_cloud_water)) != 0) {
      const CloudOpt o = sw_cloud(T, L, B, a.iceflg);
      cq = make_float4(o.tau, o.ssa, o.asm_, o.taor);
    }
    reinterpret_cast<float4 *>(sw_layrecs(a) + static_cast<size_t>(record) * kSwRec)[kSwRecCloud / 4 + B] = cq;
  }
  __syncwarp();
  float *recs = sw_layrecs(a) + kPadOfs[B];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int e = i * 32 + lane, r = e / Q, q = e - r * Q;
    const int rec = __shfl_sync(0xffffffffu, record, r);
    if (rec >= 0) {
      float4 *out = reinterpret_cast<float4 *>(recs + static_cast<size_t>(rec) * kSwRec) + q;
      out[0] = stage[r * kRow + q];
      out[kSwRecTaur / 4] = stage[r * kRow + q + kSwStage / 2];
    }
  }
}

// sw_layer_kernel: thread = (layer, chunk slot), slots fastest: the layer
// set-up (make_layer) and cldprmc_sw's activity test once, stored as layer
// fields.
__global__ void __launch_bounds__(128) sw_layer_kernel(Tables T, SwArgs a) {
  const int n = a.nk + 1;
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int l = static_cast<int>(idx / a.chunk_count);
  const int u = static_cast<int>(idx - static_cast<long long>(l) * a.chunk_count);
  if (l >= n || a.chunk_first + u >= *a.nday) return;
  const Col C = sw_colrecs(a)[u].C;
  const SLayer L = make_layer(T, a, C, l);
  // the activity test of cldprmc_sw (sw:1409-1440), the same for every band
  const float cswp = C.iceflg == 5 ? L.cswp : 0.0f;
  const bool cloud_water = a.icld != 0 && ((L.ciwp + L.clwp) + cswp) >= 1.0e-20f;
  float *fld = sw_layfields(a) + static_cast<size_t>(l) * a.chunk_capacity + u;
  const size_t fstride = static_cast<size_t>(n) * a.chunk_capacity;
  int f = 0;
#define RRTMG_SW_PUT(name) fld[static_cast<size_t>(f++) * fstride] = L.name;
#define RRTMG_SW_PUTI(name) fld[static_cast<size_t>(f++) * fstride] = __int_as_float(L.name);
  RRTMG_SW_LAYER_FLOATS(RRTMG_SW_PUT)
  RRTMG_SW_LAYER_INTS(RRTMG_SW_PUTI)
#undef RRTMG_SW_PUT
#undef RRTMG_SW_PUTI
  fld[static_cast<size_t>(f) * fstride] = __int_as_float(cloud_water ? 1 : 0);
}

#define RRTMG_SW_BAND_SWITCH(band, CALL) \
  switch (band) {                        \
    case 0: CALL(0); break;              \
    case 1: CALL(1); break;              \
    case 2: CALL(2); break;              \
    case 3: CALL(3); break;              \
    case 4: CALL(4); break;              \
    case 5: CALL(5); break;              \
    case 6: CALL(6); break;              \
    case 7: CALL(7); break;              \
    case 8: CALL(8); break;              \
    case 9: CALL(9); break;              \
    case 10: CALL(10); break;            \
    case 11: CALL(11); break;            \
    case 12: CALL(12); break;            \
    default: CALL(13); break;            \
  }

// sw_optics_kernel: one band per block.  Blocks of (layer, chunk slot) pairs
// are taken kSwOpticsGroup at a time through all 14 bands, so that a group's
// layer fields are read from L2 by the later bands and its records, which the
// bands fill piece by piece, leave L2 whole; each block runs one band's code
// only.  SW optics of 425 x 425 x 50 (day list, set-up and source included):
// 6.85 ms with groups of 128 and 5 blocks per SM (96 registers), 7.0 ms at 6
// blocks (80 registers), 9.4 ms with groups of 512; 14.2 ms with the g-points
// unrolled over unpadded tables and stores of a lane per record.
constexpr int kSwOpticsGroup = 128;
constexpr int kSwOpticsMinBlocks = 5;
constexpr int kSwSweepMinBlocks = 4;
__global__ void __launch_bounds__(128, kSwOpticsMinBlocks) sw_optics_kernel(Tables T, SwArgs a, int source_blocks) {
  // The first blocks take the solar sources, thread = (slot, band): they need
  // the layer fields only, and a launch of their own took 17 to 21 us however
  // few columns there were (a warp per slot and band instead of a thread: 6 us
  // less there, but 0.26 ms more for 300 x 300 columns).
  if (static_cast<int>(blockIdx.x) < source_blocks) {
    const int n = a.nk + 1, band = blockIdx.x % kSwBands;
    const int u = static_cast<int>(blockIdx.x / kSwBands) * blockDim.x + threadIdx.x;
    if (u >= sw_chunk_slots(a)) return;
    SwColRec &R = sw_colrecs(a)[u];
    const float *fld = sw_layfields(a) + u;
    auto field = [&](int f, int l) { return fld[(static_cast<size_t>(f) * n + l) * a.chunk_capacity]; };
    auto jp = [&](int l) { return __float_as_int(field(kSwField_jp, l)); };
#define RRTMG_SW_SRC(B)                                 \
  {                                                     \
    constexpr int gofs_ = kGofs[B];                     \
    sw_source<B>(T, R.C, jp, field, R.sflux + gofs_);   \
  }
    RRTMG_SW_BAND_SWITCH(band, RRTMG_SW_SRC)
#undef RRTMG_SW_SRC
    return;
  }
  __shared__ float4 stages[4][kSwStage];
  float4 *stage = stages[threadIdx.x >> 5];
  const int n = a.nk + 1, slots = sw_chunk_slots(a);
  const int nblk = static_cast<int>((static_cast<long long>(slots > 0 ? slots : 0) * n + 127) / 128);
  const size_t fstride = static_cast<size_t>(n) * a.chunk_capacity;
  const int step = static_cast<int>(gridDim.x) - source_blocks;
  for (long long vb = static_cast<int>(blockIdx.x) - source_blocks; vb < static_cast<long long>(nblk) * kSwBands;
       vb += step) {
    const int group = static_cast<int>(vb / (kSwOpticsGroup * kSwBands));
    const int g0 = group * kSwOpticsGroup;
    const int gsize = nblk - g0 < kSwOpticsGroup ? nblk - g0 : kSwOpticsGroup;
    const int within = static_cast<int>(vb - static_cast<long long>(group) * (kSwOpticsGroup * kSwBands));
    const int band = within / gsize;
    const int blk = g0 + (within - band * gsize);
    const long long idx = static_cast<long long>(blk) * blockDim.x + threadIdx.x;
    const int l = static_cast<int>(idx / slots);
    const int u = static_cast<int>(idx - static_cast<long long>(l) * slots);
    const bool live = l < n;
    if (!__any_sync(0xffffffffu, live)) continue;  // whole warps
    const float *fld = sw_layfields(a) + static_cast<size_t>(l) * a.chunk_capacity + u;
    const int record = live ? u * n + l : -1;
#define RRTMG_SW_OPT(B) sw_band_record<B>(T, a, fld, fstride, record, stage)
    RRTMG_SW_BAND_SWITCH(band, RRTMG_SW_OPT)
#undef RRTMG_SW_OPT
    __syncwarp();  // the stage is read out
  }
}

#undef RRTMG_SW_BAND_SWITCH

__constant__ int kSwGofsDev[kSwBands] = {0, 6, 18, 26, 34, 44, 54, 56, 66, 74, 80, 86, 94, 100};

constexpr int kSweepCols = 2;                         // day columns per block
constexpr int kSweepThreads = kSweepCols * kSwGpts;   // 224: one thread per g-point
constexpr int kRingRows = 32;                         // level terms per ordered-sum round: (level, type, column)
constexpr int kRingStride = kSwGpts + 4;              // floats per row: 29 16-byte chunks, odd, so that the lanes
                                                      // of a 16-byte read of 32 rows meet no bank conflict
static_assert(kRingStride % 4 == 0 && (kRingStride / 4) % 2 == 1, "ring rows");

// Shared memory of a sweep block: two buffers of level terms awaiting their
// g-ordered sums (one is summed while the other fills), and the sums.
struct SweepShared {
  float ring[2][kRingRows][kRingStride];
  float sums[kSweepCols][6][kMaxLev];  // type: fu, fd, cu, cd, fdir, cdir; level top-down
  uint32_t slotbits[2][kMaxLay / 32][kSweepThreads];  // per thread: cloudy slots, total = clear slots
};

// One level of one adding path, as the bottom-up pass reads it back: the
// layer's reflectances/transmittances and direct-beam transmittance, and the
// level's cumulative direct beam and downward recurrence (vrtqdr, sw:3655-3702).
struct SwLevel {
  float4 rt;   // ref, refd, tra, trad
  float4 dn;   // dbt, tdbt, tdn, rdnd
};

// Ordered sums of one full (or last) ring buffer: row (j, q, c) = level j of
// the round, term type q, column c holds the 112 terms of one level sum, and
// one lane adds them in g-point order, starting from zero as the reference's
// ordered sums do (sw:153-177).  One warp per round does it, the block's warps
// in turn, while the others fill the other buffer: the barrier here says that
// this buffer is full and that the other one's sums (of the previous round)
// are done, so a round costs one barrier.  Before: two barriers around a sum
// by 32 or 64 threads, whose rows lay 112 floats apart, a 16-way bank conflict;
// sweep of a 425 x 425 x 50 call 26.6 -> 25.9 ms, of a 64 x 64 x 44 call 0.62 ->
// 0.60 ms.
template <int NTYPES>
__device__ __forceinline__ void sweep_flush(SweepShared &S, int round, int count, int type0, int level0, int dir) {
  __syncthreads();
  if (static_cast<int>(threadIdx.x >> 5) != round % (kSweepThreads / 32)) return;
  const int row = threadIdx.x & 31;
  const int c = row % kSweepCols, q = row / kSweepCols % NTYPES, j = row / (kSweepCols * NTYPES);
  if (j >= count) return;
  const float4 *v = reinterpret_cast<const float4 *>(S.ring[round & 1][row]);
  float acc = 0.0f;
#pragma unroll 7
  for (int i = 0; i < kSwGpts / 4; ++i) {
    const float4 x = v[i];
    acc = acc + x.x;
    acc = acc + x.y;
    acc = acc + x.z;
    acc = acc + x.w;
  }
  S.sums[c][type0 + q][level0 + dir * j] = acc;
}

// A layer's optics: the checked form, or the general one where that says so
// and in the FP64 mode.
template <bool kFp64>
__device__ __forceinline__ SwOptics sw_clear(const Tables &T, float tg, float tr, float mu, float y_mu, SwClear &c) {
  if constexpr (kFp64) {
    return sw_clear_any<true>(T, tg, tr, mu, c);
  } else {
    bool ok;
    SwOptics o = sw_clear_safe(T, tg, tr, mu, y_mu, c, ok);
    c.checked = ok;
    if (!ok) o = sw_clear_slow(T, tg, tr, mu, c);
    return o;
  }
}

template <bool kFp64>
__device__ __forceinline__ SwOptics sw_cloudy(const Tables &T, const SwClear &c, const SwOptics &oc, float4 cld,
                                              float mu, float y_mu) {
  if constexpr (kFp64) {
    return sw_cloudy_any<true>(T, c, oc, cld, mu);
  } else {
    bool ok = c.checked;  // mu and the clear sky's operands
    SwOptics o = sw_cloudy_safe(T, c, cld, mu, y_mu, ok);
    if (!ok) o = sw_cloudy_slow(T, c, oc, cld, mu);
    return o;
  }
}

// Surface albedos of a g-point's band, direct (albp) and diffuse (albd), from
// the Noah-MP fields where these are given, for columns with xland < 1.5
// (sw:2519-2530): visible in bands 25-28, near infrared in 16-24 and 29
// (sw:2120-2127).
__device__ __forceinline__ void sw_albedos(const SwArgs &a, int col, int band, float &albp, float &albd) {
  if (!a.in.alswvisdir || !(ld(a.in.xland + col) < 1.5f)) return;
  const bool vis = band >= 9 && band <= 12;
  albp = ld((vis ? a.in.alswvisdir : a.in.alswnirdir) + col);
  albd = ld((vis ? a.in.alswvisdif : a.in.alswnirdif) + col);
}

// 1 / d of the adding method's denominators 1 - r r', in (0, 1] but for
// roundings and meaningless inputs.
__device__ __forceinline__ float sw_recip(float d) { return safe_size(d) ? recip_in_range(d) : 1.0f / d; }

// Upward recurrence of vrtqdr (sw:3655-3680) across the layer of slot s.
__device__ __forceinline__ void sw_up(const SwLevel &s, float &rup, float &rupd) {
  const float z = sw_recip(1.0f - rupd * s.rt.y);
  const float nrup = s.rt.x + s.rt.w * ((s.rt.z - s.dn.x) * rupd + s.dn.x * rup) * z;
  rupd = s.rt.y + s.rt.w * s.rt.w * rupd * z;
  rup = nrup;
}

// Level fluxes (sw:3703-3720); tdbt = dn.y, tdn = dn.z, rdnd = dn.w.
__device__ __forceinline__ void sw_fluxes(const SwLevel &s, float rup, float rupd, float &fu, float &fd) {
  const float z = sw_recip(1.0f - s.dn.w * rupd);
  fu = (s.dn.y * rup + (s.dn.z - s.dn.y) * rupd) * z;
  fd = s.dn.y + (s.dn.z - s.dn.y + s.dn.y * rup * s.dn.w) * z;
}

// Downward recurrence of vrtqdr (sw:3681-3702): the path's values at level
// r + 1 from those at level r and layer r's optics.
struct SwCarry {
  float tdbt, tdn, rdnd;
};

__device__ __forceinline__ SwCarry sw_down(const SwCarry &c, const SwOptics &o, bool top) {
  SwCarry n;
  n.tdbt = c.tdbt * o.dbt;
  if (top) {
    n.tdn = o.rt.tra;
    n.rdnd = o.rt.refd;
  } else {
    const float zreflect = sw_recip(1.0f - o.rt.refd * c.rdnd);
    n.tdn = c.tdbt * o.rt.tra + o.rt.trad * ((c.tdn - c.tdbt) + c.tdbt * o.rt.ref * c.rdnd) * zreflect;
    n.rdnd = o.rt.refd + o.rt.trad * o.rt.trad * c.rdnd * zreflect;
  }
  return n;
}

// Block = kSweepCols consecutive slots of the chunk; thread = (slot, g-point).
// A slot past the day count repeats the block's first slot so that every
// thread takes the same barriers; its results are not written.
//
// Work per g-point layer follows spcvmc (sw:6887-7041) statement by statement;
// operations are shared or skipped where the result is known bit for bit: the
// quotient tau / mu and its Pade lookup, computed once for the direct beam and
// reftra's exponent; divisions by a divisor that is exactly 1; in a g-point
// layer without cloud, the cloudy reflectance/transmittance, whose weight is
// zero; and above a g-point's highest cloud the whole total-sky path, which
// equals the clear-sky one.  Outside the FP64 mode the divisions themselves
// are those of rrtmg_divide.cuh.
// Bound by instruction issue, then by the stack's traffic.  Sweep of a
// 425 x 425 x 50 call: 25.7 ms with IEEE divisions throughout and the total-sky
// path followed from the top; 21.8 ms now (80 registers at 3 blocks per SM:
// 24.9).  The tables are a __grid_constant__: the out-of-line forms take their
// address, and a per-thread copy of them cost 14 ms.
template <bool kFp64>
__global__ void __launch_bounds__(kSweepThreads, kSwSweepMinBlocks) sw_sweep_kernel(const __grid_constant__ Tables T,
                                                                                        const SwArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepShared &S = *reinterpret_cast<SweepShared *>(smem_raw);
  const int nday = *a.nday;
  const int u0 = blockIdx.x * kSweepCols;
  if (u0 >= a.chunk_count || a.chunk_first + u0 >= nday || sw_small(a, sw_chunk_slots(a))) return;  // whole block
  const int cslot = threadIdx.x / kSwGpts;
  const int G = threadIdx.x - cslot * kSwGpts;
  const int u_own = u0 + cslot;
  const bool live = u_own < a.chunk_count && a.chunk_first + u_own < nday;
  const int u = live ? u_own : u0;
  const int col = a.daylist[a.chunk_first + u];
  const SwColRec &R = sw_colrecs(a)[u];
  const Col C = R.C;
  const float sflux_g = R.sflux[G];
  const int n = C.nlay;
  const float mu = C.mu;
  const float y_mu = recip_in_range(mu);
  const int clear_only = a.icld == 0;
  int band = kSwBands - 1;
  while (G < kSwGofsDev[band]) --band;
  const int P = kPadOfsDev[band] + (G - kSwGofsDev[band]);  // record position of the g-point
  // the block's layer records, addressed from one base by 32-bit byte offsets
  const char *const base =
      reinterpret_cast<const char *>(sw_layrecs(a) + static_cast<size_t>(u0) * n * kSwRec);
  constexpr uint32_t kStep = kSwRec * sizeof(float);
  const uint32_t column = static_cast<uint32_t>((u - u0) * n) * kStep;
  const uint32_t off_tau = column + 4u * P, off_cld = column + 4u * (kSwRecCloud + 4 * band);
  const uint32_t *maskbase = a.mask + col + static_cast<size_t>(G >> 5) * a.ncol;
  const size_t mstride = static_cast<size_t>(kSwMaskWords) * a.ncol;
  const uint32_t bit = 1u << (G & 31);

  // per-thread stack of the top-down pass, read back bottom-up
  SwLevel stc[kMaxLev], stt[kMaxLev];
  // per stack slot r, bit r & 31 of word r >> 5 (gathered in registers, 32
  // slots at a time, then kept in shared memory): the g-point layer is cloudy
  // (its total-sky reftra results are stored), and the slot's total-sky values
  // are the clear-sky ones (no cloud in this g-point so far: no total-sky slot
  // is stored; the bottom-up pass reuses the clear-sky slot)
  uint32_t cloudy_bits = 0, same_word = 0;

  // ---- top-down pass: layer optics, direct beam, downward adding (sw:6887-7041)
  float tdbtc_nd = 1.0f, tdbt_nd = 1.0f;
  const float zincflx = ((C.adjflux * sflux_g) * mu) * 1.0f;
  // ring position of this thread's terms: row (level * types + type) * columns + column
  float *const ring0 = &S.ring[0][cslot][G];
  constexpr int kTypeStep = kSweepCols * kRingStride, kBufStep = kRingRows * kRingStride;
  constexpr int kDownLevels = kRingRows / (2 * kSweepCols), kUpLevels = kRingRows / (4 * kSweepCols);
  ring0[0] = tdbt_nd * zincflx;
  ring0[kTypeStep] = tdbtc_nd * zincflx;
  int filled = 1, level0 = 0, round = 0;
  // the downward recurrence's values at level r; the total-sky ones count from
  // the g-point's first cloud on (differ)
  SwCarry cc{1.0f, 1.0f, 0.0f}, ct = cc;
  bool differ = false;
  // layer values are loaded one layer ahead
  float nx_tg, nx_tr;
  float4 nx_cld;
  uint32_t nx_word;
  auto load = [&](int l) {
    const uint32_t step = static_cast<uint32_t>(l) * kStep;
    nx_tg = *reinterpret_cast<const float *>(base + off_tau + step);
    nx_tr = *reinterpret_cast<const float *>(base + off_tau + step + 4 * kSwRecTaur);
    nx_cld = *reinterpret_cast<const float4 *>(base + off_cld + step);
    nx_word = maskbase[static_cast<size_t>(l) * mstride];
  };
  load(n - 1);
  for (int r = 0; r < n; ++r) {
    const int l = n - 1 - r;
    const bool cldb = !clear_only && (nx_word & bit) != 0u;
    const float tr = nx_tr, tg = nx_tg;
    const float4 cld = nx_cld;
    if (l > 0) load(l - 1);
    SwClear c;
    const SwOptics oc = sw_clear<kFp64>(T, tg, tr, mu, y_mu, c);
    stc[r].rt = make_float4(oc.rt.ref, oc.rt.refd, oc.rt.tra, oc.rt.trad);
    stc[r].dn = make_float4(oc.dbt, cc.tdbt, cc.tdn, cc.rdnd);
    if (cldb && !differ) {
      differ = true;
      ct = cc;
      tdbt_nd = tdbtc_nd;
    }
    if (differ) {
      SwOptics ot;
      if (cldb) {
        ot = sw_cloudy<kFp64>(T, c, oc, cld, mu, y_mu);
        stt[r].rt = make_float4(ot.rt.ref, ot.rt.refd, ot.rt.tra, ot.rt.trad);
        cloudy_bits |= 1u << (r & 31);
      } else {
        ot = oc;  // the reference's mix clear * c + cloud * (0, 0, 1, 1) with clear = 1, cloud = 0
      }
      stt[r].dn = make_float4(ot.dbt, ct.tdbt, ct.tdn, ct.rdnd);
      tdbt_nd = tdbt_nd * ot.dbt_nd;
      ct = sw_down(ct, ot, r == 0);
    } else {
      same_word |= 1u << (r & 31);
    }
    tdbtc_nd = tdbtc_nd * oc.dbt_nd;
    cc = sw_down(cc, oc, r == 0);
    if ((r & 31) == 31 || r == n - 1) {
      S.slotbits[0][r >> 5][threadIdx.x] = cloudy_bits;
      S.slotbits[1][r >> 5][threadIdx.x] = same_word;
      cloudy_bits = 0;
      same_word = 0;
    }
    {
      float *q = ring0 + (round & 1) * kBufStep + filled * (2 * kTypeStep);
      q[0] = (differ ? tdbt_nd : tdbtc_nd) * zincflx;
      q[kTypeStep] = tdbtc_nd * zincflx;
    }
    if (++filled == kDownLevels || r == n - 1) {
      sweep_flush<2>(S, round, filled, 4, level0, 1);
      ++round;
      level0 += filled;
      filled = 0;
    }
  }
  if (!differ) ct = cc;

  // ---- bottom-up pass: upward adding and level fluxes (vrtqdr, sw:3655-3720)
  float albp = C.albedo, albd = C.albedo;
  sw_albedos(a, col, band, albp, albd);
  float rupc = albp, rupdc = albd;
  float rupt = albp, rupdt = albd;
  level0 = n;
  // surface level n: albedo reflection, no transmission; the recurrence's level-n values
  SwLevel c = {make_float4(albp, albd, 0.0f, 0.0f), make_float4(0.0f, cc.tdbt, cc.tdn, cc.rdnd)};
  SwLevel t = {make_float4(albp, albd, 0.0f, 0.0f), make_float4(0.0f, ct.tdbt, ct.tdn, ct.rdnd)};
  if (clear_only) t = c;
  // stack slot j (layer n - 1 - j) of both paths; a layer without cloud in
  // this g-point has the clear-sky layer's optics in both
  auto load_slot = [&](int j, SwLevel &lc, SwLevel &lt) {
    lc = stc[j];
    if (clear_only || ((S.slotbits[1][j >> 5][threadIdx.x] >> (j & 31)) & 1u) != 0u) {
      lt = lc;
      return;
    }
    lt.dn = stt[j].dn;
    lt.rt = ((S.slotbits[0][j >> 5][threadIdx.x] >> (j & 31)) & 1u) != 0u ? stt[j].rt : lc.rt;
  };
  for (int k = n; k >= 0; --k) {
    SwLevel nc = c, nt = t;
    if (k > 0) load_slot(k - 1, nc, nt);
    if (k < n) {
      sw_up(c, rupc, rupdc);
      if (!clear_only) sw_up(t, rupt, rupdt);
    }
    float fuc, fdc, fut, fdt;
    sw_fluxes(c, rupc, rupdc, fuc, fdc);
    if (!clear_only) {
      sw_fluxes(t, rupt, rupdt, fut, fdt);
    } else {
      fut = fuc;
      fdt = fdc;
    }
    {
      float *q = ring0 + (round & 1) * kBufStep + filled * (4 * kTypeStep);
      q[0] = fut * zincflx;
      q[kTypeStep] = fdt * zincflx;
      q[2 * kTypeStep] = fuc * zincflx;
      q[3 * kTypeStep] = fdc * zincflx;
    }
    if (++filled == kUpLevels || k == 0) {
      sweep_flush<4>(S, round, filled, 0, level0, -1);
      ++round;
      level0 -= filled;
      filled = 0;
    }
    c = nc;
    t = nt;
  }

  __syncthreads();  // the last round's sums

  // ---- outputs of the block's live columns (sw:2285-2301, 2536-2719)
  for (int q = threadIdx.x; q < kSweepCols * kMaxLay; q += kSweepThreads) {
    const int cs = q / kMaxLay, l = q - cs * kMaxLay;
    const int uq = u0 + cs;
    if (l >= a.nk || uq >= a.chunk_count || a.chunk_first + uq >= nday) continue;
    sw_layer_output(a, sw_colrecs(a)[uq].C, l, &S.sums[cs][0][0], kMaxLev);
  }
  if (G == 0 && live) sw_column_outputs(a, C, col, &S.sums[cslot][0][0], kMaxLev);
}

// ---------------------------------------------------------------------------
// The sweep of small chunks.  With few columns the kernel above is a serial
// chain: each level's optics, some 400 dependent operations, wait for the level
// before although only the adding recurrences depend on it.  Here the optics of
// all layers are evaluated first, a thread per (slot, layer, g-point), into
// optics records, and the sweep then runs the recurrences alone, its loads four
// levels ahead.  The operations are the same functions, so the results are the
// same bits.  Sweep of 11 day columns of 50 layers 132 -> 64 us, of 180 day
// columns 181 -> 95 us, of 360 194 -> 181 us; of 720 296 us against 214, as the
// optics records (274 KB per slot) then pass through memory: hence
// kSwSmallColumns.
// ---------------------------------------------------------------------------

// Optics record of a (slot, layer): clear-sky (ref, refd, tra, trad) and (dbt,
// dbt_nd) of every g-point, then the total sky's where the g-point is cloudy.
constexpr int kSwOptClearDbt = 4 * kSwGpts, kSwOptTotal = 6 * kSwGpts, kSwOptTotalDbt = 10 * kSwGpts;
constexpr int kSwOpt = 12 * kSwGpts;
static_assert(kSwOpt % 8 == 0 && kSwOptClearDbt % 4 == 0 && kSwOptTotal % 4 == 0, "optics records");

__host__ __device__ __forceinline__ size_t sw_base_floats(int nk, int chunk) {
  const size_t f = (kSwColRecFloats + static_cast<size_t>(kSwRec + kSwLayerFields) * (nk + 1)) * chunk;
  return (f + 7) / 8 * 8;
}
__device__ __forceinline__ float *sw_optrec(const SwArgs &a, int u, int l) {
  return a.records + sw_base_floats(a.nk, a.chunk_capacity) + (static_cast<size_t>(u) * (a.nk + 1) + l) * kSwOpt;
}

// One (slot, layer) per item, g-points over the threads; the grid is bounded and
// walks the items, as the day count is known on the device only.
template <bool kFp64>
__global__ void __launch_bounds__(kSwGpts) sw_small_optics_kernel(const __grid_constant__ Tables T, const SwArgs a) {
  const int G = threadIdx.x, n = a.nk + 1;
  int band = kSwBands - 1;
  while (G < kSwGofsDev[band]) --band;
  const int P = kPadOfsDev[band] + (G - kSwGofsDev[band]);
  const int slots = sw_chunk_slots(a);
  if (!sw_small(a, slots)) return;
  const long long items = static_cast<long long>(slots) * n;
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const int u = static_cast<int>(item / n), l = static_cast<int>(item - static_cast<long long>(u) * n);
    const int col = a.daylist[a.chunk_first + u];
    const float mu = sw_colrecs(a)[u].C.mu;
    const float *rec = sw_layrecs(a) + (static_cast<size_t>(u) * n + l) * kSwRec;
    const float tg = rec[P], tr = rec[kSwRecTaur + P];
    const float4 cld = *reinterpret_cast<const float4 *>(rec + kSwRecCloud + 4 * band);
    const uint32_t word = a.mask[(static_cast<size_t>(l) * kSwMaskWords + (G >> 5)) * a.ncol + col];
    float *out = sw_optrec(a, u, l);
    auto put = [&](int rt, int dbt, const SwOptics &o) {
      reinterpret_cast<float4 *>(out + rt)[G] = make_float4(o.rt.ref, o.rt.refd, o.rt.tra, o.rt.trad);
      reinterpret_cast<float2 *>(out + dbt)[G] = make_float2(o.dbt, o.dbt_nd);
    };
    SwClear c;
    const SwOptics oc = sw_clear<kFp64>(T, tg, tr, mu, recip_in_range(mu), c);
    put(0, kSwOptClearDbt, oc);
    if (a.icld != 0 && ((word >> (G & 31)) & 1u) != 0u)
      put(kSwOptTotal, kSwOptTotalDbt, sw_cloudy<kFp64>(T, c, oc, cld, mu, recip_in_range(mu)));
  }
}

constexpr int kAhead = 4;  // levels loaded ahead by the small sweep

__global__ void __launch_bounds__(kSweepThreads, 1) sw_small_sweep_kernel(const SwArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepShared &S = *reinterpret_cast<SweepShared *>(smem_raw);
  const int slots = sw_chunk_slots(a);
  const int u0 = blockIdx.x * kSweepCols;
  if (u0 >= slots || !sw_small(a, slots)) return;  // whole block
  const int cslot = threadIdx.x / kSwGpts;
  const int G = threadIdx.x - cslot * kSwGpts;
  const bool live = u0 + cslot < slots;
  const int u = live ? u0 + cslot : u0;
  const int col = a.daylist[a.chunk_first + u];
  const SwColRec &R = sw_colrecs(a)[u];
  const Col C = R.C;
  const int n = C.nlay;
  const bool clear_only = a.icld == 0;
  int band = kSwBands - 1;
  while (G < kSwGofsDev[band]) --band;
  const float *opt = sw_optrec(a, u, 0);
  const uint32_t *mword = a.mask + col + static_cast<size_t>(G >> 5) * a.ncol;
  const size_t mstride = static_cast<size_t>(kSwMaskWords) * a.ncol;
  const uint32_t bit = 1u << (G & 31);
  const float zincflx = ((C.adjflux * R.sflux[G]) * C.mu) * 1.0f;
  float *const ring0 = &S.ring[0][cslot][G];
  constexpr int kTypeStep = kSweepCols * kRingStride, kBufStep = kRingRows * kRingStride;
  constexpr int kDownLevels = kRingRows / (2 * kSweepCols), kUpLevels = kRingRows / (4 * kSweepCols);
  static_assert(kUpLevels == kAhead && kDownLevels == 2 * kAhead, "levels per round");

  // a layer's optics on both paths (the total sky's where it is cloudy)
  struct Slot {
    float4 rt, trt;
    float2 d, td;
    bool cloudy;
  };
  auto load = [&](int l, Slot &s) {
    const float *q = opt + static_cast<size_t>(l) * kSwOpt;
    s.rt = reinterpret_cast<const float4 *>(q)[G];
    s.d = reinterpret_cast<const float2 *>(q + kSwOptClearDbt)[G];
    s.cloudy = !clear_only && (mword[static_cast<size_t>(l) * mstride] & bit) != 0u;
    s.trt = reinterpret_cast<const float4 *>(q + kSwOptTotal)[G];
    s.td = reinterpret_cast<const float2 *>(q + kSwOptTotalDbt)[G];
  };
  auto optics = [](const float4 &rt, const float2 &d) {
    SwOptics o;
    o.rt.ref = rt.x; o.rt.refd = rt.y; o.rt.tra = rt.z; o.rt.trad = rt.w;
    o.dbt = d.x;
    o.dbt_nd = d.y;
    return o;
  };

  // ---- top-down: the recurrences' values at each level go to the stacks
  SwCarry stc[kMaxLev], stt[kMaxLev];
  SwCarry cc{1.0f, 1.0f, 0.0f}, ct = cc;
  float tdbtc_nd = 1.0f, tdbt_nd = 1.0f;
  ring0[0] = tdbt_nd * zincflx;
  ring0[kTypeStep] = tdbtc_nd * zincflx;
  int filled = 1, level0 = 0, round = 0;
  Slot nx[kAhead];
#pragma unroll
  for (int j = 0; j < kAhead; ++j)
    if (j < n) load(n - 1 - j, nx[j]);
  for (int r0 = 0; r0 < n; r0 += kAhead) {
    Slot cur[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      cur[j] = nx[j];
      if (r0 + kAhead + j < n) load(n - 1 - (r0 + kAhead + j), nx[j]);
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int r = r0 + j;
      if (r >= n) break;
      const SwOptics oc = optics(cur[j].rt, cur[j].d);
      stc[r] = cc;
      stt[r] = ct;
      const SwOptics ot = cur[j].cloudy ? optics(cur[j].trt, cur[j].td) : oc;
      tdbt_nd = tdbt_nd * ot.dbt_nd;
      ct = sw_down(ct, ot, r == 0);
      tdbtc_nd = tdbtc_nd * oc.dbt_nd;
      cc = sw_down(cc, oc, r == 0);
      float *q = ring0 + (round & 1) * kBufStep + filled * (2 * kTypeStep);
      q[0] = tdbt_nd * zincflx;
      q[kTypeStep] = tdbtc_nd * zincflx;
      if (++filled == kDownLevels || r == n - 1) {
        sweep_flush<2>(S, round, filled, 4, level0, 1);
        ++round;
        level0 += filled;
        filled = 0;
      }
    }
  }

  // ---- bottom-up: adding from the surface and the level fluxes
  float albp = C.albedo, albd = C.albedo;
  sw_albedos(a, col, band, albp, albd);
  float rupc = albp, rupdc = albd, rupt = albp, rupdt = albd;
  level0 = n;
  auto level = [](const float4 &rt, float dbt, const SwCarry &c) {
    return SwLevel{rt, make_float4(dbt, c.tdbt, c.tdn, c.rdnd)};
  };
  struct Up {
    Slot s;
    SwCarry c, t;
  } up[kAhead];
  auto load_up = [&](int k, Up &v) {  // level k: the layer below it and the level's stack entries
    load(n - 1 - k, v.s);
    v.c = stc[k];
    v.t = stt[k];
  };
#pragma unroll
  for (int j = 0; j < kAhead; ++j)
    if (n - 1 - j >= 0) load_up(n - 1 - j, up[j]);
  const float4 surface = make_float4(albp, albd, 0.0f, 0.0f);
  auto emit = [&](int k, const SwLevel &c, const SwLevel &t) {
    float fuc, fdc, fut, fdt;
    sw_fluxes(c, rupc, rupdc, fuc, fdc);
    sw_fluxes(t, rupt, rupdt, fut, fdt);
    float *q = ring0 + (round & 1) * kBufStep + filled * (4 * kTypeStep);
    q[0] = fut * zincflx;
    q[kTypeStep] = fdt * zincflx;
    q[2 * kTypeStep] = fuc * zincflx;
    q[3 * kTypeStep] = fdc * zincflx;
    if (++filled == kUpLevels || k == 0) {
      sweep_flush<4>(S, round, filled, 0, level0, -1);
      ++round;
      level0 -= filled;
      filled = 0;
    }
  };
  filled = 0;
  emit(n, level(surface, 0.0f, cc), level(surface, 0.0f, ct));
  for (int k0 = n - 1; k0 >= 0; k0 -= kAhead) {
    Up cur[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      cur[j] = up[j];
      if (k0 - kAhead - j >= 0) load_up(k0 - kAhead - j, up[j]);
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int k = k0 - j;
      if (k < 0) break;
      const Slot &s = cur[j].s;
      const SwLevel c = level(s.rt, s.d.x, cur[j].c);
      const SwLevel t = s.cloudy ? level(s.trt, s.td.x, cur[j].t) : level(s.rt, s.d.x, cur[j].t);
      sw_up(c, rupc, rupdc);
      sw_up(t, rupt, rupdt);
      emit(k, c, t);
    }
  }
  __syncthreads();  // the last round's sums
  for (int q = threadIdx.x; q < kSweepCols * kMaxLay; q += kSweepThreads) {
    const int cs = q / kMaxLay, l = q - cs * kMaxLay;
    const int uq = u0 + cs;
    if (l >= a.nk || uq >= slots) continue;
    sw_layer_output(a, sw_colrecs(a)[uq].C, l, &S.sums[cs][0][0], kMaxLev);
  }
  if (G == 0 && live) sw_column_outputs(a, C, col, &S.sums[cslot][0][0], kMaxLev);
}

}  // namespace

cudaError_t launch_sw_daylist(const SwArgs &a, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(a.nday, 0, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  sw_daylist_kernel<<<(a.ncol + 255) / 256, 256, 0, stream>>>(a);
  return cudaGetLastError();
}

size_t sw_record_floats(int nk, int chunk) {
  return sw_base_floats(nk, chunk) +
         (chunk <= kSmallColumns
              ? static_cast<size_t>(kSwOpt) * (nk + 1) * (chunk < kSwSmallColumns ? chunk : kSwSmallColumns)
              : size_t(0));
}

cudaError_t launch_sw_chunk_optics(const Tables &T, const SwArgs &a, cudaStream_t stream) {
  const int threads = 128;
  const int n = a.nk + 1;
  sw_colprep_kernel<<<(a.chunk_count + 3) / 4, threads, 0, stream>>>(T, a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const long long layers = static_cast<long long>(a.chunk_count) * n;
  const long long blocks = (layers + threads - 1) / threads;
  sw_layer_kernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(T, a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // small capacities may hold few day slots: a bounded grid walks those there are
  const long long optics = blocks * kSwBands;
  const long long most = a.chunk_capacity <= kSmallColumns ? 148ll * kSwOpticsMinBlocks * 2 : optics;
  const int sources = (a.chunk_count + threads - 1) / threads * kSwBands;
  sw_optics_kernel<<<static_cast<unsigned>(sources + (optics < most ? optics : most)), threads, 0, stream>>>(T, a,
                                                                                                        sources);
  return cudaGetLastError();
}

static_assert(sizeof(SweepShared) <= 48 * 1024, "more shared memory needs the opt-in");

template <bool kFp64>
static cudaError_t launch_sweep(const Tables &T, const SwArgs &a, cudaStream_t stream) {
  const int pairs = (a.chunk_count + kSweepCols - 1) / kSweepCols;
  if (a.chunk_capacity <= kSmallColumns) {
    const int most = a.chunk_count < kSwSmallColumns ? a.chunk_count : kSwSmallColumns;
    const long long items = static_cast<long long>(most) * (a.nk + 1);
    sw_small_optics_kernel<kFp64><<<static_cast<int>(items < kSmallBlocks ? items : kSmallBlocks), kSwGpts, 0,
                                    stream>>>(T, a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    sw_small_sweep_kernel<<<(most + kSweepCols - 1) / kSweepCols, kSweepThreads, sizeof(SweepShared), stream>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess || a.chunk_count <= kSwSmallColumns) return e;
  }
  sw_sweep_kernel<kFp64><<<pairs, kSweepThreads, sizeof(SweepShared), stream>>>(T, a);
  return cudaGetLastError();
}

cudaError_t launch_sw_chunk_sweep(const Tables &T, const SwArgs &a, cudaStream_t stream) {
  return a.fp64_reftra ? launch_sweep<true>(T, a, stream) : launch_sweep<false>(T, a, stream);
}

}  // namespace rrtmg
