// RRTMG longwave on the GPU: the sweep schedule, from the WRF adapter to the
// theta tendencies.
//
// Reference call: rrtmg_lwrad_wrf_columns (src/wrf_jax/physics/module_ra_rrtmg_lw.py:6789)
// and everything below it: buffer layers (lw:6633-6786), cloud radii and paths
// (common:801-961), inatm (lw:953), setcoef (lw:1175), taumol1..16
// (lw:1597-4684), cldprmc (lw:5725), rtrnmc (lw:5476-5722), broadband sums
// (lw:170-199) and the theta tendency (lw:7040-7057).  McICA masks come from
// rrtmg_mcica.cu.
//
// Inputs are read in place from WRF's (x, z, y) layout, where neighbouring
// columns of a row are adjacent in memory at every level, so a warp's loads
// are coalesced.
#include "rrtmg_lw_common.cuh"

namespace rrtmg {
namespace {

// ---------------------------------------------------------------------------
// Sweep schedule, every domain size.  Columns are processed in chunks; per
// chunk:
//   lw_colprep_kernel  warp = column: buffer layers, column integrals (laytrop,
//                      pwvcm, summed in layer order), band diffusivities, and
//                      whether any layer is cloudy;
//   lw_layer_kernel    thread = (layer, column): the layer set-up (make_layer)
//                      once; the inputs of the gas optics go to a
//                      structure-of-arrays record, each band's Planck terms and
//                      cloud optical depth and the layer's cloud flag to the
//                      layer record;
//   lw_gas_kernel      thread = (layer, column), grid.y = band: the band's gas
//                      optical depths and Planck fractions (taumol) into the
//                      layer record, so every warp runs one band's code;
//   lw_sweep_kernel    block = kLwSweepCols columns x 140 g-points, thread =
//                      one g-point: the downward and upward radiance sweeps of
//                      rtrnmc (lw:5476-5722) from the layer records; each
//                      level's radiances go to shared memory, where they are
//                      summed in g-point order per band and the band terms in
//                      band order (lw:170-199); then fluxes, heating rates and
//                      the 2-D outputs.
// Operation for operation these are the reference's statements in its order,
// the same as the fused lw_kernel's, so the results are bit-identical.
// ---------------------------------------------------------------------------

// Layer record (kLwRec floats): taug of each band's g-points from a 16-byte
// boundary (kLwPadOfs), the Planck fractions likewise from kLwRecFracs, per
// band (blay, dplankup, dplankdn, cloud optical depth) from kLwRecBand, and
// the layer's cloud flag at kLwRecFlags.
constexpr int kLwPadOfs[kLwBands] = {0, 12, 24, 40, 56, 72, 80, 92, 100, 112, 120, 128, 136, 140, 144, 148};
constexpr int kLwPadG = 152;
static_assert(kLwPadOfs[kLwBands - 1] + lw_pad(kLwBands - 1) == kLwPadG, "padded g-points");
constexpr int kLwRecFracs = kLwPadG, kLwRecBand = 2 * kLwPadG, kLwRecFlags = kLwRecBand + 4 * kLwBands;
constexpr int kLwRec = kLwRecFlags + 4;
static_assert(kLwRec % 4 == 0, "layer records are float4 aligned");
__constant__ int kLwPadOfsDev[kLwBands] = {0, 12, 24, 40, 56, 72, 80, 92, 100, 112, 120, 128, 136, 140, 144, 148};
__constant__ int kNgcDev[kLwBands] = {10, 12, 16, 14, 16, 8, 12, 8, 12, 6, 8, 8, 4, 2, 2, 2};
__constant__ int kGofsDev[kLwBands] = {0, 10, 22, 38, 52, 68, 76, 88, 96, 108, 114, 122, 130, 134, 136, 138};

// The Layer fields taumol reads, stored field by field ([field][layer][column]).
#define RRTMG_LW_GAS_FLOATS(X)                                                                                   \
  X(pavel) X(coldry) X(wx0) X(wx1) X(wx2) X(wx3) X(colh2o) X(colco2) X(colo3) X(coln2o) X(colco) X(colch4)      \
  X(colo2) X(colbrd) X(fac00) X(fac01) X(fac10) X(fac11) X(rat_h2oco2) X(rat_h2oco2_1) X(rat_h2oo3)             \
  X(rat_h2oo3_1) X(rat_h2on2o) X(rat_h2on2o_1) X(rat_h2och4) X(rat_h2och4_1) X(rat_n2oco2) X(rat_n2oco2_1)      \
  X(rat_o3co2) X(rat_o3co2_1) X(selffac) X(selffrac) X(forfac) X(forfrac) X(minorfrac) X(scaleminor)            \
  X(scaleminorn2)
#define RRTMG_LW_GAS_INTS(X) X(jp) X(jt) X(jt1) X(indself) X(indfor) X(indminor) X(trop)
#define RRTMG_LW_COUNT(name) +1
constexpr int kLwGasFields = 0 RRTMG_LW_GAS_FLOATS(RRTMG_LW_COUNT) RRTMG_LW_GAS_INTS(RRTMG_LW_COUNT);
#undef RRTMG_LW_COUNT

// Per-column record, computed once per column.
struct ColRec {
  Col C;
  float secdiff[kLwBands];
  int has_cloud;
};
constexpr size_t kColRecFloats = (sizeof(ColRec) + 15) / 16 * 4;

// scratch of one chunk: column records, then the gas fields, then the layer records
__device__ __forceinline__ const ColRec *col_records(const LwArgs &a) {
  return reinterpret_cast<const ColRec *>(a.scratch);
}
__device__ __forceinline__ float *gas_fields(const LwArgs &a) {
  return a.scratch + kColRecFloats * static_cast<size_t>(a.chunk_capacity);
}
__device__ __forceinline__ float *layer_records(const LwArgs &a) {
  return gas_fields(a) + static_cast<size_t>(kLwGasFields) * a.nlay * a.chunk_capacity;
}

__device__ __forceinline__ bool load_mask(const LwArgs &a, int l, int col, uint32_t *mask) {
  uint32_t any = 0;
#pragma unroll
  for (int w = 0; w < kLwMaskWords; ++w) {
    mask[w] = a.mask[(static_cast<size_t>(l) * kLwMaskWords + w) * a.ncol + col];
    any |= mask[w];
  }
  return any != 0u;
}

// A warp per column: the lanes take the buffer levels of the column set-up
// and the layers of the column integrals, whose sums are then taken in layer
// order from shared memory (the operations and order of column_prologue).
__global__ void __launch_bounds__(128) lw_colprep_kernel(Tables T, LwArgs a) {
  __shared__ float s_cd[4][kMaxLay], s_wk[4][kMaxLay];
  __shared__ float s_tlev[4][kMaxBuf + 1], s_o3[4][kMaxBuf];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lc = blockIdx.x * 4 + w;
  if (lc >= a.chunk_count || dead_column(a.live, a.chunk_first + lc)) return;  // whole warps
  const int col = a.chunk_first + lc;
  ColRec r;
  Col &C = r.C;
  column_head(a, col, C);
  column_setup<true>(T, a, C, lane, s_tlev[w], s_o3[w]);
  const int nlay = C.nlay;
  int trop_count = 0;
  bool cloud = false;
  for (int l = lane; l < nlay; l += 32) {
    bool trop;
    column_layer(T, a, C, l, trop, s_cd[w][l], s_wk[w][l]);
    trop_count += trop;
    uint32_t mask[kLwMaskWords];
    cloud = load_mask(a, l, col, mask) || cloud;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) trop_count += __shfl_xor_sync(0xffffffffu, trop_count, o);
  const bool has_cloud = __any_sync(0xffffffffu, cloud);
  __syncwarp();
  float amttl = 0.0f, wvttl = 0.0f;
  for (int l = 0; l < nlay; ++l) {
    amttl = (amttl + s_cd[w][l]) + s_wk[w][l];
    wvttl = wvttl + s_wk[w][l];
  }
  C.laytrop = trop_count;
  C.pwvcm = column_pwvcm(a, C, amttl, wvttl);
  column_secdiff(T, C, r.secdiff);
  r.has_cloud = has_cloud ? 1 : 0;
  if (lane == 0) reinterpret_cast<ColRec *>(a.scratch)[lc] = r;
}

// thread = (layer, chunk column), columns fastest
// Resident blocks per SM the register allocation must allow (measured at
// 425 x 425 x 50: without a bound the layer kernel takes 242 registers, two
// blocks per SM; the gas kernel at 5 blocks (96 registers) takes as long as at
// 4 or 6 within 2%, at 8 (64 registers, spills) 10% longer; the sweep at 56
// registers instead of 67 takes 27.7 ms instead of 32.9).
constexpr int kLwLayerMinBlocks = 6;
constexpr int kLwGasMinBlocks = 5;
constexpr int kLwSweepMinBlocks = 4;
__global__ void __launch_bounds__(128, kLwLayerMinBlocks) lw_layer_kernel(Tables T, LwArgs a) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int l = static_cast<int>(idx / a.chunk_count);
  const int lc = static_cast<int>(idx - static_cast<long long>(l) * a.chunk_count);
  if (l >= a.nlay) return;
  const int col = a.chunk_first + lc;
  if (dead_column(a.live, col)) return;
  const Col &C = col_records(a)[lc].C;
  const Layer L = make_layer(T, a, C, l);
  float *gas = gas_fields(a) + static_cast<size_t>(l) * a.chunk_capacity + lc;
  const size_t fstride = static_cast<size_t>(a.nlay) * a.chunk_capacity;
  int f = 0;
#define RRTMG_LW_PUT(name) gas[static_cast<size_t>(f++) * fstride] = L.name;
#define RRTMG_LW_PUTI(name) gas[static_cast<size_t>(f++) * fstride] = __int_as_float(L.name);
  RRTMG_LW_GAS_FLOATS(RRTMG_LW_PUT)
  RRTMG_LW_GAS_INTS(RRTMG_LW_PUTI)
#undef RRTMG_LW_PUT
#undef RRTMG_LW_PUTI
  uint32_t mask[kLwMaskWords];
  const bool cloudy = load_mask(a, l, col, mask);
  float4 *rec = reinterpret_cast<float4 *>(layer_records(a) + (static_cast<size_t>(lc) * a.nlay + l) * kLwRec);
  const int iceflag = C.iceflg;
#pragma unroll 1
  for (int b = 0; b < kLwBands; ++b) {
    const float blay = planck(T, L.indlay, L.tlayfrac, b);
    const float dplankup = planck(T, L.indlev1, L.tlev1frac, b) - blay;
    const float dplankdn = planck(T, L.indlev0, L.tlev0frac, b) - blay;
    float teff = 0.0f;
    if (cloudy) {
      bool active = false;
      const float tauc = cloud_tau(T, L, b, iceflag, active);
      teff = active ? tauc : 0.0f;
    }
    rec[kLwRecBand / 4 + b] = make_float4(blay, dplankup, dplankdn, teff);
  }
  rec[kLwRecFlags / 4] = make_float4(cloudy ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f);
}

// 16-byte pieces of a warp's stage: optical depths, then fractions, of 32 rows of up to 5
constexpr int kGasStage = 2 * 32 * 5;

// Band B of the layer records of a warp's 32 (layer, column) pairs.  The gas
// fields are read here, inside the band's own code, so that each band loads
// only the ones that it uses.  The results go through the warp's shared stage
// so that neighbouring lanes write neighbouring 16-byte pieces: a store then
// touches 32 / Q records' lines instead of 32.
// record: the lane's layer record, or -1 where it has none.
template <int B>
__device__ __forceinline__ void gas_band(const Tables &T, const LwArgs &a, const float *gas, int record, float4 *stage) {
  constexpr int Q = lw_pad(B) / 4, kRow = Q | 1;  // stage rows of an odd number of 16-byte pieces
  const int lane = threadIdx.x & 31;
  if (record >= 0) {
    const size_t fstride = static_cast<size_t>(a.nlay) * a.chunk_capacity;
    Layer L{};
    int f = 0;
#define RRTMG_LW_GET(name) L.name = gas[static_cast<size_t>(f++) * fstride];
#define RRTMG_LW_GETI(name) L.name = __float_as_int(gas[static_cast<size_t>(f++) * fstride]);
    RRTMG_LW_GAS_FLOATS(RRTMG_LW_GET)
    RRTMG_LW_GAS_INTS(RRTMG_LW_GETI)
#undef RRTMG_LW_GET
#undef RRTMG_LW_GETI
    float4 *row = stage + lane * kRow;
    gas_quads<B>(T, L, [&](int q, float4 tau, float4 frac) {
      row[q] = tau;
      row[q + kGasStage / 2] = frac;
    });
  }
  __syncwarp();
  float *recs = layer_records(a) + kLwPadOfs[B];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int e = i * 32 + lane, r = e / Q, q = e - r * Q;
    const int rec = __shfl_sync(0xffffffffu, record, r);
    if (rec >= 0) {
      float4 *out = reinterpret_cast<float4 *>(recs + static_cast<size_t>(rec) * kLwRec) + q;
      out[0] = stage[r * kRow + q];
      out[kLwRecFracs / 4] = stage[r * kRow + q + kGasStage / 2];
    }
  }
}

// Blocks of (layer, chunk column) pairs taken kLwGasGroup at a time, each
// group through all 16 bands before the next: the group's gas fields and its
// layer records stay in L2 across its bands, so that records, which the bands
// fill 16 to 64 bytes at a time, leave it whole.  LW optics of 425 x 425 x 50
// (set-up included): 128 blocks 15.1 ms, 512 17.7 ms, 2,048 over 20 ms; with
// one store per lane and record instead of the stage 18.3 ms, and with the
// bands' g-points unrolled over unpadded tables 26.1 ms.
constexpr int kLwGasGroup = 128;

// thread = (layer, chunk column) of block `blk`; band from the block order above
__global__ void __launch_bounds__(128, kLwGasMinBlocks) lw_gas_kernel(Tables T, LwArgs a, int nblk) {
  const int group = blockIdx.x / (kLwGasGroup * kLwBands);
  const int g0 = group * kLwGasGroup;
  const int gsize = nblk - g0 < kLwGasGroup ? nblk - g0 : kLwGasGroup;
  const int within = blockIdx.x - group * kLwGasGroup * kLwBands;
  const int band = within / gsize;
  const int blk = g0 + (within - band * gsize);
  const long long idx = static_cast<long long>(blk) * blockDim.x + threadIdx.x;
  const int l = static_cast<int>(idx / a.chunk_count);
  const int lc = static_cast<int>(idx - static_cast<long long>(l) * a.chunk_count);
  const bool live = l < a.nlay && !dead_column(a.live, a.chunk_first + lc);
  if (!__any_sync(0xffffffffu, live)) return;  // whole warps
  __shared__ float4 stages[4][kGasStage];
  float4 *stage = stages[threadIdx.x >> 5];
  const float *gas = gas_fields(a) + static_cast<size_t>(l) * a.chunk_capacity + lc;
  const int record = live ? lc * a.nlay + l : -1;
  switch (band) {
    case 0: gas_band<0>(T, a, gas, record, stage); break;
    case 1: gas_band<1>(T, a, gas, record, stage); break;
    case 2: gas_band<2>(T, a, gas, record, stage); break;
    case 3: gas_band<3>(T, a, gas, record, stage); break;
    case 4: gas_band<4>(T, a, gas, record, stage); break;
    case 5: gas_band<5>(T, a, gas, record, stage); break;
    case 6: gas_band<6>(T, a, gas, record, stage); break;
    case 7: gas_band<7>(T, a, gas, record, stage); break;
    case 8: gas_band<8>(T, a, gas, record, stage); break;
    case 9: gas_band<9>(T, a, gas, record, stage); break;
    case 10: gas_band<10>(T, a, gas, record, stage); break;
    case 11: gas_band<11>(T, a, gas, record, stage); break;
    case 12: gas_band<12>(T, a, gas, record, stage); break;
    case 13: gas_band<13>(T, a, gas, record, stage); break;
    case 14: gas_band<14>(T, a, gas, record, stage); break;
    default: gas_band<15>(T, a, gas, record, stage); break;
  }
}

// One g-point of band_sums: the new radiances (rA, rB) after one layer, from
// the g-point's gas optical depth tg and Planck fraction fr, its band's
// (blay, dplankup, dplankdn, cloud optical depth) bq, its McICA bit cld and
// the layer's cloud flag.
template <bool kDown>
__device__ __forceinline__ void lw_step(const Tables &T, float tg, float fr, float4 bq, bool cld, bool cloudy_layer,
                                        float secdiff, float &rA, float &rB, bool sep_clear) {
  float odepth = secdiff * tg;
  if (odepth < 0.0f) odepth = 0.0f;
  float odcld = 0.0f, efcl = 0.0f;
  if (cld) {
    const float odcld_raw = secdiff * bq.w;
    const float abscld = 1.0f - glibc_expf(T, -odcld_raw);
    odcld = odcld_raw;
    efcl = abscld * 1.0f;
  }
  const Terms tm = layer_terms(T, cloudy_layer, odepth, odcld, fr, bq.x, bq.z, bq.y);
  const float cf = cld ? 1.0f : 0.0f;
  const float r = rA, rc = rB;
  float rn;
  if constexpr (kDown) {
    if (cloudy_layer) {
      rn = r - r * (tm.a + efcl * (1.0f - tm.a)) + tm.gassrc + cf * (tm.bbdtot * tm.atot - tm.gassrc);
    } else {
      rn = r + (tm.bbdgas - r) * tm.a;
    }
    rB = sep_clear ? rc + (tm.bbdgas - rc) * tm.a : rn;
  } else {
    if (cloudy_layer) {
      const float gas = tm.bbugas * tm.a;
      rn = r - r * (tm.a + efcl * (1.0f - tm.a)) + gas + cf * (tm.bbutot * tm.atot - gas);
    } else {
      rn = r + (tm.bbugas - r) * tm.a;
    }
    rB = sep_clear ? rc + (tm.bbugas - rc) * tm.a : rn;
  }
  rA = rn;
}

constexpr int kLwSweepCols = 2;                            // columns per block
constexpr int kLwSweepThreads = 288;                       // 2 x 140 g-points in 9 warps; 8 padding threads
constexpr int kLwRing = 8;                                 // levels of radiances per ordered-sum round
static_assert(kLwSweepThreads >= kLwSweepCols * kLwGpts && kLwSweepThreads % 32 == 0, "sweep block shape");

struct LwSweepShared {
  float ring[kLwRing][kLwSweepCols][2][kLwGpts];      // total, clear radiance of each g-point
  float bands[kLwRing][kLwSweepCols][2][kLwBands];    // each band's radiance sum
  float flux[kLwSweepCols][4][kMaxLay + 1];           // up total, up clear, down total, down clear per level
};

// Sums the ring's levels in two rounds of independent chains: (column,
// total/clear, level, band) adds the band's radiances in g-point order, then
// (column, total/clear, level) adds the band terms (bandsum * 0.5) * delwave in
// band order (band_step, lw:170-199) and multiplies by fluxfac.  The
// operations and their order are those of one sequential sum per level.
__device__ __forceinline__ void lw_flush(LwSweepShared &S, int count, int type0, int level0, int dir) {
  __syncthreads();
  const float pi = 3.1415926535897932384626433832795f;
  const float fluxfac = pi * 2.0e4f;
  const int band_chains = kLwSweepCols * 2 * count * kLwBands;
  for (int ch = threadIdx.x; ch < band_chains; ch += kLwSweepThreads) {
    const int b = ch % kLwBands;
    const int rest = ch / kLwBands;
    const int j = rest % count;
    const int cq = rest / count;  // column * 2 + total/clear
    const float *v = S.ring[j][cq >> 1][cq & 1] + kGofsDev[b];
    const int ngc = kNgcDev[b];
    float bandsum = 0.0f;
    for (int g = 0; g < ngc; ++g) bandsum = bandsum + v[g];
    S.bands[j][cq >> 1][cq & 1][b] = bandsum;
  }
  __syncthreads();
  const int chains = kLwSweepCols * 2 * count;
  for (int ch = threadIdx.x; ch < chains; ch += kLwSweepThreads) {
    const int j = ch % count;
    const int cq = ch / count;
    const float *bs = S.bands[j][cq >> 1][cq & 1];
    float total = 0.0f;
#pragma unroll
    for (int b = 0; b < kLwBands; ++b) total = total + (bs[b] * 0.5f) * kDelwave[b];
    S.flux[cq >> 1][type0 + (cq & 1)][level0 + dir * j] = total * fluxfac;
  }
  __syncthreads();
}

// Block = kLwSweepCols consecutive columns of the chunk.  A column past the
// chunk or the live count repeats the block's first column so that every
// thread takes the same barriers; its results are not written.
__global__ void __launch_bounds__(kLwSweepThreads, kLwSweepMinBlocks) lw_sweep_kernel(Tables T, LwArgs a) {
  __shared__ __align__(16) LwSweepShared S;
  const int lc0 = blockIdx.x * kLwSweepCols;
  if (lc0 >= a.chunk_count || dead_column(a.live, a.chunk_first + lc0)) return;  // whole block
  const int tid = threadIdx.x;
  const bool writer = tid < kLwSweepCols * kLwGpts;
  const int cslot = writer ? tid / kLwGpts : kLwSweepCols - 1;
  const int G = writer ? tid - cslot * kLwGpts : kLwGpts - 1;
  const int lc_own = lc0 + cslot;
  const bool live = lc_own < a.chunk_count && !dead_column(a.live, a.chunk_first + lc_own);
  const int lc = live ? lc_own : lc0;
  const int col = a.chunk_first + lc;
  int band = kLwBands - 1;
  while (G < kGofsDev[band]) --band;
  const int P = kLwPadOfsDev[band] + (G - kGofsDev[band]);
  const ColRec &R = col_records(a)[lc];
  const float sd = R.secdiff[band];
  const bool has_cloud = R.has_cloud != 0;
  const int nlay = a.nlay, nk = a.nk;
  const float *recs = layer_records(a) + static_cast<size_t>(lc) * nlay * kLwRec;
  const uint32_t *mword = a.mask + col + static_cast<size_t>(G >> 5) * a.ncol;
  const size_t mstride = static_cast<size_t>(kLwMaskWords) * a.ncol;
  const uint32_t bit = 1u << (G & 31);
  const float pi = 3.1415926535897932384626433832795f;
  const float fluxfac = pi * 2.0e4f;
  if (tid < kLwSweepCols * 2) S.flux[tid >> 1][2 + (tid & 1)][nlay] = 0.0f * fluxfac;  // no downward flux at the top

  // downward sweep, top to bottom: layer l gives level l; next layer loaded ahead
  float rA = 0.0f, rB = 0.0f;
  bool iclddn = false;
  int filled = 0, level0 = nlay - 1;
  const float *q = recs + static_cast<size_t>(nlay - 1) * kLwRec;
  float nx_tg = q[P], nx_fr = q[kLwRecFracs + P];
  float4 nx_bq = *reinterpret_cast<const float4 *>(q + kLwRecBand + 4 * band);
  float nx_flag = q[kLwRecFlags];
  uint32_t nx_word = mword[static_cast<size_t>(nlay - 1) * mstride];
  for (int l = nlay - 1; l >= 0; --l) {
    const float tg = nx_tg, fr = nx_fr, flag = nx_flag;
    const float4 bq = nx_bq;
    const uint32_t word = nx_word;
    if (l > 0) {
      q = recs + static_cast<size_t>(l - 1) * kLwRec;
      nx_tg = q[P];
      nx_fr = q[kLwRecFracs + P];
      nx_bq = *reinterpret_cast<const float4 *>(q + kLwRecBand + 4 * band);
      nx_flag = q[kLwRecFlags];
      nx_word = mword[static_cast<size_t>(l - 1) * mstride];
    }
    const bool cloudy = flag != 0.0f;
    iclddn = iclddn || cloudy;
    lw_step<true>(T, tg, fr, bq, (word & bit) != 0u, cloudy, sd, rA, rB, iclddn);
    if (writer) {
      S.ring[filled][cslot][0][G] = rA;
      S.ring[filled][cslot][1][G] = rB;
    }
    if (++filled == kLwRing || l == 0) {
      lw_flush(S, filled, 2, level0, -1);
      level0 -= filled;
      filled = 0;
    }
  }
  // surface emission and reflection: level 0 upward (surface_sums, lw:5648-5655)
  {
    const float bt = R.C.tsfc - 159.0f;
    const int indbound = clampi(static_cast<int>(bt), 1, 180);
    const float tbndfrac = bt - static_cast<float>(indbound);
    const float reflect = 1.0f - R.C.semiss;
    const float plankbnd = R.C.semiss * planck(T, indbound, tbndfrac, band);
    const float rad0 = recs[kLwRecFracs + P] * plankbnd;
    rA = rad0 + reflect * rA;
    rB = rad0 + reflect * rB;
    if (writer) {
      S.ring[0][cslot][0][G] = rA;
      S.ring[0][cslot][1][G] = rB;
    }
    filled = 1;
    level0 = 0;
  }
  // upward sweep, bottom to top: layer l gives level l + 1
  q = recs;
  nx_tg = q[P];
  nx_fr = q[kLwRecFracs + P];
  nx_bq = *reinterpret_cast<const float4 *>(q + kLwRecBand + 4 * band);
  nx_flag = q[kLwRecFlags];
  nx_word = mword[0];
  for (int l = 0; l < nlay; ++l) {
    const float tg = nx_tg, fr = nx_fr, flag = nx_flag;
    const float4 bq = nx_bq;
    const uint32_t word = nx_word;
    if (l + 1 < nlay) {
      q = recs + static_cast<size_t>(l + 1) * kLwRec;
      nx_tg = q[P];
      nx_fr = q[kLwRecFracs + P];
      nx_bq = *reinterpret_cast<const float4 *>(q + kLwRecBand + 4 * band);
      nx_flag = q[kLwRecFlags];
      nx_word = mword[static_cast<size_t>(l + 1) * mstride];
    }
    lw_step<false>(T, tg, fr, bq, (word & bit) != 0u, flag != 0.0f, sd, rA, rB, has_cloud);
    if (writer) {
      S.ring[filled][cslot][0][G] = rA;
      S.ring[filled][cslot][1][G] = rB;
    }
    if (++filled == kLwRing || l == nlay - 1) {
      lw_flush(S, filled, 0, level0, 1);
      level0 += filled;
      filled = 0;
    }
  }

  // heating rates and theta tendencies (lw:5706-5712, 7040-7057) and the 2-D
  // outputs (lw:7059-7077) of the block's live columns
  const float heatfac = (9.8066f * 8.6400e4f) / (1004.5f * 1.0e2f);
  for (int qq = tid; qq < kLwSweepCols * nk; qq += kLwSweepThreads) {
    const int cs = qq / nk, l = qq - cs * nk;
    const int lcq = lc0 + cs;
    if (lcq >= a.chunk_count || dead_column(a.live, a.chunk_first + lcq)) continue;
    const int cq = a.chunk_first + lcq;
    const int i = cq / a.ny, j = cq - i * a.ny;
    const float(*fx)[kMaxLay + 1] = S.flux[cs];
    const float fnet0 = fx[0][l] - fx[2][l], fnet1 = fx[0][l + 1] - fx[2][l + 1];
    const float fnetc0 = fx[1][l] - fx[3][l], fnetc1 = fx[1][l + 1] - fx[3][l + 1];
    const size_t rbase = static_cast<size_t>(i) * nk * a.ny + j;
    const size_t wbase = static_cast<size_t>(i) * (nk + 1) * a.ny + j;
    const float plev0 = pa_to_hpa(ld(a.in.p8w + wbase + static_cast<size_t>(l) * a.ny));
    const float plev1 = pa_to_hpa(ld(a.in.p8w + wbase + static_cast<size_t>(l + 1) * a.ny));
    const float dp = plev0 - plev1;
    float htr = heatfac * (fnet0 - fnet1) / dp;
    float htrc = heatfac * (fnetc0 - fnetc1) / dp;
    if (l >= a.fp64_from) {
      htr = heating64(heatfac, fx[0][l], fx[2][l], fx[0][l + 1], fx[2][l + 1], plev0, plev1);
      htrc = heating64(heatfac, fx[1][l], fx[3][l], fx[1][l + 1], fx[3][l + 1], plev0, plev1);
    }
    const float pi3d = ld(a.in.pi3d + rbase + static_cast<size_t>(l) * a.ny);
    a.rthraten[rbase + static_cast<size_t>(l) * a.ny] = (htr / 86400.0f) / pi3d;
    a.rthratenc[rbase + static_cast<size_t>(l) * a.ny] = (htrc / 86400.0f) / pi3d;
  }
  if (G == 0 && writer && live) {
    const float(*fx)[kMaxLay + 1] = S.flux[cslot];
    const float uflt = fx[0][nlay], ufltc = fx[1][nlay];
    const float dflt = 0.0f * fluxfac;
    a.upt[col] = uflt;
    a.uptc[col] = ufltc;
    a.dnt[col] = dflt;
    a.dntc[col] = dflt;
    a.upb[col] = fx[0][0];
    a.upbc[col] = fx[1][0];
    a.dnb[col] = fx[2][0];
    a.dnbc[col] = fx[3][0];
    a.glw[col] = fx[2][0];
    a.olr[col] = uflt;
    a.lwcf[col] = ufltc - uflt;
#pragma unroll
    for (int z = 0; z < 4; ++z) a.zero2[z][col] = 0.0f;
  }
}

}  // namespace

size_t lw_scratch_floats(int nlay, int chunk) {
  return (kColRecFloats + (static_cast<size_t>(kLwGasFields) + kLwRec) * nlay) * static_cast<size_t>(chunk);
}

cudaError_t launch_lw_chunk_optics(const Tables &T, const LwArgs &a, cudaStream_t stream) {
  const int threads = 128;
  lw_colprep_kernel<<<(a.chunk_count + 3) / 4, threads, 0, stream>>>(T, a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const long long layers = static_cast<long long>(a.chunk_count) * a.nlay;
  const unsigned blocks = static_cast<unsigned>((layers + threads - 1) / threads);
  lw_layer_kernel<<<blocks, threads, 0, stream>>>(T, a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  lw_gas_kernel<<<blocks * kLwBands, threads, 0, stream>>>(T, a, static_cast<int>(blocks));
  return cudaGetLastError();
}

cudaError_t launch_lw_chunk_sweep(const Tables &T, const LwArgs &a, cudaStream_t stream) {
  lw_sweep_kernel<<<(a.chunk_count + kLwSweepCols - 1) / kLwSweepCols, kLwSweepThreads, 0, stream>>>(T, a);
  return cudaGetLastError();
}

}  // namespace rrtmg
