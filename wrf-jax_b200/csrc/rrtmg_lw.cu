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
// band (blay, dplankup, dplankdn, cloud optical depth along the diffusivity
// angle) from kLwRecBand and the cloud's absorptance from kLwRecEfcl, and from
// kLwRecMask the layer's McICA mask words.  The sweep's
// downward pass leaves its transfer-table positions in place of the optical
// depths for the upward pass (lw_down).
constexpr int kLwPadOfs[kLwBands] = {0, 12, 24, 40, 56, 72, 80, 92, 100, 112, 120, 128, 136, 140, 144, 148};
constexpr int kLwPadG = 152;
static_assert(kLwPadOfs[kLwBands - 1] + lw_pad(kLwBands - 1) == kLwPadG, "padded g-points");
constexpr int kLwRecFracs = kLwPadG, kLwRecBand = 2 * kLwPadG, kLwRecEfcl = kLwRecBand + 4 * kLwBands;
constexpr int kLwRecMask = kLwRecEfcl + kLwBands;
constexpr int kLwRec = kLwRecMask + 8;
static_assert(kLwRec % 8 == 0 && kLwMaskWords <= 8, "layer records are whole sectors");
__constant__ int kLwPadOfsDev[kLwBands] = {0, 12, 24, 40, 56, 72, 80, 92, 100, 112, 120, 128, 136, 140, 144, 148};
__constant__ int kLwPadDev[kLwBands] = {12, 12, 16, 16, 16, 8, 12, 8, 12, 8, 8, 8, 4, 4, 4, 4};
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
  uint32_t cloud[kMaxLay / 32];  // bit l % 32 of word l / 32: layer l is cloudy in some g-point
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

// Columns of the launched chunk that are processed, and whether the small-chunk
// form takes them.
__device__ __forceinline__ int lw_chunk_columns(const LwArgs &a) {
  if (!a.live) return a.chunk_count;
  const int left = *a.live - a.chunk_first;
  return left < a.chunk_count ? left : a.chunk_count;
}
__device__ __forceinline__ bool lw_small(const LwArgs &a, int columns) {
  return a.chunk_capacity <= kSmallColumns && columns <= kLwSmallColumns;
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
// order from shared memory (the operations and order of column_setup).  Bound
// by latency: the record is built in shared memory and leaves it in whole
// lines; in every lane's local memory, stored by one lane, 2,048 slots took 27
// us and 4,096 columns 44 us (LW optics of 64 x 64 x 44 323 -> 300 us, of
// 300 x 300 x 50 6.56 -> 6.09 ms).
__global__ void __launch_bounds__(128) lw_colprep_kernel(const __grid_constant__ Tables T, const LwArgs a) {
  __shared__ float s_cd[4][kMaxLay], s_wk[4][kMaxLay];
  __shared__ float s_tlev[4][kMaxBuf + 2], s_o3[4][kMaxBuf + 1];
  __shared__ Col s_col[4];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lc = blockIdx.x * 4 + w;
  if (lc >= a.chunk_count || dead_column(a.live, a.chunk_first + lc)) return;  // whole warps
  const int col = a.chunk_first + lc;
  Col &C = s_col[w];
  column_head(a, col, C);
  __syncwarp();
  column_setup_warp(T, a, C, lane, s_tlev[w], s_o3[w]);
  const int nlay = C.nlay;
  int trop_count = 0;
#pragma unroll 1
  for (int i = 0; i < kMaxLay / 32; ++i) {
    const int l = 32 * i + lane;
    bool cloud = false;
    if (l < nlay) {
      bool trop;
      column_layer(T, a, C, l, trop, s_cd[w][l], s_wk[w][l]);
      trop_count += trop;
      uint32_t mask[kLwMaskWords];
      cloud = load_mask(a, l, col, mask);
    }
    const uint32_t word = __ballot_sync(0xffffffffu, cloud);
    if (lane == 0) reinterpret_cast<ColRec *>(a.scratch)[lc].cloud[i] = word;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) trop_count += __shfl_xor_sync(0xffffffffu, trop_count, o);
  __syncwarp();
  float amttl = 0.0f, wvttl = 0.0f;
  for (int l = 0; l < nlay; ++l) {
    amttl = (amttl + s_cd[w][l]) + s_wk[w][l];
    wvttl = wvttl + s_wk[w][l];
  }
  C.laytrop = trop_count;
  C.pwvcm = column_pwvcm(a, C, amttl, wvttl);
  __syncwarp();
  ColRec &out = reinterpret_cast<ColRec *>(a.scratch)[lc];
  if (lane < kLwBands) out.secdiff[lane] = band_secdiff(T, C, lane);
  static_assert(sizeof(Col) % 4 == 0, "words");
  for (int q = lane; q < static_cast<int>(sizeof(Col) / 4); q += 32)
    reinterpret_cast<float *>(&out.C)[q] = reinterpret_cast<const float *>(&C)[q];
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

// A warp's 32 layer records written Q 16-byte pieces at a time: `row` is the
// lane's row of the stage (rows of kRow pieces, an odd number, so that no banks
// conflict), its first Q pieces go to `at` floats into the lane's record.
// record: the lane's layer record, or -1 where it has none.
template <int Q, int kRow>
__device__ __forceinline__ void store_records(float *recs, int record, const float4 *stage, int at) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int e = i * 32 + lane, r = e / Q, q = e - r * Q;
    const int rec = __shfl_sync(0xffffffffu, record, r);
    if (rec >= 0) reinterpret_cast<float4 *>(recs + static_cast<size_t>(rec) * kLwRec + at)[q] = stage[r * kRow + q];
  }
  __syncwarp();
}

__global__ void __launch_bounds__(128, kLwLayerMinBlocks) lw_layer_kernel(Tables T, LwArgs a) {
  constexpr int kRow = 7;
  __shared__ float4 stages[4][32 * kRow];
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int l = static_cast<int>(idx / a.chunk_count);
  const int lc = static_cast<int>(idx - static_cast<long long>(l) * a.chunk_count);
  const int col = a.chunk_first + lc;
  const bool live = l < a.nlay && !dead_column(a.live, col);
  if (!__any_sync(0xffffffffu, live)) return;  // whole warps
  float4 *stage = stages[threadIdx.x >> 5];
  float4 *row = stage + (threadIdx.x & 31) * kRow;
  float *recs = layer_records(a);
  const int record = live ? lc * a.nlay + l : -1;
  const ColRec &R = col_records(a)[live ? lc : 0];
  Layer L{};
  uint32_t mask[kLwMaskWords] = {0};
  bool cloudy = false;
  if (live) {
    L = make_layer(T, a, R.C, l);
    float *gas = gas_fields(a) + static_cast<size_t>(l) * a.chunk_capacity + lc;
    const size_t fstride = static_cast<size_t>(a.nlay) * a.chunk_capacity;
    int f = 0;
#define RRTMG_LW_PUT(name) gas[static_cast<size_t>(f++) * fstride] = L.name;
#define RRTMG_LW_PUTI(name) gas[static_cast<size_t>(f++) * fstride] = __int_as_float(L.name);
    RRTMG_LW_GAS_FLOATS(RRTMG_LW_PUT)
    RRTMG_LW_GAS_INTS(RRTMG_LW_PUTI)
#undef RRTMG_LW_PUT
#undef RRTMG_LW_PUTI
    cloudy = load_mask(a, l, col, mask);
  }
  // four bands at a time: Planck terms and the cloud's optical depth and
  // absorptance along the diffusivity angle (lw:5562-5565).  The latter are the
  // same for all g-points of a band, so the binary64 exponential is evaluated
  // here, once per band and not once per g-point and direction.  Four bands per
  // table load and staged stores: 64 x 64 x 44 87 -> 63 us, LW optics of
  // 425 x 425 x 50 14.2 -> 13.2 ms.
  const int iceflag = a.iceflg;
  float4 efcl[kLwBands / 4];
#pragma unroll
  for (int b4 = 0; b4 < kLwBands / 4; ++b4) {
    efcl[b4] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (live) {
      const float4 blay = planck4(T, L.indlay, L.tlayfrac, b4);
      const float4 up = planck4(T, L.indlev1, L.tlev1frac, b4), dn = planck4(T, L.indlev0, L.tlev0frac, b4);
      float4 od = efcl[b4];
      if (cloudy) {
        bool active = false;
        const float4 tauc = cloud_tau4(T, L, b4, iceflag, active);
        const float *sd = R.secdiff + 4 * b4;
        const float4 t = active ? tauc : od;
        od = make_float4(sd[0] * t.x, sd[1] * t.y, sd[2] * t.z, sd[3] * t.w);
        auto absorptance = [&](float x) { return (1.0f - glibc_expf(T, -x)) * 1.0f; };
        efcl[b4] = make_float4(absorptance(od.x), absorptance(od.y), absorptance(od.z), absorptance(od.w));
      }
      row[0] = make_float4(blay.x, up.x - blay.x, dn.x - blay.x, od.x);
      row[1] = make_float4(blay.y, up.y - blay.y, dn.y - blay.y, od.y);
      row[2] = make_float4(blay.z, up.z - blay.z, dn.z - blay.z, od.z);
      row[3] = make_float4(blay.w, up.w - blay.w, dn.w - blay.w, od.w);
    }
    store_records<4, kRow>(recs, record, stage, kLwRecBand + 16 * b4);
  }
  static_assert(kLwMaskWords == 5 && kLwRecMask == kLwRecEfcl + kLwBands, "absorptances, then mask words");
#pragma unroll
  for (int b4 = 0; b4 < kLwBands / 4; ++b4) row[b4] = efcl[b4];
  row[4] = make_float4(__uint_as_float(mask[0]), __uint_as_float(mask[1]), __uint_as_float(mask[2]),
                       __uint_as_float(mask[3]));
  row[5] = make_float4(__uint_as_float(mask[4]), 0.0f, 0.0f, 0.0f);
  store_records<6, kRow>(recs, record, stage, kLwRecEfcl);
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
__global__ void __launch_bounds__(128, kLwGasMinBlocks) lw_gas_kernel(Tables T, LwArgs a) {
  __shared__ float4 stages[4][kGasStage];
  float4 *stage = stages[threadIdx.x >> 5];
  const int columns = lw_chunk_columns(a);
  const int nblk = static_cast<int>((static_cast<long long>(columns > 0 ? columns : 0) * a.nlay + 127) / 128);
  for (long long vb = blockIdx.x; vb < static_cast<long long>(nblk) * kLwBands; vb += gridDim.x) {
    const int group = static_cast<int>(vb / (kLwGasGroup * kLwBands));
    const int g0 = group * kLwGasGroup;
    const int gsize = nblk - g0 < kLwGasGroup ? nblk - g0 : kLwGasGroup;
    const int within = static_cast<int>(vb - static_cast<long long>(group) * (kLwGasGroup * kLwBands));
    const int band = within / gsize;
    const int blk = g0 + (within - band * gsize);
    const long long idx = static_cast<long long>(blk) * blockDim.x + threadIdx.x;
    const int l = static_cast<int>(idx / columns);
    const int lc = static_cast<int>(idx - static_cast<long long>(l) * columns);
    const bool live = l < a.nlay;
    if (!__any_sync(0xffffffffu, live)) continue;  // whole warps
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
    __syncwarp();  // the stage is read out
  }
}

// ---------------------------------------------------------------------------
// One g-point of one layer of rtrnmc (_rtrnmc_clear_terms / _rtrnmc_cloudy_terms,
// lw:5157-5262, and the radiance updates).  (a, x) are the layer's absorptance
// and the Planck interpolation factor of an optical depth: from the series
// where it is thin, else from the Pade tables, which the context holds as
// pairs (1 - exp, tfn).  The operations and their order are layer_terms' of
// the fused schedule; branches of it that give the same statements are merged,
// and the total-sky part is left out where the g-point has no cloud, since its
// weight there is zero.
// ---------------------------------------------------------------------------
struct LwGas {
  float a, x;
};

__device__ __forceinline__ LwGas lw_thin(float od) { return {od - (0.5f * od) * od, 0.166667f * od}; }

__device__ __forceinline__ LwGas lw_table(const Tables &T, int it) {
  const float2 v = __ldg(T.lw_pade + it);
  return {v.x, v.y};
}

// What the upward pass needs of a layer's transfer terms, in 32 bits: the gas
// optical depth itself where the series serves (sign bit clear), else the
// gas's table position, and above it (kLwTotShift) the cloudy total's.
constexpr uint32_t kLwTableBit = 0x80000000u;
constexpr int kLwTotShift = 15;
static_assert(kLwPadeMax < (1 << kLwTotShift), "table positions fit their bits");

// Total-sky (a, x) of a cloudy g-point whose gas is thin.
__device__ __forceinline__ LwGas lw_total_thin(const Tables &T, float odtot) {
  return odtot < 0.06f ? lw_thin(odtot) : lw_table(T, pade_index(T, odtot));
}

// New radiance of a g-point: rA total sky, rB clear sky.  src: the gas's
// source, tot: the cloudy total's.
__device__ __forceinline__ float lw_cloudy_radiance(float r, float a, float efcl, float src, float tot) {
  return r - r * (a + efcl * (1.0f - a)) + src + (tot - src);
}

// Downward: returns the word for the upward pass.
__device__ __forceinline__ uint32_t lw_down(const Tables &T, float tg, float fr, float4 bq, float efcl, bool cld,
                                            bool cloudy_layer, float secdiff, float &rA, float &rB, bool sep_clear) {
  float od = secdiff * tg;
  if (od <= 0.0f) od = 0.0f;
  const float odtot = od + bq.w;
  const bool thin = od <= 0.06f || (cloudy_layer && cld && odtot < 0.06f);
  LwGas g;
  uint32_t word;
  int ig = 0;
  if (thin) {
    g = lw_thin(od);
    word = __float_as_uint(od);
  } else {
    ig = pade_index(T, od);
    g = lw_table(T, ig);
    word = kLwTableBit | static_cast<uint32_t>(ig);
  }
  const float planck_dn = bq.x + g.x * bq.z;
  const float bbdgas = fr * planck_dn;
  if (cloudy_layer) {
    const float gassrc = thin ? bbdgas * g.a : (g.a * fr) * planck_dn;
    if (cld) {
      LwGas t;
      if (thin) {
        t = lw_total_thin(T, odtot);
      } else {
        const int it = pade_index(T, ld(T.lw_pade_tau + ig) + bq.w);
        t = lw_table(T, it);
        word |= static_cast<uint32_t>(it) << kLwTotShift;
      }
      const float bbdtot = fr * (bq.x + t.x * bq.z);
      rA = lw_cloudy_radiance(rA, g.a, efcl, gassrc, bbdtot * t.a);
    } else {
      rA = rA - rA * g.a + gassrc;
    }
    rB = rB + (bbdgas - rB) * g.a;
  } else {
    const float rn = rA + (bbdgas - rA) * g.a;
    rB = sep_clear ? rB + (bbdgas - rB) * g.a : rn;
    rA = rn;
  }
  return word;
}

__device__ __forceinline__ void lw_up(const Tables &T, uint32_t word, float fr, float4 bq, float efcl, bool cld,
                                      bool cloudy_layer, float &rA, float &rB, bool sep_clear) {
  const bool thin = (word & kLwTableBit) == 0u;
  const float od = __uint_as_float(word);
  constexpr uint32_t kPos = (1u << kLwTotShift) - 1u;
  const LwGas g = thin ? lw_thin(od) : lw_table(T, static_cast<int>(word & kPos));
  const float bbugas = fr * (bq.x + g.x * bq.y);
  if (cloudy_layer) {
    const float gas = bbugas * g.a;
    if (cld) {
      const LwGas t = thin ? lw_total_thin(T, od + bq.w)
                           : lw_table(T, static_cast<int>((word >> kLwTotShift) & kPos));
      const float bbutot = fr * (bq.x + t.x * bq.y);
      rA = lw_cloudy_radiance(rA, g.a, efcl, gas, bbutot * t.a);
    } else {
      rA = rA - rA * g.a + gas;
    }
    rB = rB + (bbugas - rB) * g.a;
  } else {
    const float rn = rA + (bbugas - rA) * g.a;
    rB = sep_clear ? rB + (bbugas - rB) * g.a : rn;
    rA = rn;
  }
}

// ---------------------------------------------------------------------------
// Small chunks.  With few columns a sweep is a serial chain in which each layer
// waits for its record and its table entries, although only the radiances
// depend on the layer before.  Here every layer's transfer terms are formed
// first, a thread per (column, layer, g-point), into term records, and the
// sweep reads them four layers ahead.  The operations are lw_down's and lw_up's.
// Sweep of 16 columns of 50 layers 92 -> 46 us, of 256 99 -> 70 us; of 512 107
// us against 118, as the term records (282 KB per column) then pass through
// memory: hence kLwSmallColumns.
// ---------------------------------------------------------------------------

// Transfer terms of a (layer, g-point): the gas's absorptance, the total's
// factor a + efcl (1 - a), and for either direction the gas's source function
// bb, and the gas and cloudy-total sources of the total-sky radiance.  Without
// cloud in the g-point the latter two are equal, and the radiance's last term
// is zero.
struct __align__(16) LwTerms {
  float a, atot, bbd, srcd, totd, bbu, srcu, totu;
};
constexpr int kLwTermFloats = 8 * kLwGpts;  // per (column, layer)

__device__ __forceinline__ LwTerms *lw_terms(const LwArgs &a, int lc, int l) {
  float *first = layer_records(a) + static_cast<size_t>(kLwRec) * a.nlay * a.chunk_capacity;
  return reinterpret_cast<LwTerms *>(first + (static_cast<size_t>(lc) * a.nlay + l) * kLwTermFloats);
}

__device__ __forceinline__ LwTerms lw_make_terms(const Tables &T, float tg, float fr, float4 bq, float efcl, bool cld,
                                                 bool cloudy_layer, float secdiff) {
  LwTerms t;
  float od = secdiff * tg;
  if (od <= 0.0f) od = 0.0f;
  const float odtot = od + bq.w;
  const bool thin = od <= 0.06f || (cloudy_layer && cld && odtot < 0.06f);
  int ig = 0;
  LwGas g;
  if (thin) {
    g = lw_thin(od);
  } else {
    ig = pade_index(T, od);
    g = lw_table(T, ig);
  }
  t.a = g.a;
  const float planck_dn = bq.x + g.x * bq.z;
  t.bbd = fr * planck_dn;
  t.bbu = fr * (bq.x + g.x * bq.y);
  t.srcd = thin ? t.bbd * g.a : (g.a * fr) * planck_dn;
  t.srcu = t.bbu * g.a;
  t.atot = g.a;
  t.totd = t.srcd;
  t.totu = t.srcu;
  if (cloudy_layer && cld) {
    const LwGas c = thin ? lw_total_thin(T, odtot) : lw_table(T, pade_index(T, ld(T.lw_pade_tau + ig) + bq.w));
    t.atot = g.a + efcl * (1.0f - g.a);
    t.totd = (fr * (bq.x + c.x * bq.z)) * c.a;
    t.totu = (fr * (bq.x + c.x * bq.y)) * c.a;
  }
  return t;
}

// One (column, layer) per item, a thread per g-point; the grid is bounded and
// walks the items, as the live count is known on the device only.
constexpr int kLwTermThreads = 160;
__global__ void __launch_bounds__(kLwTermThreads) lw_small_terms_kernel(const __grid_constant__ Tables T, LwArgs a) {
  const int columns = lw_chunk_columns(a);
  const int G = threadIdx.x;
  if (G >= kLwGpts || !lw_small(a, columns)) return;
  int band = kLwBands - 1;
  while (G < kGofsDev[band]) --band;
  const int P = kLwPadOfsDev[band] + (G - kGofsDev[band]);
  const int items = columns * a.nlay;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int lc = item / a.nlay, l = item - lc * a.nlay;
    const float *q = layer_records(a) + static_cast<size_t>(item) * kLwRec;
    const ColRec &R = col_records(a)[lc];
    const bool cloudy = (R.cloud[l >> 5] >> (l & 31)) & 1u;
    const bool cld = (__float_as_uint(q[kLwRecMask + (G >> 5)]) >> (G & 31)) & 1u;
    lw_terms(a, lc, l)[G] = lw_make_terms(T, q[P], q[kLwRecFracs + P],
                                          *reinterpret_cast<const float4 *>(q + kLwRecBand + 4 * band),
                                          q[kLwRecEfcl + band], cld, cloudy, R.secdiff[band]);
  }
}

constexpr int kLwSweepCols = 2;                            // columns per block
constexpr int kLwSweepThreads = 288;                       // 2 x 140 g-points in 9 warps; 8 padding threads
constexpr int kLwRing = 4;                                 // levels of radiances per ordered-sum round
constexpr int kLwRows = kLwRing * 2 * kLwSweepCols;        // (level, total / clear, column) rows of a round
constexpr int kLwRowStride = kLwPadG + 4;                  // an odd number of 16-byte pieces: no bank conflicts
static_assert(kLwSweepThreads >= kLwSweepCols * kLwGpts && kLwSweepThreads % 32 == 0, "sweep block shape");
static_assert(kLwRows == 16 && kLwBands == 16 && kLwSweepThreads / 32 == 9, "sum chains of a round: two bands a warp");
static_assert(kLwRowStride % 4 == 0 && (kLwRowStride / 4) % 2 == 1, "ring rows");

struct LwSweepShared {
  float ring[2][kLwRows][kLwRowStride];        // radiances of each g-point, bands padded with zeros
  float bands[2][kLwRows][kLwBands + 1];       // each band's radiance sum
  float flux[kLwSweepCols][4][kMaxLay + 1];    // up total, up clear, down total, down clear per level
  uint32_t cloud[kLwSweepCols][kMaxLay / 32];  // the columns' cloudy layers
};

// One round of levels awaiting its sums.
struct LwRound {
  int count, type0, level0, dir;
};

// bands of the two half warps of warp w < 8, of like length
__constant__ int kLwSumBand[2][8] = {{0, 2, 4, 8, 7, 10, 12, 14}, {1, 3, 6, 5, 9, 11, 13, 15}};

// Band terms (bandsum * 0.5) * delwave added in band order (lw:170-199) and
// multiplied by fluxfac: one lane per row of round `number`.
__device__ __forceinline__ void lw_band_terms(LwSweepShared &S, int number, const LwRound &r) {
  const float pi = 3.1415926535897932384626433832795f;
  const float fluxfac = pi * 2.0e4f;
  const int row = threadIdx.x & 31;
  if (row >= 2 * kLwSweepCols * r.count) return;
  const float *bs = S.bands[number & 1][row];
  float total = 0.0f;
#pragma unroll
  for (int b = 0; b < kLwBands; ++b) total = total + (bs[b] * 0.5f) * kDelwave[b];
  const int c = row % kLwSweepCols, type = row / kLwSweepCols % 2, j = row / (2 * kLwSweepCols);
  S.flux[c][r.type0 + type][r.level0 + r.dir * j] = total * fluxfac;
}

// Ordered sums of a round whose radiances have just been stored: warps 0-7
// add each band's radiances in g-point order (a half warp per band, a lane per
// row; the zero padding of a band adds nothing), and warp 8 adds the previous
// round's band terms.  The next round fills the other ring buffer meanwhile,
// so a round of four levels costs one barrier.  The operations and their order
// are those of one sequential sum per level.
// chain: the lane's band sum of every round (warps 0-7), found once.
struct LwChain {
  const float4 *v;  // its radiances in ring buffer 0
  float *sum;       // its place in bands[0]
  int quads;
};

__device__ __forceinline__ LwChain lw_chain(LwSweepShared &S) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = lane & 15, b = kLwSumBand[lane >> 4][warp & 7];
  return {reinterpret_cast<const float4 *>(S.ring[0][row] + kLwPadOfsDev[b]), &S.bands[0][row][b], kLwPadDev[b] / 4};
}

__device__ __forceinline__ void lw_sum_round(LwSweepShared &S, const LwChain &chain, int number, const LwRound &prev) {
  __syncthreads();
  if (threadIdx.x >= 256) {
    if (number > 0) lw_band_terms(S, number - 1, prev);
    return;
  }
  const float4 *v = chain.v + (number & 1) * (kLwRows * kLwRowStride / 4);
  float sum = 0.0f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (q < chain.quads) {
      const float4 x = v[q];
      sum = sum + x.x;
      sum = sum + x.y;
      sum = sum + x.z;
      sum = sum + x.w;
    }
  }
  chain.sum[(number & 1) * (kLwRows * (kLwBands + 1))] = sum;
}

// Block = kLwSweepCols consecutive columns of the chunk.  Threads without a
// column of their own (padding threads, a column past the chunk or the live
// count) only take the barriers and their part of the sums.
// Bound by instruction issue and the latency of record loads and table gathers.
// 425 x 425 x 50 (180,625 columns of 63 layers): 27.6 ms before the cloud's
// exponential moved to the layer kernel, the upward pass reused the downward
// pass's table positions, and the sums took 16-byte reads of padded bands with
// one barrier in four levels (before, three in eight and 4-byte reads): 22.4 ms;
// with four levels unrolled (no register moves of the layer loaded ahead) and
// records addressed by 32-bit offsets from the block's first: 20.6 ms.  At 5
// blocks per SM (40 registers) 21.9 ms.
// kSmall: the small-chunk form, which reads every layer's transfer terms from
// the term records instead of forming them (lw_small_terms_kernel).
template <bool kSmall>
__global__ void __launch_bounds__(kLwSweepThreads, kSmall ? 1 : kLwSweepMinBlocks) lw_sweep_kernel(Tables T, LwArgs a) {
  __shared__ __align__(16) LwSweepShared S;
  const int lc0 = blockIdx.x * kLwSweepCols;
  if (lc0 >= a.chunk_count || dead_column(a.live, a.chunk_first + lc0)) return;  // whole block
  if (lw_small(a, lw_chunk_columns(a)) != kSmall) return;                         // the other form's
  const int tid = threadIdx.x;
  const bool slot = tid < kLwSweepCols * kLwGpts;
  const int cslot = slot ? tid / kLwGpts : kLwSweepCols - 1;
  const int G = slot ? tid - cslot * kLwGpts : kLwGpts - 1;
  const int lc = lc0 + cslot;
  const bool live = slot && lc < a.chunk_count && !dead_column(a.live, a.chunk_first + lc);
  const int col = a.chunk_first + lc;
  int band = kLwBands - 1;
  while (G < kGofsDev[band]) --band;
  const int P = kLwPadOfsDev[band] + (G - kGofsDev[band]);
  const ColRec &R = col_records(a)[live ? lc : lc0];
  const float sd = R.secdiff[band];
  const int nlay = a.nlay, nk = a.nk;
  const uint32_t bit = 1u << (G & 31);
  const float pi = 3.1415926535897932384626433832795f;
  const float fluxfac = pi * 2.0e4f;
  for (int q = tid; q < 2 * kLwRows * kLwRowStride; q += kLwSweepThreads) (&S.ring[0][0][0])[q] = 0.0f;
  if (tid < kLwSweepCols * 2) S.flux[tid >> 1][2 + (tid & 1)][nlay] = 0.0f * fluxfac;  // no downward flux at the top
  bool has_cloud = false;
  if (live) {
#pragma unroll
    for (int w = 0; w < kMaxLay / 32; ++w) {
      const uint32_t word = 32 * w < nlay ? R.cloud[w] : 0u;
      has_cloud = has_cloud || word != 0u;
      if (G == 0) S.cloud[cslot][w] = word;
    }
  }
  __syncthreads();
  const LwChain chain = lw_chain(S);
  // this thread's radiances in the ring: row (level * 2 + total / clear) * columns + column
  float *const ring0 = &S.ring[0][cslot][P];
  constexpr int kTypeStep = kLwSweepCols * kLwRowStride, kBufStep = kLwRows * kLwRowStride;
  auto put = [&](int number, int filled, float total, float clear) {
    float *q = ring0 + (number & 1) * kBufStep + filled * (2 * kTypeStep);
    q[0] = total;
    q[kTypeStep] = clear;
  };
  // the block's layer records, addressed from one base by 32-bit byte offsets
  char *const base = reinterpret_cast<char *>(layer_records(a) + static_cast<size_t>(lc0) * nlay * kLwRec);
  constexpr uint32_t kStep = kLwRec * sizeof(float);
  const uint32_t column = static_cast<uint32_t>(cslot * nlay) * kStep;
  const uint32_t off_tau = column + 4u * P, off_band = column + 4u * (kLwRecBand + 4 * band);
  const uint32_t off_efcl = column + 4u * (kLwRecEfcl + band), off_mask = column + 4u * (kLwRecMask + (G >> 5));
  auto at = [&](uint32_t off) -> float & { return *reinterpret_cast<float *>(base + off); };
  struct Next {
    float tg, fr, efcl;
    float4 bq;
    uint32_t word;
    bool cloudy;
  } nx{};
  auto load = [&](int l) {
    const uint32_t step = static_cast<uint32_t>(l) * kStep;
    nx.tg = at(off_tau + step);
    nx.fr = at(off_tau + step + 4 * kLwRecFracs);
    nx.bq = *reinterpret_cast<const float4 *>(base + off_band + step);
    nx.cloudy = (S.cloud[cslot][l >> 5] >> (l & 31)) & 1u;
    if (nx.cloudy) {
      nx.efcl = at(off_efcl + step);
      nx.word = __float_as_uint(at(off_mask + step));
    }
  };

  // surface emission and reflection (surface_sums, lw:5648-5655)
  auto surface = [&](float fr, float &total, float &clear) {
    const float bt = R.C.tsfc - 159.0f;
    const int indbound = clampi(static_cast<int>(bt), 1, 180);
    const float tbndfrac = bt - static_cast<float>(indbound);
    const float reflect = 1.0f - R.C.semiss;
    const float plankbnd = R.C.semiss * planck(T, indbound, tbndfrac, band);
    const float rad0 = fr * plankbnd;
    total = rad0 + reflect * total;
    clear = rad0 + reflect * clear;
  };
  float rA = 0.0f, rB = 0.0f;
  bool iclddn = false;
  int number = 0;
  LwRound prev{0, 2, nlay - 1, -1};
  if constexpr (kSmall) {
    // the layers' terms four ahead; layer l gives level l downward, l + 1 upward
    const LwTerms *terms = lw_terms(a, live ? lc : lc0, 0) + G;
    auto fetch = [&](int l) { return terms[static_cast<size_t>(l) * kLwGpts]; };
    auto cloudy_at = [&](int l) { return ((S.cloud[cslot][l >> 5] >> (l & 31)) & 1u) != 0u; };
    LwTerms ahead[kLwRing];
    LwRound round = prev;
    if (live) {
#pragma unroll
      for (int j = 0; j < kLwRing; ++j)
        if (nlay - 1 - j >= 0) ahead[j] = fetch(nlay - 1 - j);
    }
    for (int l0 = nlay - 1; l0 >= 0; l0 -= kLwRing) {
      if (live) {
        LwTerms cur[kLwRing];
#pragma unroll
        for (int j = 0; j < kLwRing; ++j) {
          cur[j] = ahead[j];
          if (l0 - kLwRing - j >= 0) ahead[j] = fetch(l0 - kLwRing - j);
        }
#pragma unroll
        for (int j = 0; j < kLwRing; ++j) {
          const int l = l0 - j;
          if (l < 0) break;
          const LwTerms &t = cur[j];
          const bool cloudy = cloudy_at(l);
          iclddn = iclddn || cloudy;
          const float rn = cloudy ? rA - rA * t.atot + t.srcd + (t.totd - t.srcd) : rA + (t.bbd - rA) * t.a;
          rB = iclddn ? rB + (t.bbd - rB) * t.a : rn;
          rA = rn;
          put(number, j, rA, rB);
        }
      }
      round.count = l0 + 1 < kLwRing ? l0 + 1 : kLwRing;
      lw_sum_round(S, chain, number, prev);
      prev = round;
      round.level0 -= kLwRing;
      ++number;
    }
    round = LwRound{0, 0, 0, 1};
    if (live) {
      surface(at(off_tau + 4 * kLwRecFracs), rA, rB);
#pragma unroll
      for (int j = 0; j < kLwRing; ++j)
        if (j < nlay) ahead[j] = fetch(j);
    }
    // level 0, then layer l0 - 1 + j at place j of the following rounds
    for (int l0 = 0; l0 <= nlay; l0 += kLwRing) {
      if (live) {
        LwTerms cur[kLwRing];
#pragma unroll
        for (int j = 0; j < kLwRing; ++j) {
          const int l = l0 - 1 + j;  // its terms are ahead[l mod 4]
          if (l >= 0 && l < nlay) {
            cur[j] = ahead[(j + kLwRing - 1) % kLwRing];
            if (l + kLwRing < nlay) ahead[(j + kLwRing - 1) % kLwRing] = fetch(l + kLwRing);
          }
        }
#pragma unroll
        for (int j = 0; j < kLwRing; ++j) {
          const int l = l0 - 1 + j;
          if (l >= nlay) break;
          if (l >= 0) {
            const LwTerms &t = cur[j];
            const float rn =
                cloudy_at(l) ? rA - rA * t.atot + t.srcu + (t.totu - t.srcu) : rA + (t.bbu - rA) * t.a;
            rB = has_cloud ? rB + (t.bbu - rB) * t.a : rn;
            rA = rn;
          }
          put(number, j, rA, rB);
        }
      }
      round.count = nlay + 1 - l0 < kLwRing ? nlay + 1 - l0 : kLwRing;
      lw_sum_round(S, chain, number, prev);
      prev = round;
      round.level0 += kLwRing;
      ++number;
    }
  } else {
    // downward sweep, top to bottom: layer l gives level l; next layer loaded ahead
    LwRound round = prev;
    if (live) load(nlay - 1);
    for (int l0 = nlay - 1; l0 >= 0; l0 -= kLwRing) {
      if (live) {
#pragma unroll
        for (int j = 0; j < kLwRing; ++j) {
          const int l = l0 - j;
          if (l < 0) break;
          const Next cur = nx;
          if (l > 0) load(l - 1);
          iclddn = iclddn || cur.cloudy;
          const uint32_t up = lw_down(T, cur.tg, cur.fr, cur.bq, cur.efcl, (cur.word & bit) != 0u, cur.cloudy, sd, rA,
                                      rB, iclddn);
          at(off_tau + static_cast<uint32_t>(l) * kStep) = __uint_as_float(up);
          put(number, j, rA, rB);
        }
      }
      round.count = l0 + 1 < kLwRing ? l0 + 1 : kLwRing;
      lw_sum_round(S, chain, number, prev);
      prev = round;
      round.level0 -= kLwRing;
      ++number;
    }
    // upward sweep, bottom to top: level 0 from the surface, then layer l gives level l + 1
    round = LwRound{0, 0, 0, 1};
    for (int l0 = 0; l0 <= nlay; l0 += kLwRing) {
      if (live) {
#pragma unroll
        for (int j = 0; j < kLwRing; ++j) {
          const int level = l0 + j;
          if (level > nlay) break;
          if (j == 0 && level == 0) {
            load(0);
            surface(nx.fr, rA, rB);
          } else {
            const Next cur = nx;
            if (level < nlay) load(level);
            lw_up(T, __float_as_uint(cur.tg), cur.fr, cur.bq, cur.efcl, (cur.word & bit) != 0u, cur.cloudy, rA, rB,
                  has_cloud);
          }
          put(number, j, rA, rB);
        }
      }
      round.count = nlay + 1 - l0 < kLwRing ? nlay + 1 - l0 : kLwRing;
      lw_sum_round(S, chain, number, prev);
      prev = round;
      round.level0 += kLwRing;
      ++number;
    }
  }
  __syncthreads();
  if (tid >= 256) lw_band_terms(S, number - 1, prev);
  __syncthreads();

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
  if (G == 0 && live) {
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
  const size_t small = chunk <= kSmallColumns ? (chunk < kLwSmallColumns ? chunk : kLwSmallColumns) : 0;
  return (kColRecFloats + (static_cast<size_t>(kLwGasFields) + kLwRec) * nlay) * static_cast<size_t>(chunk) +
         small * nlay * kLwTermFloats;
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
  // a live count may leave few columns: a bounded grid walks those there are
  // (2,048 slots with a few hundred live: 54 us when every block of the
  // capacity was launched to find itself dead; 1,000,000-column inference
  // 2.84 ms before, 2.80 ms with this and the same in sw_optics_kernel)
  const unsigned gas = blocks * kLwBands, most = a.live ? 148u * kLwGasMinBlocks * 2u : gas;
  lw_gas_kernel<<<gas < most ? gas : most, threads, 0, stream>>>(T, a);
  return cudaGetLastError();
}

cudaError_t launch_lw_chunk_sweep(const Tables &T, const LwArgs &a, cudaStream_t stream) {
  if (a.chunk_capacity <= kSmallColumns && (a.live || a.chunk_count <= kLwSmallColumns)) {
    const int most = a.chunk_count < kLwSmallColumns ? a.chunk_count : kLwSmallColumns;
    const int items = most * a.nlay;
    lw_small_terms_kernel<<<items < kSmallBlocks ? items : kSmallBlocks, kLwTermThreads, 0, stream>>>(T, a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    lw_sweep_kernel<true><<<(most + kLwSweepCols - 1) / kLwSweepCols, kLwSweepThreads, 0, stream>>>(T, a);
    e = cudaGetLastError();
    if (e != cudaSuccess || a.chunk_count <= kLwSmallColumns) return e;
  }
  lw_sweep_kernel<false><<<(a.chunk_count + kLwSweepCols - 1) / kLwSweepCols, kLwSweepThreads, 0, stream>>>(T, a);
  return cudaGetLastError();
}

}  // namespace rrtmg
