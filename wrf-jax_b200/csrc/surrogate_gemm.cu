// BF16 GEMM on the 5th-generation tensor cores (tcgen05) with fused MLP
// epilogues, for the radiation surrogate's training and inference.
//
//   C[M x N] = A[M x K] * B[N x K]^T      (A, B row-major BF16, FP32 accumulate)
//
// One CTA of 256 threads owns a 128 x BN output tile (BN = 128; 64 where that
// leaves SMs idle; 256 on request).  Its accumulator lives in tensor memory (128 lanes x BN FP32
// columns).  K advances in blocks of 64: all threads copy the A and B blocks
// into shared memory (cp.async, three stages) in the 128-byte swizzled
// K-major layout, and one thread issues four tcgen05.mma (K = 16 each)
// whose completion is committed to the stage's mbarrier before the stage is
// refilled.  With BN <= 128 two CTAs share an SM, one's epilogue under the
// other's loads and MMAs.  The epilogue reads the accumulator back with
// tcgen05.ld (warp w owns tile rows 32 (w mod 4) .. and column half w / 4), 32
// columns at a time, and passes them through a shared stage of the warp's own
// so that every global access is a run of whole sectors along a row:
//   kEpiF32    C (+ bias) as FP32, one slab per K split (split-K partials)
//   kEpiGelu   Z = acc + bias (FP32), H = GELU(Z) as BF16 row-major and
//              transposed (the transposed copy feeds the weight gradient)
//   kEpiDgelu  dZ = acc * GELU'(aux) as BF16 row-major and transposed
// Bound by the epilogue's traffic at the surrogate's shapes (K = 512).
//
// Shared-memory layout of an operand block (R rows x 64 K, BF16): the
// canonical K-major SWIZZLE_128B layout, row r at r * 128 bytes with its eight
// 16-byte chunks permuted by XOR with r mod 8, 8-row groups 1024 bytes apart;
// each block stage starts on a 1024-byte boundary.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "surrogate_kernels.h"
#include "umma_common.cuh"

namespace rrtmg {
namespace {

using umma::gelu;
using umma::gelu_grad;
using umma::mbar_wait;
using umma::smem_desc;
using umma::smem_u32;
using umma::swz;

constexpr int kBM = 128, kBK = 64;
constexpr int kThreads = 256;

// The epilogue's stages (EpiStage of each warp) lie over the pipeline's.
constexpr int kEpiBytes = (32 * 36 * 4 + 2 * 32 * 40 * 2) * (kThreads / 32);

template <int BN>
struct Tile {
  static constexpr int kStages = 3;
  static constexpr int kBytesA = kBM * kBK * 2;
  static constexpr int kBytesB = BN * kBK * 2;
  static constexpr int kStageBytes = kBytesA + kBytesB;
  // one extra KB so the stages can start on a 1024-byte boundary
  static constexpr int kSmemBytes = (BN == 64 ? kEpiBytes : kStages * kStageBytes) + 1024;
  static constexpr uint32_t kIdesc = umma::idesc_bf16(kBM, BN);
};

// A warp's stage of the epilogue, over the pipeline's shared memory: 32 rows x
// 32 FP32 values, and the BF16 results by rows and by columns.  Row pitches are
// odd numbers of 16 bytes, so that neither side of the transposition conflicts.
constexpr int kEpiCols = 32;
struct EpiStage {
  float z[32][36];
  __nv_bfloat16 h[32][40];
  __nv_bfloat16 ht[kEpiCols][40];
};
static_assert(sizeof(EpiStage) * (kThreads / 32) == kEpiBytes && kEpiBytes <= 3 * Tile<128>::kStageBytes &&
                  kEpiBytes >= 3 * Tile<64>::kStageBytes, "stages of the epilogue");

__device__ unsigned g_gemm_error;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}

// One tile: m-tile `my`, n-tile `nx`, K split `z` of problem g (its K blocks
// are dealt to the splits as evenly as they go).  The n-tiles of one m-tile are
// neighbouring CTAs, so they share the A rows in L2.
// K blocks stream through kStages shared-memory stages: the copies of block
// kb + kStages - 1 are in flight while the tensor cores work on block kb.
template <int BN>
__device__ __forceinline__ void gemm_tile(const GemmArgs &g, int nx, int my, int z) {
  using TL = Tile<BN>;
  constexpr int S = TL::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t mbar[S];
  __shared__ uint32_t tmem_sh;
  __shared__ int fail_sh;
  __shared__ __align__(16) float bias_sh[BN];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = nx * BN, m0 = my * kBM;
  const int blocks = g.K / kBK;
  const int kb0 = static_cast<int>(static_cast<long long>(blocks) * z / g.ksplit);
  const int kbeg = kb0 * kBK;
  const int nkb = static_cast<int>(static_cast<long long>(blocks) * (z + 1) / g.ksplit) - kb0;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                 "r"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < S; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[s])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_sh = 0;
  }
  for (int j = tid; j < BN; j += kThreads) bias_sh[j] = g.bias && z == 0 ? g.bias[n0 + j] : 0.0f;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_sh;

  uint8_t *tiles = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
  auto stage_a = [&](int s) { return tiles + s * TL::kStageBytes; };
  auto stage_b = [&](int s) { return tiles + s * TL::kStageBytes + TL::kBytesA; };
  auto load = [&](int kb, int s) {
    const int k0 = kbeg + kb * kBK;
    uint8_t *a = stage_a(s), *b = stage_b(s);
    // 8 consecutive threads copy one 128-byte row: coalesced global reads and
    // conflict-free swizzled shared-memory writes
#pragma unroll
    for (int i = 0; i < (kBM * kBK / 8) / kThreads; ++i) {
      const int q = tid + i * kThreads;
      const int r = q >> 3, kc = q & 7;
      cp_async16(a + swz(r, kc), g.A + static_cast<size_t>(m0 + r) * g.lda + k0 + kc * 8);
    }
#pragma unroll
    for (int i = 0; i < (BN * kBK / 8) / kThreads; ++i) {
      const int q = tid + i * kThreads;
      const int r = q >> 3, kc = q & 7;
      cp_async16(b + swz(r, kc), g.B + static_cast<size_t>(n0 + r) * g.ldb + k0 + kc * 8);
    }
  };

  // prologue: blocks 0 .. S-2, one commit group each (empty groups keep the count)
#pragma unroll
  for (int s = 0; s < S - 1; ++s) {
    if (s < nkb) load(s, s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  bool ok = true;
  int issued = 0;
  for (int kb = 0; kb < nkb; ++kb) {
    const int s = kb % S;
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    // make the generic-proxy shared-memory writes visible to the tensor cores
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t abase = smem_u32(stage_a(s)), bbase = smem_u32(stage_b(s));
#pragma unroll
      for (int kk = 0; kk < kBK / 16; ++kk) {
        const uint64_t adesc = smem_desc(abase + kk * 32);
        const uint64_t bdesc = smem_desc(bbase + kk * 32);
        const uint32_t accumulate = (kb > 0 || kk > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            :
            : "r"(tmem), "l"(adesc), "l"(bdesc), "r"(TL::kIdesc), "r"(accumulate)
            : "memory");
      }
      // (the failure-detection test withholds block 0's commit: the wait for it
      // below runs out, and block 1's commit, which covers every earlier MMA,
      // still lets the CTA drain before it frees its tensor memory)
      if (!(g.withhold_commit0 && kb == 0))
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&mbar[s]))
                     : "memory");
    }
    issued = kb + 1;
    const int next = kb + S - 1;
    if (next < nkb) {
      // stage next % S was last read by the MMAs of block kb - 1
      if (kb >= 1 && !mbar_wait(smem_u32(&mbar[(kb - 1) % S]), static_cast<uint32_t>((kb - 1) / S) & 1u, g.wait_ns))
        ok = false;
      if (__syncthreads_or(!ok)) {
        if (tid == 0) fail_sh = 1;
        break;
      }
      load(next, next % S);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // wait for the last committed group (it covers every earlier MMA) before
  // the tensor memory is freed; this drain keeps the default limit even when
  // the pipeline waits above run with a shorter one
  if (issued > 0) {
    const int last = issued - 1;
    if (tid == 0 && !mbar_wait(smem_u32(&mbar[last % S]), static_cast<uint32_t>(last / S) & 1u)) fail_sh = 1;
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const bool failed = fail_sh != 0 || issued != nkb;
  if (failed) {
    if (tid == 0) atomicOr(&g_gemm_error, 1u);
  } else {
    // rows r0 .. r0 + 31 of the output, columns n0 + c .. of the warp's half
    const int r0 = m0 + (warp & 3) * 32;
    const uint32_t trow = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    EpiStage &st = reinterpret_cast<EpiStage *>(tiles)[warp];
    const int zr = lane >> 3, zc = (lane & 7) * 4;  // a row's 32 FP32 values: 8 lanes
    const int hr = lane >> 2, hc = (lane & 3) * 8;  // 32 BF16 values: 4 lanes
    const bool ht_rows = (g.ldht % 8) == 0 && (reinterpret_cast<uintptr_t>(g.Ht) & 15u) == 0;
    auto put_rows = [&](float *dst, size_t ld) {  // the FP32 stage to rows of dst
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4 *>(dst + static_cast<size_t>(r0 + 4 * i + zr) * ld + zc) =
            *reinterpret_cast<const float4 *>(&st.z[4 * i + zr][zc]);
    };
#pragma unroll 1
    for (int c = (warp >> 2) * (BN / 2); c < (warp >> 2) * (BN / 2) + BN / 2; c += kEpiCols) {
      const int nc = n0 + c;
      __syncwarp();  // the stage's previous readers are done
      if (g.epi == kEpiDgelu) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float4 *>(&st.z[4 * i + zr][zc]) = *reinterpret_cast<const float4 *>(
              g.aux + static_cast<size_t>(r0 + 4 * i + zr) * g.ldaux + nc + zc);
        __syncwarp();
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[16];
        umma::tmem_ld16(trow + static_cast<uint32_t>(c + 16 * half), v);
        umma::tmem_ld_wait();
        float acc[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] = __uint_as_float(v[j]);
        float4 *zs = reinterpret_cast<float4 *>(&st.z[lane][16 * half]);
        __align__(16) __nv_bfloat16 h[16];
        if (g.epi == kEpiDgelu) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 zz = zs[q];
            h[4 * q + 0] = __float2bfloat16_rn(acc[4 * q + 0] * gelu_grad(zz.x));
            h[4 * q + 1] = __float2bfloat16_rn(acc[4 * q + 1] * gelu_grad(zz.y));
            h[4 * q + 2] = __float2bfloat16_rn(acc[4 * q + 2] * gelu_grad(zz.z));
            h[4 * q + 3] = __float2bfloat16_rn(acc[4 * q + 3] * gelu_grad(zz.w));
          }
        } else {
          // (a split's partial sums take no bias: bias_sh is zero there)
          const float4 *b4 = reinterpret_cast<const float4 *>(bias_sh + c + 16 * half);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 b = b4[q];
            if (g.bias) {
              acc[4 * q] += b.x;
              acc[4 * q + 1] += b.y;
              acc[4 * q + 2] += b.z;
              acc[4 * q + 3] += b.w;
            }
            zs[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
          }
          if (g.epi == kEpiF32) continue;
#pragma unroll
          for (int j = 0; j < 16; ++j) h[j] = __float2bfloat16_rn(gelu(acc[j]));
        }
        uint4 *hs = reinterpret_cast<uint4 *>(&st.h[lane][16 * half]);
        hs[0] = *reinterpret_cast<const uint4 *>(&h[0]);
        hs[1] = *reinterpret_cast<const uint4 *>(&h[8]);
        if (g.Ht) {
#pragma unroll
          for (int j = 0; j < 16; ++j) st.ht[16 * half + j][lane] = h[j];
        }
      }
      if (g.epi == kEpiF32) {
        put_rows(g.C + static_cast<size_t>(z) * g.split_stride + nc, g.ldc);
        continue;
      }
      if (g.epi == kEpiGelu && g.Z) put_rows(g.Z + nc, g.ldz);
      __syncwarp();
      if (g.H) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4 *>(g.H + static_cast<size_t>(r0 + 8 * i + hr) * g.ldh + nc + hc) =
              *reinterpret_cast<const uint4 *>(&st.h[8 * i + hr][hc]);
      }
      if (g.Ht && ht_rows) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4 *>(g.Ht + static_cast<size_t>(nc + 8 * i + hr) * g.ldht + r0 + hc) =
              *reinterpret_cast<const uint4 *>(&st.ht[8 * i + hr][hc]);
      } else if (g.Ht) {
        for (int j = 0; j < kEpiCols; ++j)
          g.Ht[static_cast<size_t>(nc + j) * g.ldht + r0 + lane] = st.ht[j][lane];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
  }
}

template <int BN>
__global__ void __launch_bounds__(kThreads, BN == 256 ? 1 : 2) umma_gemm_kernel(const __grid_constant__ GemmArgs g) {
  gemm_tile<BN>(g, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Several problems in one launch (their K split and tile shape are common): the
// weight gradients of a training step, each too small to fill the GPU alone.
struct GemmGroup {
  GemmArgs g[kGemmGroup];
  int first[kGemmGroup + 1];  // first tile of each problem
};

__global__ void __launch_bounds__(kThreads, 1) umma_gemm_group_kernel(const __grid_constant__ GemmGroup p) {
  int q = 0;
  while (q + 1 < kGemmGroup && static_cast<int>(blockIdx.x) >= p.first[q + 1]) ++q;
  const GemmArgs &g = p.g[q];
  const int tile = blockIdx.x - p.first[q], nt = g.N / 256;
  gemm_tile<256>(g, tile % nt, tile / nt, blockIdx.y);
}

// Opts a kernel in to its shared memory, once per device (a bit of `done` each).
template <class Kernel>
cudaError_t raise_smem(Kernel kernel, int bytes, std::atomic<unsigned long long> &done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && ((done.load() >> dev) & 1ull)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev);
  return e;
}

template <int BN>
cudaError_t launch_tile(const GemmArgs &g, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = raise_smem(umma_gemm_kernel<BN>, Tile<BN>::kSmemBytes, configured);
  if (e != cudaSuccess) return e;
  dim3 grid(g.N / BN, g.M / kBM, g.ksplit);
  umma_gemm_kernel<BN><<<grid, kThreads, Tile<BN>::kSmemBytes, stream>>>(g);
  return cudaGetLastError();
}

}  // namespace

namespace {
// 0 automatic (64 or 128: two CTAs per SM), else 128 or 256
int g_tile_choice = 0;
// Up to this many 128-wide tiles, twice as many 64-wide ones are used: they
// still find an SM each, and a tile's epilogue, most of its time, is half as
// long.  Training step of 1,024 columns (32 tiles per layer) 117 us with
// 128-wide tiles, 104 us with 64; 2,048 (64 tiles) 128 and 111 us; 3,072 (96
// tiles) 135 and 139 us.
constexpr long long kNarrowTiles = 74;
}  // namespace

void set_gemm_tile(int bn) { g_tile_choice = bn; }

bool gemm_wide(int n) { return n % 256 == 0 && g_tile_choice == 256; }

int gemm_stages(int n) { return gemm_wide(n) ? Tile<256>::kStages : Tile<128>::kStages; }

cudaError_t launch_umma_gemm(const GemmArgs &g, cudaStream_t stream) {
  if (gemm_wide(g.N)) return launch_tile<256>(g, stream);
  const long long tiles = static_cast<long long>(g.N / 128) * (g.M / kBM) * g.ksplit;
  if (g_tile_choice == 0 && tiles <= kNarrowTiles) return launch_tile<64>(g, stream);
  return launch_tile<128>(g, stream);
}

cudaError_t launch_umma_gemm_group(const GemmArgs *g, int count, cudaStream_t stream) {
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = raise_smem(umma_gemm_group_kernel, Tile<256>::kSmemBytes, configured);
  if (e != cudaSuccess) return e;
  GemmGroup p{};
  int tiles = 0;
  for (int q = 0; q < kGemmGroup; ++q) {
    p.first[q] = tiles;
    if (q < count) {
      p.g[q] = g[q];
      tiles += (g[q].M / kBM) * (g[q].N / 256);
    }
  }
  p.first[kGemmGroup] = tiles;
  umma_gemm_group_kernel<<<dim3(tiles, g[0].ksplit), kThreads, Tile<256>::kSmemBytes, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t gemm_error_flag(unsigned *out, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_gemm_error, sizeof(unsigned));
  if (e != cudaSuccess || !reset) return e;
  const unsigned zero = 0;
  return cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof(unsigned));
}

}  // namespace rrtmg
