// C-ABI of the surrogate kernels.  See include/rrtmg_surrogate.h.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "../../include/rrtmg_surrogate.h"
#include "surrogate_kernels.h"

using namespace rrtmg;

namespace {
bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

constexpr unsigned long long kDefaultWaitNs = 2000000000ull;  // 2 s
std::atomic<unsigned long long> g_wait_ns{kDefaultWaitNs};
std::atomic<int> g_withhold_commit{0};
}  // namespace

extern "C" rrtmg_status rrtmg_gemm_bf16(const rrtmg_gemm_args *a, void *stream) {
  if (!a || !a->A || !a->B) return RRTMG_BAD_ARG;
  if (a->M <= 0 || a->N <= 0 || a->K <= 0 || a->ksplit <= 0) return RRTMG_BAD_ARG;
  if (a->M % 128 || a->N % 128 || a->K % (64 * a->ksplit)) return RRTMG_BAD_ARG;
  if (a->lda % 8 || a->ldb % 8 || a->lda < a->K || a->ldb < a->K) return RRTMG_BAD_ARG;
  if (!aligned16(a->A) || !aligned16(a->B)) return RRTMG_BAD_ARG;
  // the epilogue stores 16-byte vectors along rows
  if ((a->C && (!aligned16(a->C) || a->ldc % 4 || a->split_stride % 4)) || (a->Z && (!aligned16(a->Z) || a->ldz % 4)) ||
      (a->aux && (!aligned16(a->aux) || a->ldaux % 4)) || (a->H && (!aligned16(a->H) || a->ldh % 8)))
    return RRTMG_BAD_ARG;
  switch (a->epilogue) {
    case RRTMG_EPI_F32:
      if (!a->C || a->ldc < a->N) return RRTMG_BAD_ARG;
      if (a->ksplit > 1 && a->split_stride < static_cast<size_t>(a->M) * a->ldc) return RRTMG_BAD_ARG;
      break;
    case RRTMG_EPI_GELU:
      if (a->ksplit != 1) return RRTMG_BAD_ARG;
      if ((a->Z && a->ldz < a->N) || (a->H && a->ldh < a->N) || (a->Ht && a->ldht < a->M)) return RRTMG_BAD_ARG;
      break;
    case RRTMG_EPI_DGELU:
      if (a->ksplit != 1 || !a->aux || a->ldaux < a->N) return RRTMG_BAD_ARG;
      if ((a->H && a->ldh < a->N) || (a->Ht && a->ldht < a->M)) return RRTMG_BAD_ARG;
      break;
    default:
      return RRTMG_BAD_ARG;
  }
  GemmArgs g{};
  g.A = static_cast<const __nv_bfloat16 *>(a->A);
  g.lda = a->lda;
  g.B = static_cast<const __nv_bfloat16 *>(a->B);
  g.ldb = a->ldb;
  g.M = a->M; g.N = a->N; g.K = a->K; g.ksplit = a->ksplit; g.epi = a->epilogue;
  g.bias = a->bias;
  g.C = a->C; g.ldc = a->ldc; g.split_stride = a->split_stride;
  g.H = static_cast<__nv_bfloat16 *>(a->H); g.ldh = a->ldh;
  g.Ht = static_cast<__nv_bfloat16 *>(a->Ht); g.ldht = a->ldht;
  g.aux = a->aux; g.ldaux = a->ldaux;
  g.Z = a->Z; g.ldz = a->ldz;
  g.wait_ns = g_wait_ns.load();
  g.withhold_commit0 = g_withhold_commit.load();
  // the hook needs a later commit to drain behind the withheld one and a wait
  // on the withheld one inside the K loop: more K blocks than stages
  if (g.withhold_commit0 && a->K / (64 * a->ksplit) <= gemm_stages(a->N)) return RRTMG_BAD_ARG;
  return launch_umma_gemm(g, static_cast<cudaStream_t>(stream)) == cudaSuccess ? RRTMG_OK : RRTMG_CUDA;
}

extern "C" rrtmg_status rrtmg_gemm_error(int reset, unsigned *flag) {
  if (!flag) return RRTMG_BAD_ARG;
  unsigned g = 0, m = 0;
  if (gemm_error_flag(&g, reset != 0) != cudaSuccess || mlp_error_flag(&m, reset != 0) != cudaSuccess)
    return RRTMG_CUDA;
  *flag = g | m;
  return *flag ? RRTMG_TIMEOUT : RRTMG_OK;
}

extern "C" rrtmg_status rrtmg_gemm_set_wait_ns(unsigned long long wait_ns) {
  g_wait_ns.store(wait_ns ? wait_ns : kDefaultWaitNs);
  return RRTMG_OK;
}

extern "C" rrtmg_status rrtmg_gemm_test_withhold_commit(int enable) {
  g_withhold_commit.store(enable != 0);
  return RRTMG_OK;
}

namespace {
rrtmg_status cuda_status(cudaError_t e) { return e == cudaSuccess ? RRTMG_OK : RRTMG_CUDA; }

// A pointer the kernels may dereference: device memory, managed memory, or
// page-locked host memory mapped at the same address (unified addressing).
bool device_reachable(const void *p) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();  // clear the sticky error of an unknown pointer
    return false;
  }
  if (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged) return true;
  return at.type == cudaMemoryTypeHost && at.devicePointer == p;
}
cudaStream_t as_stream(void *s) { return static_cast<cudaStream_t>(s); }
}  // namespace

extern "C" rrtmg_status rrtmg_sur_features(const rrtmg_sur_features_args *a, void *stream) {
  if (!a || a->ncol < 0 || a->nk <= 0 || a->ny <= 0 || a->row_offset < 0) return RRTMG_BAD_ARG;
  if (!a->p3d || !a->p8w || !a->t3d || !a->qv || !a->qc || !a->qi || !a->qs || !a->cldfra || !a->o3 || !a->tsk ||
      !a->albedo || !a->coszr || !a->emiss)
    return RRTMG_BAD_ARG;
  const int nf = 9 * a->nk + 4;
  if (a->raw && a->ldf < nf) return RRTMG_BAD_ARG;
  if (a->X && (a->ldx < nf || !a->mean || !a->rstd)) return RRTMG_BAD_ARG;
  if (a->Xt && (!a->X || a->ldxt < a->row_offset + a->ncol)) return RRTMG_BAD_ARG;
  if (a->x_layout != 0 && (a->x_layout != 1 || !a->X || a->ldx != 512 || !aligned16(a->X) || a->raw || a->Xt ||
                           9 * a->nk + 4 > 512))
    return RRTMG_BAD_ARG;
  if ((a->lo == nullptr) != (a->hi == nullptr)) return RRTMG_BAD_ARG;
  if (a->ncol == 0) return RRTMG_OK;
  return cuda_status(launch_sur_features(*a, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_targets(const rrtmg_sur_targets_args *a, void *stream) {
  if (!a || a->ncol < 0 || a->nk <= 0 || a->ny <= 0 || a->row_offset < 0 || !a->T || a->ldt < 2 * a->nk + 6)
    return RRTMG_BAD_ARG;
  if (!a->rthratenlw || !a->rthratensw || !a->pi3d || !a->p8w || !a->glw || !a->lwupb || !a->swdnb || !a->swupb)
    return RRTMG_BAD_ARG;
  if (a->ncol == 0) return RRTMG_OK;
  return cuda_status(launch_sur_targets(*a, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_column_stats(const float *F, int n, int ld, int nf, float *mean, float *rstd,
                                               float *lo, float *hi, void *stream) {
  if (!F || n <= 0 || nf <= 0 || ld < nf || !mean || !rstd) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_column_stats(F, n, ld, nf, mean, rstd, lo, hi, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_gather(const void *X, int ldx, const float *T, int ldt, const int *idx, int B,
                                         void *Xb, void *Xbt, int ldxbt, float *Tb, void *stream) {
  if (!X || !idx || B <= 0 || ldx <= 0 || !Xb || !Xbt || ldxbt < B || (Tb && (!T || ldt <= 0))) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_gather(static_cast<const __nv_bfloat16 *>(X), ldx, T, ldt, idx, B,
                                       static_cast<__nv_bfloat16 *>(Xb), static_cast<__nv_bfloat16 *>(Xbt), ldxbt,
                                       Tb, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_loss_grad(const float *Y, const float *T, const float *w, int B, int ld,
                                            float scale, void *dY, void *dYt, int lddyt, float *loss, void *stream) {
  if (!Y || !T || !w || B <= 0 || ld <= 0 || !dY || !dYt || lddyt < B) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_loss_grad(Y, T, w, B, ld, scale, static_cast<__nv_bfloat16 *>(dY),
                                          static_cast<__nv_bfloat16 *>(dYt), lddyt, loss, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_row_sum(const void *Gt, int ld, int rows, int B, float *db, void *stream) {
  if (!Gt || !db || rows <= 0 || B <= 0 || ld < B) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_row_sum(static_cast<const __nv_bfloat16 *>(Gt), ld, rows, B, db, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_reduce_splits(const float *P, int splits, size_t n, float *G, void *stream) {
  if (!P || !G || splits <= 0 || n == 0) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_reduce_splits(P, splits, n, G, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_adam(const rrtmg_sur_adam_args *a, void *stream) {
  if (!a || a->rows <= 0 || a->cols <= 0 || !a->w || !a->m || !a->v || !a->grad) return RRTMG_BAD_ARG;
  if ((a->wb && a->ldwb < a->cols) || (a->wbt && a->ldwbt < a->rows)) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_adam(*a, as_stream(stream)));
}

// ---------------------------------------------------------------------------
// training step
// ---------------------------------------------------------------------------
namespace {

constexpr int kTrainLayers = 4, kTrainWidth = 512, kTrainOut = 128;

int train_rows(int layer) { return layer == 3 ? kTrainOut : kTrainWidth; }

// K splits of the weight gradients: 26 tiles of 128 x 256 in all, so 5 splits
// give each SM one tile, but a split keeps at least four 64-row blocks so that
// its pipeline fills.  More than 5 where a split would sum over 1,024 rows: the
// tensor cores' accumulation loses about 1.2e-6 of the gradient's norm there,
// growing with the rows, and the splits' sums in binary32 next to nothing
// (batch of 16,384: 16 splits 1.2e-6, 5 splits 4.0e-6).
int train_splits(int batch) {
  const int blocks = batch / 64;
  const int fill = blocks / 4 < 1 ? 1 : (blocks / 4 > 5 ? 5 : blocks / 4), precise = (blocks + 15) / 16;
  return precise <= fill ? fill : (precise > 16 ? 16 : precise);
}

}  // namespace

extern "C" size_t rrtmg_sur_train_part_floats(int batch) {
  if (batch <= 0 || batch % 128) return 0;
  return static_cast<size_t>(train_splits(batch)) * kTrainWidth * (3 * kTrainWidth + kTrainOut);
}

extern "C" rrtmg_status rrtmg_sur_train_step(const rrtmg_sur_train_args *a, void *stream) {
  if (!a || a->batch <= 0 || a->batch % 128 || a->ldx != kTrainWidth || a->ldt != kTrainOut) return RRTMG_BAD_ARG;
  const void *need[] = {a->Xb, a->Xbt, a->Tb, a->Y, a->dY, a->dYt, a->part};
  for (const void *p : need)
    if (!p || !aligned16(p)) return RRTMG_BAD_ARG;
  if (!a->X || !a->T || !a->idx || !a->weights || !a->loss) return RRTMG_BAD_ARG;
  for (int i = 0; i < kTrainLayers; ++i) {
    if (!a->wb[i] || !aligned16(a->wb[i]) || !a->wbt[i] || !aligned16(a->wbt[i])) return RRTMG_BAD_ARG;
    if (!a->w[i] || !a->mw[i] || !a->vw[i] || !a->gw[i] || !a->b[i] || !a->mb[i] || !a->vb[i] || !a->gb[i])
      return RRTMG_BAD_ARG;
  }
  for (int i = 0; i < 3; ++i) {
    const void *per[] = {a->Z[i], a->H[i], a->Ht[i], a->dZ[i], a->dZt[i]};
    for (const void *p : per)
      if (!p || !aligned16(p)) return RRTMG_BAD_ARG;
  }
  cudaStream_t s = as_stream(stream);
  const int B = a->batch;
  auto bf = [](const void *p) { return static_cast<const __nv_bfloat16 *>(p); };
  auto bfo = [](void *p) { return static_cast<__nv_bfloat16 *>(p); };
  cudaError_t e = launch_sur_gather(bf(a->X), a->ldx, a->T, a->ldt, a->idx, B, bfo(a->Xb), bfo(a->Xbt), B, a->Tb, s);
  auto gemm = [&](const void *A, int lda, const void *W, int ldb, int M, int N, int K) {
    GemmArgs g{};
    g.A = bf(A);
    g.lda = lda;
    g.B = bf(W);
    g.ldb = ldb;
    g.M = M;
    g.N = N;
    g.K = K;
    g.ksplit = 1;
    g.wait_ns = g_wait_ns.load();
    return g;
  };
  // forward
  const void *in = a->Xb;
  for (int i = 0; i < 3 && e == cudaSuccess; ++i) {
    GemmArgs g = gemm(in, kTrainWidth, a->wb[i], kTrainWidth, B, kTrainWidth, kTrainWidth);
    g.epi = kEpiGelu;
    g.bias = a->b[i];
    g.Z = a->Z[i];
    g.ldz = kTrainWidth;
    g.H = bfo(a->H[i]);
    g.ldh = kTrainWidth;
    g.Ht = bfo(a->Ht[i]);
    g.ldht = B;
    e = launch_umma_gemm(g, s);
    in = a->H[i];
  }
  if (e == cudaSuccess) {
    GemmArgs g = gemm(in, kTrainWidth, a->wb[3], kTrainWidth, B, kTrainOut, kTrainWidth);
    g.epi = kEpiF32;
    g.bias = a->b[3];
    g.C = a->Y;
    g.ldc = kTrainOut;
    e = launch_umma_gemm(g, s);
  }
  if (e == cudaSuccess)
    e = launch_sur_loss_grad(a->Y, a->Tb, a->weights, B, kTrainOut, a->loss_scale, bfo(a->dY), bfo(a->dYt), B, a->loss,
                             s);
  // backward: d(pre-activation) of layers 2, 1, 0
  for (int i = 3; i > 0 && e == cudaSuccess; --i) {
    GemmArgs g = gemm(i == 3 ? a->dY : a->dZ[i], train_rows(i), a->wbt[i], train_rows(i), B, kTrainWidth, train_rows(i));
    g.epi = kEpiDgelu;
    g.aux = a->Z[i - 1];
    g.ldaux = kTrainWidth;
    g.H = bfo(a->dZ[i - 1]);
    g.ldh = kTrainWidth;
    g.Ht = bfo(a->dZt[i - 1]);
    g.ldht = B;
    e = launch_umma_gemm(g, s);
  }
  if (e != cudaSuccess) return cuda_status(e);
  // weight gradients d(pre-activation)^T x inputs^T, then the update
  const int splits = train_splits(B);
  GemmArgs group[kTrainLayers];
  SurUpdateArgs u{};
  u.layers = kTrainLayers;
  u.splits = splits;
  u.batch = B;
  u.lr = a->lr; u.beta1 = a->beta1; u.beta2 = a->beta2; u.eps = a->eps;
  u.bc1 = a->bc1; u.bc2 = a->bc2; u.weight_decay = a->weight_decay;
  float *part = a->part;
  for (int i = 0; i < kTrainLayers; ++i) {
    const int rows = train_rows(i);
    const size_t slab = static_cast<size_t>(rows) * kTrainWidth;
    GemmArgs g = gemm(i == 3 ? a->dYt : a->dZt[i], B, i == 0 ? a->Xbt : a->Ht[i - 1], B, rows, kTrainWidth, B);
    g.epi = kEpiF32;
    g.ksplit = splits;
    g.C = part;
    g.ldc = kTrainWidth;
    g.split_stride = slab;
    group[i] = g;
    u.rows[i] = rows;
    u.cols[i] = kTrainWidth;
    u.aligned[i] = aligned16(a->w[i]) && aligned16(a->mw[i]) && aligned16(a->vw[i]) && aligned16(a->gw[i]);
    u.gt[i] = g.A;
    u.part[i] = part;
    u.w[i] = a->w[i]; u.mw[i] = a->mw[i]; u.vw[i] = a->vw[i]; u.gw[i] = a->gw[i];
    u.b[i] = a->b[i]; u.mb[i] = a->mb[i]; u.vb[i] = a->vb[i]; u.gb[i] = a->gb[i];
    u.wb[i] = bfo(a->wb[i]);
    u.wbt[i] = bfo(a->wbt[i]);
    part += splits * slab;
  }
  e = launch_umma_gemm_group(group, kTrainLayers, s);
  if (e == cudaSuccess) e = launch_sur_update(u, s);
  return cuda_status(e);
}

extern "C" rrtmg_status rrtmg_sur_decode(const rrtmg_sur_decode_args *a, void *stream) {
  if (!a || a->ncol < 0 || a->nk <= 0 || a->ny <= 0 || !a->Y || a->ldy < 2 * a->nk + 6 || 2 * a->nk + 6 > 128 ||
      !a->out_mean ||
      !a->out_std || !a->coszr || !a->pi3d || !a->p8w || !a->rthratenlw || !a->rthratensw || !a->glw || !a->lwupb ||
      !a->swdnb || !a->swupb || !a->flags)
    return RRTMG_BAD_ARG;
  if (a->ncol == 0) return RRTMG_OK;
  return cuda_status(launch_sur_decode(*a, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_compact(const unsigned *flags, int ncol, int *list, int *count, void *stream) {
  if (!flags || ncol < 0 || !list || !count) return RRTMG_BAD_ARG;
  if (ncol == 0) return RRTMG_OK;
  return cuda_status(launch_sur_compact(flags, ncol, list, count, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_move_columns(const int *list, const int *count, int max_n, int nz, int ny,
                                               const float *src, float *dst, int to_compact, int stride, int offset,
                                               void *stream) {
  if (!list || !count || max_n < 0 || nz <= 0 || ny <= 0 || !src || !dst || offset < 0 || stride < offset + max_n)
    return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_move_columns(list, count, max_n, nz, ny, src, dst, to_compact, stride, offset,
                                             as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_gemm_set_tile(int bn) {
  if (bn != 0 && bn != 128 && bn != 256) return RRTMG_BAD_ARG;
  set_gemm_tile(bn);
  return RRTMG_OK;
}

extern "C" rrtmg_status rrtmg_sur_normalize(const float *in, int ldi, int n, int nf, const float *mean,
                                            const float *rstd, void *out, int ldo, int out_bf16, void *stream) {
  if (!in || !mean || !rstd || !out || n <= 0 || nf <= 0 || ldi < nf || ldo < nf) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_normalize(in, ldi, n, nf, mean, rstd, out, ldo, out_bf16, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_timestamp(unsigned long long *slot, void *stream) {
  if (!slot) return RRTMG_BAD_ARG;
  return cuda_status(launch_timestamp(slot, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_pack_weights(const void *const W[4], void *image, void *stream) {
  if (!W || !image || !aligned16(image)) return RRTMG_BAD_ARG;
  for (int l = 0; l < 4; ++l)
    if (!W[l] || !aligned16(W[l])) return RRTMG_BAD_ARG;
  return cuda_status(launch_sur_pack_weights(W, image, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_mlp(const rrtmg_sur_mlp_args *a, void *stream) {
  if (!a || a->ncol < 0 || a->nk != 50 || a->ny <= 0 || !a->X || !a->W || !aligned16(a->X) || !aligned16(a->W))
    return RRTMG_BAD_ARG;
  for (int l = 0; l < 4; ++l)
    if (!a->bias[l]) return RRTMG_BAD_ARG;
  if (!a->out_mean || !a->out_std || !a->coszr || !a->pi3d || !a->p8w || !a->rthratenlw || !a->rthratensw ||
      !a->glw || !a->lwupb || !a->swdnb || !a->swupb || !a->flags)
    return RRTMG_BAD_ARG;
  if (a->ncol == 0) return RRTMG_OK;
  return cuda_status(launch_sur_mlp(*a, as_stream(stream)));
}

extern "C" rrtmg_status rrtmg_sur_move_fields(const int *list, const int *count, int max_n, int ny,
                                              const rrtmg_sur_fields *f, int to_compact, int stride, int offset,
                                              void *stream) {
  if (!list || !count || !f || max_n < 0 || ny <= 0 || offset < 0 || stride < offset + max_n || f->nfields < 0 ||
      f->nfields > RRTMG_SUR_MAX_FIELDS)
    return RRTMG_BAD_ARG;
  for (int i = 0; i < f->nfields; ++i) {
    if (!f->src[i] || !f->dst[i] || f->nz[i] <= 0) return RRTMG_BAD_ARG;
    if (!device_reachable(f->src[i]) || !device_reachable(f->dst[i])) return RRTMG_BAD_ARG;
  }
  return cuda_status(launch_sur_move_fields(list, count, max_n, ny, *f, to_compact, stride, offset,
                                            as_stream(stream)));
}
