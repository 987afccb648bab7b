// tl_batch.cu -- many independent decks of uneven sizes solved by CG in one
// cooperative launch.
//
// The blocks form groups of equal size; a group takes the next deck from a
// queue, largest first, runs that deck's whole solve as the single-deck kernels
// do (tl_cg64.cuh, or with FP32 refinement tl_ir_cg.cuh) with barriers and sums
// over its own blocks alone, and takes the next when it has converged.  Decks
// share nothing but the queue.
//
// An iteration of one deck costs some 5.5 us (FP64: 8) in barriers and
// reductions however few its cells, which the groups spend at the same time;
// the passes take the same SM time however the SMs are grouped.  So more,
// smaller groups are better until the last decks leave too many SMs idle:
// the number of groups is the one for which a list schedule of the decks ends
// first.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <queue>
#include <vector>

#include "tl_cg64.cuh"
#include "tl_ir_cg.cuh"
#include "tl_solvers.h"

namespace tl {
namespace {

constexpr int BATCH_MAX = 1024;  // decks per batch

// Zeroed before each launch.
struct BatchQueue {
  unsigned next;                            // decks handed out
  unsigned finished;                        // groups that found the queue empty
  GridBar bar[PERSIST_MAX_BLOCKS];          // of each group
  unsigned slot[PERSIST_MAX_BLOCKS][2];     // the group's deck, two in turn
};

// Takes decks for this block's group until none is left.  `solve(grid, args)`
// runs one deck on the first blocks of the group, as many as its tiling uses; the
// others wait at the group's barrier for as long as the deck's own counts on.
template <class Args, class Solve, class Blocks>
__device__ __forceinline__ void take_decks(const Args *decks, Args &A, BatchQueue *Q, int n, int size, Blocks &&blocks,
                                           Solve &&solve) {
  const int group = blockIdx.x / size;
  const Grid grid{size, (int)(blockIdx.x % size)};
  unsigned target = 0;
  for (unsigned turn = 0;; ++turn) {
    if (grid.id == 0 && threadIdx.x == 0) __stcg(&Q->slot[group][turn & 1], atomicAdd(&Q->next, 1u));
    if (!grid_barrier(grid, &Q->bar[group], target, turn ? &A.F.sc->bar.count : nullptr)) return;
    const int d = (int)__ldcg(&Q->slot[group][turn & 1]);
    if (d >= n) {
      if (grid.id == 0 && threadIdx.x == 0) atomicAdd(&Q->finished, 1u);
      return;
    }
    for (int k = threadIdx.x; k < (int)(sizeof(Args) / 4); k += blockDim.x)
      reinterpret_cast<unsigned *>(&A)[k] = reinterpret_cast<const unsigned *>(decks + d)[k];
    __syncthreads();
    const int nb = blocks(A);
    if (grid.id < nb && !solve(Grid{nb, grid.id})) return;
  }
}

__global__ void __launch_bounds__(PERSIST_THREADS, 1) k_batch_ir(const IrCg *decks, BatchQueue *Q, int n, int size) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ Shared S;
  __shared__ IrCg A;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING_BYTES;
  take_decks(decks, A, Q, n, size, [](const IrCg &a) { return a.t.blocks; },
             [&](Grid g) { return ir_solve(g, A, S, ring); });
}

__global__ void __launch_bounds__(WARPS64 * 32, 1) k_batch_64(const Cg64 *decks, BatchQueue *Q, int n, int size) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ Shared64 S;
  __shared__ Cg64 A;
  const Mem64 mem(ring_mem);
  take_decks(decks, A, Q, n, size, [](const Cg64 &a) { return a.tw.blocks; },
             [&](Grid g) { return cg64_solve(g, A, S, mem); });
}

// When the last deck ends with `groups` groups of sms/groups blocks, in
// microseconds: `fixed` + `cell` x cells / blocks an iteration, iterations as the
// square root of the cells (the condition number's growth with the grid).
double makespan(const std::vector<double> &cells, int groups, int sms, double fixed, double cell) {
  const int size = sms / groups;
  std::priority_queue<double, std::vector<double>, std::greater<double>> ends;
  for (int g = 0; g < groups; ++g) ends.push(0.0);
  double last = 0.0;
  for (double c : cells) {
    const double t = ends.top() + std::sqrt(c) * (fixed + cell * c / size);
    ends.pop();
    ends.push(t);
    last = std::max(last, t);
  }
  return last;
}

int best_groups(const std::vector<double> &cells, int sms, double fixed, double cell) {
  int best = 1;
  double t = makespan(cells, 1, sms, fixed, cell);
  for (int g = 2; g <= sms && g <= (int)cells.size(); ++g) {
    const double s = makespan(cells, g, sms, fixed, cell);
    if (s < t) {
      t = s;
      best = g;
    }
  }
  return best;
}

}  // namespace
}  // namespace tl

using namespace tl;

struct tl_batch {
  std::vector<tl_ctx *> ctx;
  std::vector<int> order;  // decks by falling cells
  int device = 0, sms = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  BatchQueue *queue = nullptr;
  Cg64 *d64 = nullptr;     // the decks in `order`, on the first FP64 solve
  IrCg *d32 = nullptr;     // on the first FP32-refined solve
  int size64 = 0, size32 = 0, groups64 = 0, groups32 = 0;
  double last_ms = 0.0;
  char msg[512] = {};
};

namespace {

int bfail(tl_batch *b, cudaError_t e, const char *what) {
  snprintf(b->msg, sizeof b->msg, "CUDA error in %s: %s", what, cudaGetErrorString(e));
  return TL_ERR_CUDA;
}
#define BCK(x)                                  \
  do {                                          \
    cudaError_t e_ = (x);                       \
    if (e_ != cudaSuccess) return bfail(b, e_, #x); \
  } while (0)

// The decks' kernel arguments on the device, in queue order, and the groups.
template <class Args, class Make>
int place_decks(tl_batch *b, Args **dev, int *groups, int *size, double fixed, double cell, Make &&make) {
  if (*dev) return TL_OK;
  std::vector<double> cells;
  for (int k : b->order) cells.push_back((double)b->ctx[k]->g.nx * b->ctx[k]->g.ny);
  *groups = best_groups(cells, b->sms, fixed, cell);
  *size = b->sms / *groups;
  std::vector<Args> h(b->order.size());
  for (size_t k = 0; k < h.size(); ++k) make(h[k], b->ctx[b->order[k]], *size);
  Args *d = nullptr;
  BCK(cudaMalloc(&d, sizeof(Args) * h.size()));
  const cudaError_t e = cudaMemcpyAsync(d, h.data(), sizeof(Args) * h.size(), cudaMemcpyHostToDevice, b->stream);
  if (e != cudaSuccess || cudaStreamSynchronize(b->stream) != cudaSuccess) {
    cudaFree(d);
    return bfail(b, e, "the batch's deck table");
  }
  *dev = d;
  return TL_OK;
}

// One launch over all decks, timed.
int run_decks(tl_batch *b, const void *kernel, const void *decks, int groups, int size, int threads, size_t smem) {
  int n = (int)b->ctx.size();
  BCK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  BCK(cudaMemsetAsync(b->queue, 0, sizeof(BatchQueue), b->stream));
  BCK(cudaEventRecord(b->ev0, b->stream));
  void *args[] = {&decks, &b->queue, &n, &size};
  BCK(cudaLaunchCooperativeKernel(kernel, dim3(groups * size), dim3(threads), args, smem, b->stream));
  BCK(cudaEventRecord(b->ev1, b->stream));
  return TL_OK;
}

int loop_ms(tl_batch *b) {
  float ms = 0.f;
  BCK(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
  b->last_ms = ms;
  return TL_OK;
}

}  // namespace

extern "C" int tl_batch_create(tl_batch **out, tl_ctx *const *ctxs, int n) {
  if (!out) return TL_ERR_ARG;
  *out = nullptr;
  tl_batch *b = new (std::nothrow) tl_batch();
  if (!b) return TL_ERR_NOMEM;
  *out = b;
  if (!ctxs || n < 1 || n > BATCH_MAX) {
    snprintf(b->msg, sizeof b->msg, "batch of %d decks outside 1..%d", n, BATCH_MAX);
    return TL_ERR_ARG;
  }
  BCK(cudaGetDevice(&b->device));
  BCK(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device));
  b->sms = persist_blocks(b->sms);
  for (int k = 0; k < n; ++k) {
    tl_ctx *c = ctxs[k];
    if (!c || c->cfg.mode != TL_MODE_TEALEAF || c->device != b->device) {
      snprintf(b->msg, sizeof b->msg, "deck %d: needs a tealeaf-mode context on the current device", k);
      return TL_ERR_ARG;
    }
    b->ctx.push_back(c);
    b->order.push_back(k);
  }
  auto cells = [b](int k) { return (long long)b->ctx[k]->g.nx * b->ctx[k]->g.ny; };
  std::stable_sort(b->order.begin(), b->order.end(), [&](int x, int y) { return cells(x) > cells(y); });
  BCK(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
  BCK(cudaEventCreate(&b->ev0));
  BCK(cudaEventCreate(&b->ev1));
  BCK(cudaMalloc(&b->queue, sizeof(BatchQueue)));
  return TL_OK;
}

extern "C" int tl_batch_destroy(tl_batch *b) {
  if (!b) return TL_OK;
  if (b->stream) cudaStreamSynchronize(b->stream);
  if (b->queue) cudaFree(b->queue);
  if (b->d64) cudaFree(b->d64);
  if (b->d32) cudaFree(b->d32);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return TL_OK;
}

extern "C" const char *tl_batch_last_error(const tl_batch *b) { return b ? b->msg : "null batch"; }

namespace {

int fetch_scalars(tl_ctx *ctx) {
  CK(cudaMemcpyAsync(ctx->host_sc, ctx->F.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream));
  return TL_OK;
}

// Every deck's work on the batch stream: set-up, the loop, what follows it.
int batch_solve(tl_batch *b, const double *rx, const double *ry, const tl_params *prm, tl_result *results) {
  const int n = (int)b->ctx.size();
  const bool ir = prm->precision == TL_PREC_FP32_IR;
  tl_params p = *prm;
  if (ir) p.criterion = TL_CRIT_RELATIVE;
  int rc = TL_OK;
  for (int k = 0; k < n && !rc; ++k) {
    tl_ctx *ctx = b->ctx[k];
    memset(&results[k], 0, sizeof(tl_result));
    if (ir) results[k].r0_plain = results[k].r0_pred = -1.0;
    ctx->launches = 0;
    rc = tl_solve_start(ctx, rx[k], ry[k], &p, 0, ir ? TL_START_FP32 : TL_START_FP64);
    ctx->bar_clean = 0;  // the batch's kernel uses it
    if (rc) snprintf(b->msg, sizeof b->msg, "deck %d: %.480s", k, ctx->msg);
  }
  if (rc) return rc;
  if (ir) {
    rc = run_decks(b, (const void *)k_batch_ir, b->d32, b->groups32, b->size32, PERSIST_THREADS,
                   (size_t)RING_BYTES * PERSIST_WARPS);
  } else if (p.maxiters >= 1) {
    rc = run_decks(b, (const void *)k_batch_64, b->d64, b->groups64, b->size64, WARPS64 * 32, CG64_SMEM);
  }
  if (rc) return rc;
  // per deck, FP32, the halo of u, p and, FP64 under the relative criterion, the
  // true residual as in the single-deck solve; one wait for all
  for (int k = 0; k < n && !rc; ++k) {
    tl_ctx *ctx = b->ctx[k];
    if (ir) rc = tl_halo_update(ctx, 1, nullptr, -1, 1);
    if (!ir && p.criterion == TL_CRIT_RELATIVE)
      launch_true_resid(ctx->stream, ctx->F, ctx->g, ctx->walk_short, TL_MODE_TEALEAF, 0);
    if (!rc) rc = fetch_scalars(ctx);
    if (rc) snprintf(b->msg, sizeof b->msg, "deck %d: %.480s", k, ctx->msg);
  }
  if (rc) return rc;
  unsigned finished = 0;
  BCK(cudaMemcpyAsync(&finished, &b->queue->finished, sizeof finished, cudaMemcpyDeviceToHost, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  if (ir || p.maxiters >= 1) {
    if ((int)finished != (ir ? b->groups32 : b->groups64)) {
      snprintf(b->msg, sizeof b->msg, "a wait of the batch's kernel gave up: its blocks did not all arrive");
      return TL_ERR_CUDA;
    }
    if ((rc = loop_ms(b))) return rc;
  }
  for (int k = 0; k < n; ++k) {
    tl_ctx *ctx = b->ctx[k];
    if ((rc = tl_persist_check(ctx))) {
      snprintf(b->msg, sizeof b->msg, "deck %d: %.480s", k, ctx->msg);
      return rc;
    }
    const DevScalars &sc = *ctx->host_sc;
    results[k].iters = results[k].cg_iters = sc.iter;
    if (ir) {
      results[k].error = sc.red[0];
      results[k].rel_residual = sc.red[1];
      results[k].converged = sc.converged;
      results[k].refinements = sc.refinements;
      continue;
    }
    double rel = -1.0;
    if (p.criterion == TL_CRIT_RELATIVE) rel = sc.bb > 0 ? sqrt(sc.red[0] / sc.bb) : sqrt(sc.red[0]);
    results[k].error = p.maxiters >= 1 ? sc.error : ERROR_START;
    results[k].converged = p.criterion == TL_CRIT_RELATIVE ? (rel >= 0 && rel < p.eps) : sc.converged;
    results[k].rel_residual = rel;
  }
  return TL_OK;
}

}  // namespace

extern "C" int tl_batch_solve(tl_batch *b, const double *rx, const double *ry, const tl_params *prm,
                              tl_result *results) {
  if (!b || !rx || !ry || !prm || !results) return TL_ERR_ARG;
  if (prm->solver != TL_SOLVER_CG || prm->exact ||
      (prm->precision != TL_PREC_FP64 && prm->precision != TL_PREC_FP32_IR)) {
    snprintf(b->msg, sizeof b->msg, "batched solves run CG (fused FP64 or FP32-refined, exact 0)");
    return TL_ERR_ARG;
  }
  const int n = (int)b->ctx.size();
  const bool ir = prm->precision == TL_PREC_FP32_IR;
  for (int k = 0; k < n; ++k) {
    tl_ctx *ctx = b->ctx[k];
    if (!ctx->initialised || prm->maxiters > ctx->cfg.maxiters) {
      snprintf(b->msg, sizeof b->msg, "deck %d: not initialised, or maxiters beyond its tables", k);
      return TL_ERR_STATE;
    }
    const int rc = ir ? tl_ensure_ir(ctx) : TL_OK;
    if (rc) {
      snprintf(b->msg, sizeof b->msg, "deck %d: %.480s", k, ctx->msg);
      return rc;
    }
    // what the deck's own stream still holds comes before the batch's work
    BCK(cudaEventRecord(ctx->ev0, ctx->stream));
    BCK(cudaStreamWaitEvent(b->stream, ctx->ev0, 0));
  }
  // fixed and per-cell microseconds of an iteration: 5.5 and 11.5 at 1024^2 on 152 SMs, FP64 8 and 30
  int rc = ir ? place_decks(b, &b->d32, &b->groups32, &b->size32, 5.5, 0.87e-3,
                            [](IrCg &A, tl_ctx *ctx, int size) { ir_cg_args(A, ctx, size, false); })
              : place_decks(b, &b->d64, &b->groups64, &b->size64, 8.0, 3.1e-3, [](Cg64 &A, tl_ctx *ctx, int size) {
                  A.F = ctx->F;
                  A.g = ctx->g;
                  A.sums = static_cast<GridSums *>(ctx->grid_sums);
                  A.check = 0;
                  cg64_tilings(A, size);
                });
  if (rc) return rc;
  std::vector<cudaStream_t> own(n);
  for (int k = 0; k < n; ++k) {
    own[k] = b->ctx[k]->stream;
    b->ctx[k]->stream = b->stream;
  }
  rc = batch_solve(b, rx, ry, prm, results);
  for (int k = 0; k < n; ++k) b->ctx[k]->stream = own[k];
  return rc;
}

extern "C" int tl_batch_last_ms(tl_batch *b, double *ms) {
  if (!b || !ms) return TL_ERR_ARG;
  *ms = b->last_ms;
  return TL_OK;
}
