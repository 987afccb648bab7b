// tl_ir.cu -- CG with FP32 inner sweeps inside FP64 refinement: the host side of
// the single-deck solve and of the presteps that Chebyshev and PPCG share
// (kernels: tl_ir_cg.cuh, tl_ir_sweeps.cu).
//
// The inner iteration is CG on FP32 vectors (p, r and the correction x) with
// the stencil faces formed from FP32 inverse weights; each sum adds 16 products
// in FP32 and those partial sums with at least 48 bits.  Whenever the FP32
// residual has dropped by a factor delta since the last refinement, or claims
// convergence, the loop returns to a refinement step done entirely in FP64:
//     u += x;  x = 0;  r = u0 - A u (true residual);  test ||r|| / ||u0||.
// The FP32 residual is then replaced by the true one and the search
// direction is kept (the reliable-update form of iterative refinement), so
// the Krylov space built so far is not thrown away.
//
// The FP32 stencil uses the difference form
// w = p + kx1 (p - pE) + kx0 (p - pW) + ky1 (p - pN) + ky0 (p - pS), which
// keeps the identity term exact where the large coupling terms cancel, with
// kx = rx/2 (iw_W + iw) and ky = ry/2 (iw_S + iw) from the inverse weights.
#include <cmath>
#include <new>

#include "tl_ir_ops.cuh"

using namespace tl;

// r32 = (float) r on the interior.
static __global__ void k_ir_residual(const double *r, Geom g, G32 g32, float *r32) {
  const long long n = (long long)g.nx * g.ny;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k % g.nx), j = (int)(k / g.nx);
    r32[g32.at(i, j)] = (float)r[g.at(i, j)];
  }
}

static int grid_for(long long n) {
  long long b = (n + 255) / 256;
  if (b > 152LL * 32) b = 152LL * 32;
  return (int)(b < 1 ? 1 : b);
}

// The FP32 buffers of a context, allocated on first use.
int tl_ensure_ir(tl_ctx *ctx) {
  if (ctx->ir) return TL_OK;
  tl_ir_state *ir = new (std::nothrow) tl_ir_state();
  if (!ir) return TL_ERR_NOMEM;
  ctx->ir = ir;
  constexpr int NBUF = 7;
  const Geom &g = ctx->g;
  ir->pitch = (g.X + 31) / 32 * 32;
  ir->lead = (32 - g.hd % 32) % 32;
  ir->stride = (ir->lead + ir->pitch * (long long)g.Y + 64 + 63) / 64 * 64;
  CK(cudaMalloc(&ir->buf, sizeof(float) * ir->stride * NBUF));
  CK(cudaMemsetAsync(ir->buf, 0, sizeof(float) * ir->stride * NBUF, ctx->stream));
  float *f[NBUF];
  for (int k = 0; k < NBUF; ++k) f[k] = ir->buf + ir->stride * k + ir->lead;
  ir->p = f[0]; ir->pb = f[1]; ir->r = f[2]; ir->x = f[3]; ir->sd = f[4]; ir->sdb = f[5]; ir->iw = f[6];
  return TL_OK;
}

void tl_release_ir(tl_ctx *ctx) {
  if (!ctx->ir) return;
  if (ctx->ir->buf) cudaFree(ctx->ir->buf);
  delete ctx->ir;
  ctx->ir = nullptr;
}

// The inner loop with its refinements, from the state tl_solve_start left (u,
// r = p = u0 - A u, r.r in rro, the FP32 copies).  Runs until the relative true
// residual is below eps, the iteration budget is spent or, as CG presteps of
// Chebyshev (switch rule 1), the switch test held; the FP32 search direction
// is exported into p.  Returns the last true r.r and its relative value.
static int ir_loop(tl_ctx *ctx, double *rr_out, double *rel_out, int *refinements) {
  ctx->last_solve_ms = 0.0;
  int rc = tl_ir_cg_run(ctx);
  if (rc) return rc;
  const int up[2] = {TL_EX_U, TL_EX_P};
  if ((rc = tl_halo_update(ctx, 1, up, 2, 1))) return rc;
  ctx->launches += 1;
  *rr_out = ctx->host_sc->red[0];
  *rel_out = ctx->host_sc->red[1];
  *refinements = ctx->host_sc->refinements;
  return TL_OK;
}

int tl_ir_solve(tl_ctx *ctx, double rx, double ry, const tl_params *prm, tl_result *res) {
  if (ctx->cfg.mode != TL_MODE_TEALEAF) {
    tl_set_error(ctx, "FP32 refinement needs the tealeaf (5-point) semantics");
    return TL_ERR_ARG;
  }
  int rc = tl_ensure_ir(ctx);
  if (rc) return rc;
  tl_params p = *prm;
  p.criterion = TL_CRIT_RELATIVE;
  if ((rc = tl_solve_start(ctx, rx, ry, &p, 0, TL_START_FP32))) return rc;
  if (prm->warmstart) {
    if ((rc = tl_warm_try(ctx, rx, ry, prm->warmstart, res))) return rc;
    // the residual of the start it chose
    const Geom &g = ctx->g;
    k_ir_residual<<<grid_for((long long)g.nx * g.ny), 256, 0, ctx->stream>>>(ctx->F.r, g, g32_of(ctx), ctx->ir->r);
    CKL();
    ctx->launches += 1;
  }
  double rr = 0.0, rel = 0.0;
  int refinements = 0;
  if ((rc = ir_loop(ctx, &rr, &rel, &refinements))) return rc;
  res->iters = ctx->host_sc->iter;
  res->cg_iters = ctx->host_sc->iter;
  res->error = rr;
  res->rel_residual = rel;
  res->converged = rel < p.eps;
  res->refinements = refinements;
  res->launches = (int)ctx->launches;
  return TL_OK;
}

// The CG presteps of Chebyshev (Cheby.jl:15-35, tealeaf mode) as FP32 inner
// sweeps inside FP64 refinement.  The FP32 epilogues record alpha and beta in
// the coefficient tables for the eigenvalue estimate and apply the switch
// test (Cheby.jl:25-29) to the inner r.r; when it holds, the correction is
// folded into u and the true residual measured before the Chebyshev phase
// takes over.  On return u (with its halo) is the iterate, the host scalars
// hold the loop's end state, *switched says whether the Chebyshev (or PPCG)
// phase takes over (the switch test held and the true residual is not yet
// below eps), *rr_out is the true r.r and *rel_out its relative value.  The
// same presteps serve PPCG (PPCG.jl:27-31 is the same test).
int tl_ir_presteps(tl_ctx *ctx, double rx, double ry, const tl_params *prm, int *refinements, double *rr_out,
                   double *rel_out, int *switched) {
  int rc = tl_ensure_ir(ctx);
  if (rc) return rc;
  tl_params p = *prm;
  p.criterion = TL_CRIT_RELATIVE;
  // with the stored diagonal, which the FP64 Chebyshev step after the switch reads
  if ((rc = tl_solve_start(ctx, rx, ry, &p, 1, TL_START_FP32_DIAG))) return rc;
  if ((rc = ir_loop(ctx, rr_out, rel_out, refinements))) return rc;
  *switched = ctx->host_sc->prestep_switch && *rel_out >= p.eps;
  return TL_OK;
}
