// tl_start.cu -- what one step does around the iteration, a kernel each: the
// start of a solve (tea_leaf_init, the halo of u and p, copyu!: CG.jl:10-12,
// 47-79, kernels.jl:191-220) and its end (solvefinished!, kernels.jl:166-170),
// tealeaf semantics.  The same operations in the same order per cell as the
// separate kernels in tl_kernels_common.cu, which the exact path keeps for their
// order of summation.
#include "tl_ir_ops.cuh"
#include "tl_march.cuh"

namespace tl {
namespace {

// ---------------------------------------------------------------------------
// the start
// ---------------------------------------------------------------------------
//
// Everything follows from density and energy, so one pass does it: a warp takes
// 30 columns of the full array (lanes 0 and 31 are their neighbours) and marches
// over some rows, the face below carried on, the faces and values to the left
// and right by shuffles.  The cells at the domain's edge also write the halo
// next to them.
//
// On a small deck what counts is the chain of dependent kernels: the seven this
// replaces took 48 us, two of them adding up eight rows one by one.  With the
// end's three as one, the halo after the loop in the loop's kernel and one wait
// of the host less, a step of 10 x 10 went from 175 to 120 us, of 257 x 191 from
// 363 to 285, of 512^2 from 826 to 777.  On a large deck it is the FP64 pipe: two divisions a
// cell, three where FP32 weights go with it.
constexpr int START_COLS = 30, START_WARPS = 4;

struct Start {
  Fields F;
  Geom g;
  LoopParams p;
  double rx, ry;
  int recip, diag;  // w = 1/density; store the fused kernels' diagonal
  float *r32, *iw;  // the FP32 loop's residual and inverse weights, or null
  long long pitch32;
  int strips, rows;
  long long tiles;
};

struct StartEnd {  // what the last block does with the sums r.r and u.u
  Fields F;
  LoopParams p;
  double rxh, ryh;
  __device__ void fin(const double *tot) const {
    DevScalars *sc = F.sc;
    sc->rro = tot[0];
    sc->bb = tot[1];
    sc->error = ERROR_START;
    sc->iter = 0;
    sc->done = 0;
    sc->converged = 0;
    sc->switched = 0;
    sc->beta = 0.0;
    sc->first = 1;
    set_params(sc, p);
    sc->rxh = rxh;
    sc->ryh = ryh;
    sc->bar = GridBar{0u, 0u, 0u};
  }
};

__global__ void __launch_bounds__(32 * START_WARPS) k_solve_start(const Start A) {
  const Fields &F = A.F;
  const Geom &g = A.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, hd = g.hd;
  double acc[2] = {0.0, 0.0};
  for (long long t = (long long)blockIdx.x * START_WARPS + warp; t < A.tiles; t += (long long)gridDim.x * START_WARPS) {
    const int I = (int)(t % A.strips) * START_COLS + lane - 1, j0 = (int)(t / A.strips) * A.rows;
    const int j1 = min(j0 + A.rows, g.Y);
    const bool col = I >= 0 && I < g.X, owns = lane >= 1 && lane <= START_COLS && I < g.X;
    const bool kcol = I >= hd && I < g.X - 1, icol = I >= hd && I < g.X - hd;
    auto load = [&](int J, double &rho, double &e) {
      const bool in = col && J >= 0 && J < g.Y;
      rho = in ? __ldg(F.density + g.full(I, J)) : 1.0;
      e = in ? __ldg(F.energy + g.full(I, J)) : 0.0;
    };
    auto weight = [&](double rho) { return A.recip ? ddiv(1.0, rho) : rho; };
    // a face from the weights on its sides; outside the range of tea_leaf_init what the field holds
    auto face = [&](double k, double wl, double wc, const double *field, int J) {
      if (kcol && J >= hd && J < g.Y - 1) return ddiv(dmul(k, dadd(wl, wc)), dmul(dmul(2.0, wl), wc));
      return hd == 1 && col && J < g.Y ? field[g.full(I, J)] : 0.0;
    };
    double rs, es, rho, e, rn, en;
    load(j0 - 1, rs, es);
    load(j0, rho, e);
    load(j0 + 1, rn, en);
    double us = dmul(es, rs), u = dmul(e, rho), w = weight(rho);
    double ky = face(A.ry, weight(rs), w, F.ky, j0);
    for (int J = j0; J < j1; ++J) {
      double r2, e2;
      load(J + 2, r2, e2);
      const double un = dmul(en, rn), wn = weight(rn);
      const double kyn = face(A.ry, w, wn, F.ky, J + 1);
      const double kx = face(A.rx, __shfl_up_sync(FULL, w, 1), w, F.kx, J);
      const double kxr = __shfl_down_sync(FULL, kx, 1);
      const double uw = __shfl_up_sync(FULL, u, 1), ue = __shfl_down_sync(FULL, u, 1);
      const bool irow = J >= hd && J < g.Y - hd;
      if (owns) {
        const size_t c = g.full(I, J);
        float r32 = 0.f;
        if (irow && icol) {
          const double consum = dadd(dadd(dadd(dadd(1.0, kxr), kx), kyn), ky);
          double v = dmul(consum, u);
          v = dsub(v, dadd(dmul(kxr, ue), dmul(kx, uw)));
          v = dsub(v, dadd(dmul(kyn, un), dmul(ky, us)));
          const double r = dsub(u, v);
          F.u[c] = u;
          F.u0[c] = u;
          F.p[c] = r;
          F.r[c] = r;
          F.w[c] = v;
          if (A.diag) F.diag[c] = consum;
          put_faces(F.u, g, c, I - hd, J - hd, u);
          put_faces(F.p, g, c, I - hd, J - hd, r);
          acc[0] = dadd(acc[0], dmul(r, r));
          acc[1] = dadd(acc[1], dmul(u, u));
          r32 = (float)r;
        } else {
          if (!(irow && (I == hd - 1 || I == g.X - hd)) && !(icol && (J == hd - 1 || J == g.Y - hd))) {
            F.u[c] = u;
            F.p[c] = 0.0;
          }
          F.r[c] = 0.0;
          F.w[c] = w;
        }
        if (kcol && J >= hd && J < g.Y - 1) {
          F.kx[c] = kx;
          F.ky[c] = ky;
        }
        if (A.iw) {
          const size_t c32 = (size_t)I + (size_t)J * (size_t)A.pitch32;
          A.r32[c32] = r32;
          A.iw[c32] = (float)(A.recip ? rho : ddiv(1.0, rho));
        }
      }
      us = u;
      u = un;
      w = wn;
      ky = kyn;
      rho = rn;
      rn = r2;
      en = e2;
    }
  }
  finish_reduction<2>(acc, StartEnd{F, A.p, 0.5 * A.rx, 0.5 * A.ry});
}

// ---------------------------------------------------------------------------
// the end
// ---------------------------------------------------------------------------

// residual! (`check`), finalise! and the halo of energy.
__global__ void k_solve_end(Fields F, Geom g, int check) {
  const long long n = (long long)g.nx * g.ny;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k % g.nx), j = (int)(k / g.nx);
    const size_t c = g.at(i, j);
    if (check) F.r[c] = dsub(F.u0[c], smvp_exact(F, g, F.u, c, TL_MODE_TEALEAF));
    const double e = ddiv(F.u[c], F.density[c]);
    F.energy[c] = e;
    put_faces(F.energy, g, c, i, j, e);
  }
}

int blocks_for(long long n, int per, int most) {
  const long long b = (n + per - 1) / per;
  return (int)(b < 1 ? 1 : b > most ? most : b);
}

}  // namespace
}  // namespace tl

using namespace tl;

// The state an iteration starts from (u, u0, r = p = u0 - A u, the faces, r.r,
// u.u, the loop's parameters, a zeroed grid barrier), with the halo of u and p.
int tl_solve_start(tl_ctx *ctx, double rx, double ry, const tl_params *prm, int switch_rule, int kind) {
  const int up[2] = {TL_EX_U, TL_EX_P};
  int rc;
  if (kind == TL_START_EXACT) {
    if ((rc = tl_cg_init(ctx, rx, ry, prm->coefficient))) return rc;
    if ((rc = tl_set_loop_params(ctx, prm, switch_rule, 0))) return rc;
    if ((rc = tl_halo_update(ctx, 1, up, 2, 1))) return rc;  // CG.jl:11
    ctx->launches += 6;
    return tl_copy_u(ctx);                                   // CG.jl:12
  }
  if ((rc = tl_check_coefficient(ctx, prm->coefficient))) return rc;
  if ((rc = tl_halo_check(ctx, 1))) return rc;
  Start A{};
  A.F = ctx->F;
  A.g = ctx->g;
  A.p = loop_params(prm, switch_rule, 0);
  A.rx = rx;
  A.ry = ry;
  A.recip = prm->coefficient != TL_CONDUCTIVITY;
  A.diag = kind == TL_START_FP64 || kind == TL_START_FP32_DIAG;
  if (kind != TL_START_FP64) {
    A.r32 = ctx->ir->r;
    A.iw = ctx->ir->iw;
    A.pitch32 = ctx->ir->pitch;
  }
  // Rows a tile: one until two warps run on each quarter of an SM; a tile starts
  // with one more division, so beyond that as many as keep that.
  A.strips = (A.g.X + START_COLS - 1) / START_COLS;
  const long long rows = (long long)A.strips * A.g.Y / (8LL * ctx->sm_count);
  A.rows = (int)(rows < 1 ? 1 : rows > 32 ? 32 : rows);
  A.tiles = (long long)A.strips * ((A.g.Y + A.rows - 1) / A.rows);
  k_solve_start<<<blocks_for(A.tiles, START_WARPS, ctx->max_blocks), 32 * START_WARPS, 0, ctx->stream>>>(A);
  CKL();
  ctx->launches += 1;
  ctx->bar_clean = 1;
  for (int k = 0; k < TL_NEX; ++k) ctx->toexchange[k] = k == TL_EX_U || k == TL_EX_P;
  return TL_OK;
}

// The grid barrier of the next persistent launch at zero.
int tl_bar_ready(tl_ctx *ctx) {
  if (!ctx->bar_clean) CK(cudaMemsetAsync(&ctx->F.sc->bar, 0, sizeof(GridBar), ctx->stream));
  ctx->bar_clean = 0;
  return TL_OK;
}

// solvefinished! without its wait (tealeaf mode).
int tl_solve_end(tl_ctx *ctx, int checkresult) {
  int rc = tl_halo_check(ctx, 1);
  if (rc) return rc;
  k_solve_end<<<blocks_for((long long)ctx->g.nx * ctx->g.ny, 256, 152 * 32), 256, 0, ctx->stream>>>(ctx->F, ctx->g,
                                                                                                    checkresult);
  CKL();
  ctx->toexchange[TL_EX_ENERGY] = 1;
  return TL_OK;
}
