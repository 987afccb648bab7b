// tl_ir_cg.cuh -- the FP32-refined CG solve for persistent kernels, one deck
// (tl_ir_cg.cu) or a batch (tl_batch.cu): the FP32 iterations, the FP64
// refinements between them and the last search direction's export, with no
// launch and no host round trip in between.
//
// The iteration is CG with one reduction (Chronopoulos and Gear).  With
// s = A p carried beside p, one pass over the fields does
//     w = A r;  s = w + beta s;  p = r + beta p;  x += alpha p;  r -= alpha s
// and the three sums of the new r that the next scalars need,
//     gamma = r.r,  delta = r.A r = gamma + (sum over faces k (r - r_nbr)^2),  rho = r.s,
//     beta = gamma / gamma_old,  sigma = delta + 2 beta rho + beta^2 sigma_old (= p.A p),  alpha = gamma / sigma.
// rho is summed, not taken from the identity -gamma/alpha, so a residual that a
// refinement has replaced keeps sigma exact.  w is recomputed from r instead
// of stored, and delta's face sums need the new r only at the cell and its
// east and north neighbours: a warp forms one more row and one lane of its
// neighbours' new r.  p and x enter nothing else, so every second pass does two
// steps' worth of them.
//
// Bytes per cell: r, s, iw read, r, s written (20), and in every second pass
// the older r, p, x read, p, x written (20): 30 on average against the 40 of
// the two-kernel form (direction with its dot, update with its dot), which
// needs two reductions.
//
// What bounds it: HBM on large grids; on small ones (everything in L2) the
// grid barrier and the reduction behind it, 2.1 us of an iteration.
#pragma once

#include <cmath>

#include "tl_ir_ops.cuh"
#include "tl_march.cuh"
#include "tl_persist.cuh"

namespace tl {
namespace {

constexpr int STRIP = 120;      // columns a warp owns: lanes 1..30, the outer two are its neighbours' cells
constexpr int RING_BYTES = 12288;  // ring of one warp: 8 rows of r, iw, s, or 4 rows of those and r_old, p, x
enum { PASS_START = 0, PASS_STEP = 1, PASS_STEP2 = 2 };

struct IrCg {
  Fields F;
  Geom g;
  G32 g32;
  float *r[2], *s[2], *p, *x;
  const float *iw;
  double delta2;
  Tiling t;    // FP32 passes
  Tiling t64;  // FP64 residual
  GridSums *sums;
};

struct PassArgs {
  const float *rc, *sc;     // the current r and s
  float *rn, *sn;           // the next ones (r_old, for PASS_STEP2, is read from rn first)
  float alpha, beta;        // this step
  float alpha0, beta0;      // PASS_STEP2: the step before, whose p and x are formed here
  float down;               // the sums' scale
  bool s_valid, p_valid, x_valid;  // false: zero, whatever the buffer holds
  bool mirrored;            // from the last rows to the first
};

__device__ __forceinline__ float4 f4(float a, float b, float c, float d) { return make_float4(a, b, c, d); }

// One pass over the grid: this warp's share of gamma, the face sums and rho in
// lanes 0, 8 and 16, as digits where tiles are handed out, else as pairs.
template <int PASS, bool HANDED>
__device__ __forceinline__ void ir_pass(Grid grid, const IrCg &A, const PassArgs &q, unsigned ring, float rxh, float ryh,
                                        unsigned &handed, PassSums &sums) {
  constexpr int NARR = PASS == PASS_STEP2 ? 6 : 3;
  constexpr int DEPTH = RING_BYTES / (NARR * 512);
  const int nx = A.g32.nx, ny = A.g32.ny;
  const int lane = threadIdx.x & 31;
  const unsigned slot0 = ring + 16 * lane;
  TileWalk walk(grid, A.t, ny, q.mirrored, &A.F.sc->bar.next_tile, handed);
  if (HANDED) handed += walk.requests();
  while (walk.valid()) {
    int strip, j0, j1;
    walk.place(strip, j0, j1);
    const unsigned asked = HANDED ? walk.ask() : 0u;
    const int i0 = strip * STRIP - 4 + 4 * lane;
    const bool in = i0 >= 0 && i0 < nx;
    const bool owns = lane >= 1 && lane <= 30 && i0 < nx;
    Pair acc[3] = {};
    // a face to the east of cell i exists for 0 <= i and i + 1 < nx
    float fe[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) fe[m] = (i0 + m >= 0 && i0 + m + 1 < nx) ? rxh : 0.f;
    const int qlast = min(j1 + 1, ny);
    // a copy that reads nothing still needs a 16-byte aligned address: cell 0 of the first row
    const size_t col = in ? A.g32.at(i0, 0) : (size_t)A.g32.hd;
    size_t next = col + (in ? (long long)(j0 - 1) * A.g32.pitch : 0);  // of the next row to copy
    const size_t step = in ? (size_t)A.g32.pitch : 0;
    auto issue = [&](int row, unsigned slot) {
      if (row <= qlast && row >= 0 && row < ny) {
        const unsigned a = slot0 + slot * (NARR * 512);
        cp16(a, q.rc + next, in);
        cp16(a + 512, A.iw + next, in);
        if (row >= j0) {
          cp16(a + 1024, q.sc + next, in && q.s_valid);
          if (PASS == PASS_STEP2 && row < j1) {
            cp16(a + 1536, q.rn + next, in);
            cp16(a + 2048, A.p + next, in && q.p_valid);
            cp16(a + 2560, A.x + next, in && q.x_valid);
          }
        }
      }
      next += step;
      cp_commit();
    };
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) issue(j0 - 1 + d, d);
    float4 rs = f4(0, 0, 0, 0), rc = rs, ic = rs, ks = rs, rp = rs;
    float ps[3] = {0.f, 0.f, 0.f};
    int nrow = 0;
    unsigned slot = 0, prev = DEPTH - 1;
    for (int row = j0 - 1; row <= qlast; ++row) {
      cp_wait<DEPTH - 2>();
      const unsigned a = slot0 + slot * (NARR * 512);
      float4 rn = f4(0, 0, 0, 0), iwn = rn;
      if (row >= 0 && row < ny) {
        rn = lds4(a);
        iwn = lds4(a + 512);
      }
      float4 kn = f4(0, 0, 0, 0);
      if (row >= j0 && row > 0 && row < ny)  // the faces between rows row-1 and row
        kn = f4(ryh * (ic.x + iwn.x), ryh * (ic.y + iwn.y), ryh * (ic.z + iwn.z), ryh * (ic.w + iwn.w));
      const int j = row - 1;
      if (j >= j0) {
        const unsigned b = slot0 + prev * (NARR * 512);
        const float4 sv = lds4(b + 1024);
        const float ie = __shfl_down_sync(FULL, ic.x, 1);
        float4 ke;
        ke.x = fe[0] * (ic.x + ic.y);
        ke.y = fe[1] * (ic.y + ic.z);
        ke.z = fe[2] * (ic.z + ic.w);
        ke.w = fe[3] * (ic.w + ie);
        float4 s1 = sv, r1 = rc;
        if (PASS != PASS_START) {
          const float kw = __shfl_up_sync(FULL, ke.w, 1);
          const float re = __shfl_down_sync(FULL, rc.x, 1), rw = __shfl_up_sync(FULL, rc.w, 1);
          float4 w;
          w.x = fmaf(ks.x, rc.x - rs.x, fmaf(kn.x, rc.x - rn.x, fmaf(kw, rc.x - rw, fmaf(ke.x, rc.x - rc.y, rc.x))));
          w.y = fmaf(ks.y, rc.y - rs.y, fmaf(kn.y, rc.y - rn.y, fmaf(ke.x, rc.y - rc.x, fmaf(ke.y, rc.y - rc.z, rc.y))));
          w.z = fmaf(ks.z, rc.z - rs.z, fmaf(kn.z, rc.z - rn.z, fmaf(ke.y, rc.z - rc.y, fmaf(ke.z, rc.z - rc.w, rc.z))));
          w.w = fmaf(ks.w, rc.w - rs.w, fmaf(kn.w, rc.w - rn.w, fmaf(ke.z, rc.w - rc.z, fmaf(ke.w, rc.w - re, rc.w))));
          s1 = f4(fmaf(q.beta, sv.x, w.x), fmaf(q.beta, sv.y, w.y), fmaf(q.beta, sv.z, w.z), fmaf(q.beta, sv.w, w.w));
          r1 = f4(fmaf(-q.alpha, s1.x, rc.x), fmaf(-q.alpha, s1.y, rc.y), fmaf(-q.alpha, s1.z, rc.z),
                  fmaf(-q.alpha, s1.w, rc.w));
        }
        if (j > j0) {  // north faces of the row below, with both rows' new r
          const float dx = rp.x - r1.x, dy = rp.y - r1.y, dz = rp.z - r1.z, dw = rp.w - r1.w;
          ps[1] = fmaf(ks.x * dx, dx, fmaf(ks.y * dy, dy, fmaf(ks.z * dz, dz, fmaf(ks.w * dw, dw, ps[1]))));
        }
        if (j < j1) {
          const float r1e = __shfl_down_sync(FULL, r1.x, 1);
          const float dx = r1.x - r1.y, dy = r1.y - r1.z, dz = r1.z - r1.w, dw = r1.w - r1e;
          ps[1] = fmaf(ke.x * dx, dx, fmaf(ke.y * dy, dy, fmaf(ke.z * dz, dz, fmaf(ke.w * dw, dw, ps[1]))));
          ps[0] = fmaf(r1.x, r1.x, fmaf(r1.y, r1.y, fmaf(r1.z, r1.z, fmaf(r1.w, r1.w, ps[0]))));
          ps[2] = fmaf(r1.x, s1.x, fmaf(r1.y, s1.y, fmaf(r1.z, s1.z, fmaf(r1.w, s1.w, ps[2]))));
          if (PASS != PASS_START && owns) {
            const size_t c = col + (size_t)j * A.g32.pitch;
            st4(q.sn + c, s1);
            if (PASS == PASS_STEP2) {
              const float4 ro = lds4(b + 1536), po = lds4(b + 2048);
              float4 xo = lds4(b + 2560);
              float4 p1 = f4(fmaf(q.beta0, po.x, ro.x), fmaf(q.beta0, po.y, ro.y), fmaf(q.beta0, po.z, ro.z),
                             fmaf(q.beta0, po.w, ro.w));
              xo = f4(fmaf(q.alpha0, p1.x, xo.x), fmaf(q.alpha0, p1.y, xo.y), fmaf(q.alpha0, p1.z, xo.z),
                      fmaf(q.alpha0, p1.w, xo.w));
              p1 = f4(fmaf(q.beta, p1.x, rc.x), fmaf(q.beta, p1.y, rc.y), fmaf(q.beta, p1.z, rc.z),
                      fmaf(q.beta, p1.w, rc.w));
              xo = f4(fmaf(q.alpha, p1.x, xo.x), fmaf(q.alpha, p1.y, xo.y), fmaf(q.alpha, p1.z, xo.z),
                      fmaf(q.alpha, p1.w, xo.w));
              st4(A.p + c, p1);
              st4(A.x + c, xo);
            }
            st4(q.rn + c, r1);
          }
          rp = r1;
        }
        if (++nrow == 4) {  // 16 products in FP32, then the pair
          acc[0].add(q.down * ps[0]);
          acc[1].add(q.down * ps[1]);
          acc[2].add(q.down * ps[2]);
          ps[0] = ps[1] = ps[2] = 0.f;
          nrow = 0;
        }
      }
      rs = rc;
      rc = rn;
      ic = iwn;
      ks = kn;
      issue(row + DEPTH - 1, prev);  // its last reader was this trip
      prev = slot;
      slot = slot + 1 == DEPTH ? 0 : slot + 1;
    }
    cp_wait<0>();
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      acc[d].add(q.down * ps[d]);
      if (lane == 0 || lane == 31) acc[d] = Pair{0.f, 0.f};
    }
    add_tile<HANDED>(sums, warp_pairs(acc));
    if (HANDED) walk.take(asked);
    else walk.step();
  }
}

// ---- the solve ---------------------------------------------------------------

// u read past L1: the refinement before this launch's last grid barrier wrote it.
struct SrcU {
  const double *f;
  struct Raw {
    double2 v;
    double ev;
  };
  __device__ __forceinline__ void load(Raw &o, size_t c, long long ec) const {
    o.v = __ldcg(reinterpret_cast<const double2 *>(f + c));
    if (ec >= 0) o.ev = __ldcg(f + ec);
  }
  __device__ __forceinline__ double2 val(const Raw &o) const { return o.v; }
  __device__ __forceinline__ double val_edge(const Raw &o) const { return o.ev; }
};

// The true residual r = u0 - A u in FP64, its FP32 copy in `r32` and r.r in
// `rr`.  In difference form: the couplings multiply differences of neighbouring
// cells, so u's own rounding is not scaled by them.
__device__ __forceinline__ bool ir_residual(Grid grid, const Fields &F, const Geom &g, const G32 &g32, const Tiling &T,
                                            GridSums *sums, SumShared &S, float *r32, unsigned &target, unsigned &set,
                                            unsigned &handed, double &rr) {
  __shared__ double tot;
  const int lane = threadIdx.x & 31;
  SrcU src;
  src.f = F.u;
  Digits share;
  TileWalk walk(grid, T, g.ny, false, &F.sc->bar.next_tile, handed);
  handed += walk.requests();
  while (walk.valid()) {
    int strip, j0, j1;
    walk.place(strip, j0, j1);
    const unsigned asked = walk.ask();
    const int i0 = strip * 64 + 2 * lane;
    double acc = 0.0;
    march<false>(g, F.kx, F.ky, nullptr, src, i0, j0, j1,
                 [&](int j, const Nbr &c0, const Nbr &c1, bool has1, double2) {
                   const size_t c = g.at(i0, j), c32 = g32.at(i0, j);
                   auto resid = [](const Nbr &n, double u0) {
                     double t = u0 - n.c;
                     t = fma(n.kx1, n.e - n.c, t);
                     t = fma(n.kx0, n.w - n.c, t);
                     t = fma(n.ky1, n.n - n.c, t);
                     return fma(n.ky0, n.s - n.c, t);
                   };
                   const double2 b = ld2(F.u0 + c);
                   const double t0 = resid(c0, b.x);
                   acc = fma(t0, t0, acc);
                   if (has1) {
                     const double t1 = resid(c1, b.y);
                     acc = fma(t1, t1, acc);
                     st2(F.r + c, make_double2(t0, t1));
                     *reinterpret_cast<float2 *>(r32 + c32) = make_float2((float)t0, (float)t1);
                   } else {
                     F.r[c] = t0;
                     r32[c32] = (float)t0;
                   }
                 });
    add_lanes(share, acc);
    walk.take(asked);
  }
  if (!grid_sum<1>(grid, S, &F.sc->bar, sums, share, target, set, [&](double a) {
        if (lane == 0) tot = a;
      }))
    return false;
  rr = tot;
  return true;
}

// Up to four FP32 numbers added to, or stored as, the FP64 cells at `c`.
__device__ __forceinline__ void add_f32(double *c, float4 v, int cells) {
  if (cells >= 4) {
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(c)), b = __ldcg(reinterpret_cast<const double2 *>(c + 2));
    st2(c, make_double2(a.x + (double)v.x, a.y + (double)v.y));
    st2(c + 2, make_double2(b.x + (double)v.z, b.y + (double)v.w));
  } else {
    for (int m = 0; m < cells; ++m) c[m] = __ldcg(c + m) + (double)comp(v, m);
  }
}
// An FP32 field's interior in FP64.
__device__ __forceinline__ void export_f32(Grid grid, const Geom &g, const G32 &g32, const float *src, double *dst) {
  const int nx = g.nx, lane = threadIdx.x & 31, chunks = (nx + 127) / 128;
  const long long n = (long long)chunks * g.ny;
  for (long long w = grid.id * PERSIST_WARPS + (threadIdx.x >> 5); w < n; w += grid.nb * PERSIST_WARPS) {
    const int j = (int)(w / chunks), i0 = (int)(w % chunks) * 128 + 4 * lane;
    if (i0 >= nx) continue;
    const float4 v = __ldcg(reinterpret_cast<const float4 *>(src + g32.at(i0, j)));
    double *p = dst + g.at(i0, j);
    if (i0 + 3 < nx) {
      st2(p, make_double2((double)v.x, (double)v.y));
      st2(p + 2, make_double2((double)v.z, (double)v.w));
    } else {
      for (int m = 0; m < nx - i0; ++m) p[m] = (double)comp(v, m);
    }
  }
}

// Scalars of one block, the same on every block.
struct Shared {
  SumShared sum;
  double alpha, beta, gamma, inv_gamma, sigma;
  float alpha_f, beta_f;  // of the next step
  Scale scale;
  int done, sw;
};

// alpha of the next step and 1/gamma, from delta and rho of the current r: both
// quotients in one division, on lanes 0 and 1.
__device__ __forceinline__ void next_scalars(Shared &S, double gamma, double beta, double delta, double rho) {
  const int lane = threadIdx.x & 31;
  const double sigma = fma(beta, fma(beta, S.sigma, rho + rho), delta);
  __syncwarp();  // every lane has read the last step's scalars
  const double quot = (lane == 0 ? gamma : 1.0) / (lane == 0 ? sigma : gamma);
  const float f = (float)(lane == 0 ? quot : beta);
  if (lane == 0) {
    S.alpha = quot;
    S.alpha_f = f;
    S.beta = beta;
    S.gamma = gamma;
    S.sigma = sigma;
  } else if (lane == 1) {
    S.inv_gamma = quot;
    S.beta_f = f;
  }
}

// HANDED: tiles are handed out.
template <bool HANDED>
__device__ __forceinline__ bool ir_loop(Grid grid, const IrCg &A, Shared &S, unsigned ring) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = grid.nb * PERSIST_WARPS, me = grid.id * PERSIST_WARPS + warp;
  GridBar *bar = &A.F.sc->bar;
  const bool lead = grid.id == 0 && threadIdx.x == 0;
  DevScalars *sc = A.F.sc;
  const int nx = A.g.nx, ny = A.g.ny;
  const float rxh = (float)sc->rxh, ryh = (float)sc->ryh;
  const double eps = sc->eps, bb = sc->bb, epslim = sc->epslim;
  const int maxiters = sc->maxiters, presteps = sc->presteps, errorswitch = sc->errorswitch;
  const bool prestep_rule = sc->switch_rule == 1;
  const RootTest test(eps, bb);
  double rr = sc->rro;
  double rel = bb > 0 ? sqrt(rr / bb) : sqrt(rr);
  int iter = sc->iter, nref = 0, sw = 0;
  float *rc = A.r[0], *rn = A.r[1], *sc_ = A.s[0], *sn = A.s[1];
  bool sv = false, pv = false, xv = false, pend = false, mirrored = false;
  float alpha0 = 0.f, beta0 = 0.f;
  unsigned target = 0, set = 0, handed = 0;
  double beta = 0.0, err = 0.0;
  if (threadIdx.x == 0) S.sigma = 0.0;
  __syncthreads();

  while (rel >= eps && iter < maxiters && !sw) {
    const double refine_below = A.delta2 * rr;
    Scale scale = scale_of(rr, Scale{});
    {  // the sums of the residual that the refinement (or the start) left
      PassArgs q{};
      q.rc = rc;
      q.sc = sc_;
      q.s_valid = sv;
      q.mirrored = mirrored;
      q.down = scale.down;
      PassSums sums;
      ir_pass<PASS_START, HANDED>(grid, A, q, ring, rxh, ryh, handed, sums);
      auto fin = [&](double, double f, double r) { next_scalars(S, rr, beta, rr + f, r); };
      if (!grid_sums<HANDED>(grid, S.sum, bar, A.sums, sums, scale.up, target, set, fin)) return false;
      mirrored = !mirrored;
    }
    for (;;) {
      if (lead && prestep_rule && iter < maxiters) A.F.cgalpha[iter + 1] = S.alpha;
      PassArgs q;
      q.rc = rc;
      q.sc = sc_;
      q.rn = rn;
      q.sn = sn;
      q.alpha = S.alpha_f;
      q.beta = S.beta_f;
      q.alpha0 = alpha0;
      q.beta0 = beta0;
      q.s_valid = sv;
      q.p_valid = pv;
      q.x_valid = xv;
      q.mirrored = mirrored;
      q.down = scale.down;
      PassSums sums;
      if (pend) ir_pass<PASS_STEP2, HANDED>(grid, A, q, ring, rxh, ryh, handed, sums);
      else ir_pass<PASS_STEP, HANDED>(grid, A, q, ring, rxh, ryh, handed, sums);
      auto fin = [&](double g, double f, double r) {
        const double b = g * S.inv_gamma;
        const bool claim = test.met(g);
        bool switched = false;
        if (prestep_rule) {
          const int tt = iter + 2;  // the solver loop's next trip (Cheby.jl:25-29, PPCG.jl:27-31)
          switched = errorswitch ? (g < epslim && tt > CGEIGENITERS) : (tt > presteps && g < ERROR_SWITCH_MAX);
          if (lead && iter < maxiters) A.F.cgbeta[iter + 1] = b;
        }
        const bool done = claim || below(g, refine_below) || switched || iter + 1 >= maxiters;
        if (!done) {
          next_scalars(S, g, b, g + f, r);
        } else if (lane == 0) {
          S.beta = b;
          S.gamma = g;
          S.sw = switched;
        }
        if (lane == 0) {
          S.done = done;
          S.scale = scale_of(g, scale);
        }
      };
      if (!grid_sums<HANDED>(grid, S.sum, bar, A.sums, sums, scale.up, target, set, fin)) return false;
      mirrored = !mirrored;
      float *t = rc;
      rc = rn;
      rn = t;
      t = sc_;
      sc_ = sn;
      sn = t;
      sv = true;
      if (pend) pv = xv = true;
      pend = !pend;
      alpha0 = q.alpha;
      beta0 = q.beta;
      ++iter;
      scale = S.scale;
      if (S.done) break;
    }
    beta = S.beta;
    err = S.gamma;
    sw = S.sw;
    // refinement: u += x (with the step whose p and x are still to be formed), x = 0
    const int chunks = (nx + 127) / 128;
    const long long nfold = (long long)chunks * ny;
    for (long long w = me; w < nfold; w += warps) {
      const int j = (int)(w / chunks), i0 = (int)(w % chunks) * 128 + 4 * lane;
      if (i0 >= nx) continue;
      const size_t c = A.g32.at(i0, j), cu = A.g.at(i0, j);
      float4 xo = xv ? __ldcg(reinterpret_cast<const float4 *>(A.x + c)) : f4(0, 0, 0, 0);
      if (pend) {
        const float4 ro = __ldcg(reinterpret_cast<const float4 *>(rn + c));
        const float4 po = pv ? __ldcg(reinterpret_cast<const float4 *>(A.p + c)) : f4(0, 0, 0, 0);
        const float4 p1 = f4(fmaf(beta0, po.x, ro.x), fmaf(beta0, po.y, ro.y), fmaf(beta0, po.z, ro.z),
                             fmaf(beta0, po.w, ro.w));
        xo = f4(fmaf(alpha0, p1.x, xo.x), fmaf(alpha0, p1.y, xo.y), fmaf(alpha0, p1.z, xo.z), fmaf(alpha0, p1.w, xo.w));
        st4(A.p + c, p1);
      }
      add_f32(A.F.u + cu, xo, nx - i0);
    }
    pv = pv || pend;
    pend = false;
    xv = false;
    if (!grid_barrier(grid, bar, target)) return false;
    rc = A.r[0];
    rn = A.r[1];
    if (!ir_residual(grid, A.F, A.g, A.g32, A.t64, A.sums, S.sum, rc, target, set, handed, rr)) return false;
    rel = bb > 0 ? sqrt(rr / bb) : sqrt(rr);
    ++nref;
  }
  // the last search direction in FP64
  if (pv) export_f32(grid, A.g, A.g32, A.p, A.F.p);
  if (lead) {  // none of these is read above once another block may still be at its start
    sc->red[0] = rr;
    sc->red[1] = rel;
    sc->refinements = nref;
    sc->prestep_switch = sw;
    sc->converged = rel < eps;
    if (nref > 0) {
      sc->iter = iter;
      sc->beta = beta;
      sc->error = err;
      sc->alpha = (double)alpha0;
      sc->first = 0;
      sc->done = 1;
    }
  }
  return true;
}

// The solve of one deck by the blocks of `grid`; false when a wait gave up.
__device__ __forceinline__ bool ir_solve(Grid grid, const IrCg &A, Shared &S, unsigned ring) {
  return A.t.handed ? ir_loop<true>(grid, A, S, ring) : ir_loop<false>(grid, A, S, ring);
}

// `set`: in the layout that tl_set_layout has set, if any.
inline void ir_cg_args(IrCg &A, tl_ctx *ctx, int blocks, bool set) {
  tl_ir_state *ir = ctx->ir;
  A.F = ctx->F;
  A.g = ctx->g;
  A.g32 = g32_of(ctx);
  A.r[0] = ir->r;
  A.r[1] = ir->pb;
  A.s[0] = ir->sd;
  A.s[1] = ir->sdb;
  A.p = ir->p;
  A.x = ir->x;
  A.iw = ir->iw;
  A.delta2 = IR_DELTA * IR_DELTA;
  A.sums = static_cast<GridSums *>(ctx->grid_sums);
  // cycles and issue slots of a row and a tile, from the kernel's own counters
  const TileCost pass{2.0, 300.0, 1500.0, 200.0, 400.0, 16, 24, 8}, resid{1.0, 1200.0, 1500.0, 1100.0, 200.0, 0, 48, 4};
  A.t = make_tiling(ctx->g.nx, ctx->g.ny, STRIP, pass, blocks, PERSIST_WARPS);
  if (set && ir->set_rows) {  // equal shares of bands of these rows
    A.t.rows = ir->set_rows < ctx->g.ny ? ir->set_rows : ctx->g.ny;
    A.t.split = ctx->g.ny;
    A.t.tiles = A.t.tiles1 = A.t.ntx * ((ctx->g.ny + A.t.rows - 1) / A.t.rows);
    A.t.blocks = ir->set_blocks < blocks ? ir->set_blocks : blocks;
    A.t.warps = A.t.blocks * PERSIST_WARPS;
    A.t.handed = false;
  }
  A.t64 = make_tiling_on(A.t, ctx->g.nx, ctx->g.ny, 64, resid, PERSIST_WARPS);
}

}  // namespace
}  // namespace tl
