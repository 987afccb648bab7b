// tl_sweeps64.cu -- the fused FP64 loops of Chebyshev, PPCG and Jacobi (tealeaf
// semantics) as persistent kernels: src/solvers/Cheby.jl:81-106, PPCG.jl:64-94,
// Jacobi.jl:59-80.
//
// Every pass is a ring64 march, bound by the FP64 pipe on large grids; on small
// ones a pass cost 4-7 us as a kernel of a graph, and costs a grid barrier
// (1.2 us) here, with the reduction (1.4 us more) only where a test reads it:
// each Jacobi sweep, the last sweep of a PPCG step, and the Chebyshev steps
// that take the norm (Cheby.jl:48), which are also the only ones that can be
// the last and so the only ones that store w and r.
#include "tl_march.cuh"
#include "tl_ring64.cuh"
#include "tl_solvers.h"

namespace tl {
namespace {

struct Loop64 {
  Fields F;
  Geom g;
  Tiling t;   // strips of 60 columns
  Tiling te;  // elementwise pass: strips of 64
  GridSums *sums;
  int ninner;  // PPCG inner sweeps
};

struct SharedLoop {
  SumShared sum;
  double a, b;
  int done, conv, first;
};

// The state every loop carries.
struct LoopState {
  unsigned ring, target = 0, set = 0, handed = 0;
  bool mirrored = false;
};

__device__ __forceinline__ Ring64 ring_of(const Loop64 &A, const double *m, const double *o0, const double *o1) {
  Ring64 q;
  q.g = A.g;
  q.m = m;
  q.m2 = nullptr;
  q.kx = A.F.kx;
  q.ky = A.F.ky;
  q.dg = A.F.diag;
  q.own[0] = o0;
  q.own[1] = o1;
  q.beta = 0.0;
  q.m_valid = true;
  return q;
}

// loop_control's test on the loop's error (no presteps' switch here).
struct LoopTest {
  RootTest root;
  double eps;
  bool relative;
  __device__ __forceinline__ LoopTest(const DevScalars *sc)
      : root(sc->eps, sc->bb), eps(sc->eps), relative(sc->crit == TL_CRIT_RELATIVE) {}
  __device__ __forceinline__ bool met(double error) const { return relative ? root.met(error) : below(error, eps); }
};

// ---- Chebyshev ---------------------------------------------------------------

__global__ void __launch_bounds__(WARPS64 * 32, 1) k_cheby64(const Loop64 A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ SharedLoop S;
  const Fields &F = A.F;
  DevScalars *sc = F.sc;
  LoopState L;
  L.ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING64_BYTES;
  const LoopTest test(sc);
  const int maxiters = sc->maxiters, est = sc->est_iters;
  int k = sc->cheby_iters, iter = sc->iter, conv = 0;
  double error = sc->error;
  double *u = (k & 1) ? F.ub : F.u, *un = (k & 1) ? F.u : F.ub;
  for (;;) {
    ++k;
    const int tt = iter + 1, idx = min(k + 1, maxiters + 1);  // the tables hold maxiters + 2 entries
    const double ca = F.chebyalpha[idx], cb = F.chebybeta[idx];
    const bool norm = k >= est && (tt + 1) % 10 == 0;  // Cheby.jl:48
    const bool store = norm || tt >= maxiters;
    double acc = 0.0;
    Digits sum;
    ring64<false, 2>(whole_grid(), ring_of(A, u, F.u0, F.p), A.t, L.ring, L.mirrored, &A.F.sc->bar.next_tile, L.handed,
                     [&](int j, int i0, bool has1, bool owns, const Row64 &q) {
                       const double2 w = apply64(q, has1);
                       const double2 r = make_double2(q.own[0].x - w.x, q.own[0].y - w.y);
                       const double2 p = make_double2(fma(ca, q.own[1].x, cb * r.x), fma(ca, q.own[1].y, cb * r.y));
                       if (owns) {
                         const size_t c = A.g.at(i0, j);
                         if (norm) {
                           acc = fma(r.x, r.x, acc);
                           if (has1) acc = fma(r.y, r.y, acc);
                         }
                         if (store) {
                           put64(F.w + c, w, has1);
                           put64(F.r + c, r, has1);
                         }
                         put64(F.p + c, p, has1);
                         put64(un + c, make_double2(q.c.x + p.x, q.c.y + p.y), has1);
                       }
                     },
                     [&]() {
                       if (norm) add_lanes(sum, acc);
                       acc = 0.0;
                     });
    L.mirrored = !L.mirrored;
    iter = tt;
    double *t = u;
    u = un;
    un = t;
    if (norm) {
      if (!grid_sum<1>(whole_grid(), S.sum, &sc->bar, A.sums, sum, L.target, L.set, [&](double rr) {
            const bool cv = test.met(rr);
            if ((threadIdx.x & 31) == 0) {
              S.a = rr;
              S.conv = cv;
            }
          }))
        return;
      error = S.a;
      conv = S.conv;
    } else if (!grid_barrier(whole_grid(), &sc->bar, L.target)) {
      return;
    }
    if (conv || iter >= maxiters) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->cheby_iters = k;
    sc->iter = iter;
    sc->error = error;
    sc->converged = conv;
    sc->done = 1;
  }
}

// ---- PPCG --------------------------------------------------------------------

// u += alpha p, r -= alpha w, sd = r / theta on this warp's tiles.
__device__ __forceinline__ void ppcg_update(const Loop64 &A, LoopState &L, const double *p, double alpha, double rtheta) {
  const int nx = A.g.nx, lane = threadIdx.x & 31;
  TileWalk walk(whole_grid(), A.te, A.g.ny, L.mirrored, &A.F.sc->bar.next_tile, L.handed);
  L.handed += walk.requests();
  while (walk.valid()) {
    int strip, j0, j1;
    walk.place(strip, j0, j1);
    const unsigned asked = walk.ask();
    const int i0 = strip * 64 + 2 * lane;
    if (i0 < nx) {
      const bool has1 = i0 + 1 < nx;
#pragma unroll 4
      for (int j = j0; j < j1; ++j) {
        const size_t c = A.g.at(i0, j);
        auto ld = [&](const double *f) { return __ldcg(reinterpret_cast<const double2 *>(f + c)); };
        const double2 pv = ld(p), wv = ld(A.F.w), uv = ld(A.F.u), rv = ld(A.F.r);
        const double2 r = make_double2(fma(-alpha, wv.x, rv.x), fma(-alpha, wv.y, rv.y));
        put64(A.F.u + c, make_double2(fma(alpha, pv.x, uv.x), fma(alpha, pv.y, uv.y)), has1);
        put64(A.F.r + c, r, has1);
        put64(A.F.sd + c, make_double2(r.x * rtheta, r.y * rtheta), has1);
      }
    }
    __syncwarp();
    walk.take(asked);
  }
}

__global__ void __launch_bounds__(WARPS64 * 32, 1) k_ppcg64(const Loop64 A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ SharedLoop S;
  const Fields &F = A.F;
  DevScalars *sc = F.sc;
  LoopState L;
  L.ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING64_BYTES;
  const LoopTest test(sc);
  const int maxiters = sc->maxiters;
  const double rtheta = 1.0 / sc->theta;
  int outer = sc->cheby_iters, iter = sc->iter;
  double rro = sc->rro, alpha = 0.0, beta = sc->beta, pw = 0.0;
  bool first = sc->first != 0;  // the first direction is p itself
  double *p = F.p, *pn = F.pb;
  for (;;) {
    double acc = 0.0;
    Digits sum;
    auto tile_end = [&]() {
      add_lanes(sum, acc);
      acc = 0.0;
    };
    auto direction = [&](int j, int i0, bool has1, bool owns, const Row64 &q) {
      const double2 w = apply64(q, has1);
      if (owns) {
        const size_t c = A.g.at(i0, j);
        acc = fma(w.y, q.c.y, fma(w.x, q.c.x, acc));
        put64(F.w + c, w, has1);
        put64(pn + c, q.c, has1);
      }
    };
    Ring64 d = ring_of(A, p, nullptr, nullptr);
    d.m2 = F.r;
    d.beta = beta;
    if (first) ring64<false, 0>(whole_grid(), d, A.t, L.ring, L.mirrored, &A.F.sc->bar.next_tile, L.handed, direction, tile_end);
    else ring64<true, 0>(whole_grid(), d, A.t, L.ring, L.mirrored, &A.F.sc->bar.next_tile, L.handed, direction, tile_end);
    if (!grid_sum<1>(whole_grid(), S.sum, &sc->bar, A.sums, sum, L.target, L.set, [&](double pw) {
          const double a = ddiv(rro, pw);
          if ((threadIdx.x & 31) == 0) {
            S.a = a;
            S.b = pw;
          }
        }))
      return;
    alpha = S.a;
    pw = S.b;
    {
      double *t = p;
      p = pn;
      pn = t;
    }
    first = false;
    L.mirrored = !L.mirrored;
    ppcg_update(A, L, p, alpha, rtheta);
    if (!grid_barrier(whole_grid(), &sc->bar, L.target)) return;
    sum = Digits{};
    for (int pp = 1; pp <= A.ninner; ++pp) {
      const double ca = F.chebyalpha[pp], cb = F.chebybeta[pp];
      const double *src = (pp & 1) ? F.sd : F.sdb;
      double *dst = (pp & 1) ? F.sdb : F.sd;
      const bool last = pp == A.ninner;
      L.mirrored = !L.mirrored;
      ring64<false, 2>(whole_grid(), ring_of(A, src, F.r, F.u), A.t, L.ring, L.mirrored, &A.F.sc->bar.next_tile, L.handed,
                       [&](int j, int i0, bool has1, bool owns, const Row64 &q) {
                         const double2 a = apply64(q, has1);
                         const double2 r = make_double2(q.own[0].x - a.x, q.own[0].y - a.y);
                         if (owns) {
                           const size_t c = A.g.at(i0, j);
                           if (last) {
                             acc = fma(r.x, r.x, acc);
                             if (has1) acc = fma(r.y, r.y, acc);
                           }
                           put64(F.r + c, r, has1);
                           put64(F.u + c, make_double2(q.own[1].x + q.c.x, q.own[1].y + q.c.y), has1);
                           put64(dst + c, make_double2(fma(ca, q.c.x, cb * r.x), fma(ca, q.c.y, cb * r.y)), has1);
                         }
                       },
                       [&]() {
                         if (last) add_lanes(sum, acc);
                         acc = 0.0;
                       });
      if (!last && !grid_barrier(whole_grid(), &sc->bar, L.target)) return;
    }
    if (!grid_sum<1>(whole_grid(), S.sum, &sc->bar, A.sums, sum, L.target, L.set, [&](double rrn) {
          const double b = ddiv(rrn, rro);  // PPCG.jl:89-92
          const bool cv = test.met(rrn);
          if ((threadIdx.x & 31) == 0) {
            S.a = b;
            S.b = rrn;
            S.conv = cv;
            S.done = cv || iter + 1 >= maxiters;
          }
        }))
      return;
    beta = S.a;
    rro = S.b;
    L.mirrored = !L.mirrored;
    ++iter;
    ++outer;
    if (S.done) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->alpha = alpha;
    sc->pw = pw;
    sc->beta = beta;
    sc->rro = rro;
    sc->error = rro;
    sc->iter = iter;
    sc->cheby_iters = outer;
    sc->first = 0;
    sc->converged = S.conv;
    sc->done = 1;
  }
}

// ---- Jacobi ------------------------------------------------------------------

// One sweep of a row: u' = (u0 + sum k u) / (1 + sum k), diag holding the reciprocal.
__device__ __forceinline__ double2 jacobi_row(const Row64 &q, bool has1) {
  double a = fma(q.kx.y, has1 ? q.c.y : q.c.x, q.own[0].x), b = fma(q.kxe, q.e, q.own[0].y);
  a = fma(q.kx.x, q.w, a);
  b = fma(q.kx.y, q.c.x, b);
  a = fma(q.kyn.x, q.n.x, a);
  b = fma(q.kyn.y, q.n.y, b);
  a = fma(q.ky.x, q.s.x, a) * q.dg.x;
  b = fma(q.ky.y, q.s.y, b) * q.dg.y;
  return make_double2(a, b);
}
__device__ __forceinline__ double add_change(double acc, double2 now, double2 before, bool has1) {
  acc = dadd(acc, fabs(dsub(now.x, before.x)));
  return has1 ? dadd(acc, fabs(dsub(now.y, before.y))) : acc;
}
// u0 - A u of a row, in the exact path's order.
__device__ __forceinline__ double2 residual_row(const Row64 &q, bool has1) {
  const Nbr c0 = {q.c.x, has1 ? q.c.y : q.c.x, q.w, q.n.x, q.s.x, q.kx.x, q.kx.y, q.ky.x, q.kyn.x, 0.0};
  const Nbr c1 = {q.c.y, q.e, q.c.x, q.n.y, q.s.y, q.kx.y, q.kxe, q.ky.y, q.kyn.y, 0.0};
  return make_double2(dsub(q.own[0].x, apply_a<true>(c0)), dsub(q.own[0].y, apply_a<true>(c1)));
}

__global__ void __launch_bounds__(WARPS64 * 32, 1) k_jacobi64(const Loop64 A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ SharedLoop S;
  const Fields &F = A.F;
  DevScalars *sc = F.sc;
  LoopState L;
  L.ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING64_BYTES;
  const LoopTest test(sc);
  const int maxiters = sc->maxiters, lane = threadIdx.x & 31;
  int iter = sc->iter;
  double error = sc->error;
  double *u = F.u, *un = F.ub;
  bool checked = false;
  for (;;) {
    double acc = 0.0;
    Digits sum;
    ring64<false, 1>(whole_grid(), ring_of(A, u, F.u0, nullptr), A.t, L.ring, L.mirrored, &A.F.sc->bar.next_tile, L.handed,
                     [&](int j, int i0, bool has1, bool owns, const Row64 &q) {
                       const double2 v = jacobi_row(q, has1);
                       if (owns) {
                         acc = add_change(acc, v, q.c, has1);
                         put64(un + A.g.at(i0, j), v, has1);
                       }
                     },
                     [&]() {
                       add_lanes(sum, acc);
                       acc = 0.0;
                     });
    ++iter;
    checked = iter % 50 == 0;
    if (!grid_sum<1>(whole_grid(), S.sum, &sc->bar, A.sums, sum, L.target, L.set, [&](double e) {
          const bool cv = !checked && test.met(e);
          if (lane == 0) {
            S.a = e;
            S.conv = cv;
            S.done = !checked && (cv || iter >= maxiters);
          }
        }))
      return;
    error = S.a;
    L.mirrored = !L.mirrored;
    double *t = u;
    u = un;
    un = t;
    if (checked) {  // every 50th sweep r = u0 - A u joins the error (Jacobi.jl:16-21)
      sum = Digits{};
      ring64<false, 1>(whole_grid(), ring_of(A, u, F.u0, nullptr), A.t, L.ring, L.mirrored, &A.F.sc->bar.next_tile, L.handed,
                       [&](int j, int i0, bool has1, bool owns, const Row64 &q) {
                         const double2 r = residual_row(q, has1);
                         if (owns) {
                           put64(F.r + A.g.at(i0, j), r, has1);
                           acc = dadd(acc, dmul(r.x, r.x));
                           if (has1) acc = dadd(acc, dmul(r.y, r.y));
                         }
                       },
                       [&]() {
                         add_lanes(sum, acc);
                         acc = 0.0;
                       });
      if (!grid_sum<1>(whole_grid(), S.sum, &sc->bar, A.sums, sum, L.target, L.set, [&](double rr) {
            const double e = dadd(error, rr);
            const bool cv = test.met(e);
            if (lane == 0) {
              S.a = e;
              S.conv = cv;
              S.done = cv || iter >= maxiters;
            }
          }))
        return;
      L.mirrored = !L.mirrored;
    }
    error = S.a;
    if (S.done) break;
  }
  // r .= u copies the last sweep's input, its depth-1 halo (the reflection)
  // included; after a check the interior holds the residual.  u ends in its own
  // buffer, with its halo.
  const int nx = A.g.nx, ny = A.g.ny, chunks = (nx + 31) / 32, warps = gridDim.x * WARPS64;
  const long long n = (long long)chunks * ny;
  for (long long k = blockIdx.x * WARPS64 + (threadIdx.x >> 5); k < n; k += warps) {
    const int j = (int)(k / chunks), i = (int)(k % chunks) * 32 + lane;
    if (i >= nx) continue;
    const size_t c = A.g.at(i, j);
    const double v = __ldcg(un + c);
    if (!checked) F.r[c] = v;
    put_faces(F.r, A.g, c, i, j, v);
    const double uv = __ldcg(u + c);
    if (u != F.u) F.u[c] = uv;
    put_faces(F.u, A.g, c, i, j, uv);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->error = error;
    sc->iter = iter;
    sc->converged = S.conv;
    sc->done = 1;
  }
}

// Jacobi on a deck whose rows fit the grid at once, two sweeps a grid barrier.
// A block keeps up to RES_ROWS rows of one strip: the operands in registers, u
// in shared memory, where it makes the first sweep of a pair for one more row
// on each side and two more columns; from memory come the four rows
// and the edge lanes that the neighbours made, before each pair.
//
// What a sweep of a small deck costs is a grid barrier with its reduction and
// the latency of its loads, which the pair has once and the operands not at
// all; 28 FP64 instructions a row and pair, 10 for each of the two more.
// A sweep: 250^2 3.5 us against 4.7 swept one by one (k_jacobi64), 100^2 2.6 against
// 3.9, 400^2 5.0 against 9.1; of 6.9 us a pair at 250^2, 1.2 wait at the barrier and 1.8
// add up its sums.
constexpr int RES_ROWS = 30;  // two rows a warp with those on the sides

struct Jacobi64 {
  Fields F;
  Geom g;
  GridSums *sums;
  int strips, rows;
};

__global__ void __launch_bounds__(WARPS64 * 32, 1) k_jacobi64_resident(const Jacobi64 A) {
  __shared__ double2 su[RES_ROWS + 4][32];  // u, from row j0 - 2
  __shared__ double2 ss[RES_ROWS + 2][32];  // the first sweep's, from row j0 - 1
  __shared__ SharedLoop S;
  const Fields &F = A.F;
  const Geom &g = A.g;
  DevScalars *sc = F.sc;
  const LoopTest test(sc);
  const int maxiters = sc->maxiters, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nx = g.nx, ny = g.ny;
  const int strip = blockIdx.x % A.strips, j0 = blockIdx.x / A.strips * A.rows, j1 = min(j0 + A.rows, ny);
  const int i0 = strip * STRIP64 - 2 + 2 * lane;
  const bool in = i0 >= 0 && i0 < nx, has1 = i0 + 1 < nx, owns = in && lane >= 1 && lane <= 30;
  Row64 q[2];
  bool made[2], own[2];  // this warp makes the row's first sweep; its second
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int row = j0 - 1 + warp + WARPS64 * m;
    made[m] = row >= 0 && row < ny && row <= j1;
    own[m] = row >= j0 && row < j1;
    const double2 zero = make_double2(0.0, 0.0);
    q[m].kx = q[m].ky = q[m].kyn = q[m].dg = q[m].own[0] = zero;
    if (made[m] && i0 >= 0 && i0 <= nx) q[m].kx = ld2(F.kx + g.at(i0, row));  // the first halo column closes the last cell
    if (made[m] && in) {
      const size_t c = g.at(i0, row);
      q[m].ky = ld2(F.ky + c);
      q[m].kyn = ld2(F.ky + c + g.pitch);
      q[m].dg = ld2(F.diag + c);
      q[m].own[0] = ld2(F.u0 + c);
    }
    q[m].kxe = __shfl_down_sync(FULL, q[m].kx.x, 1);
  }
  // u's rows from memory: the neighbours' cells, or all
  auto fetch = [&](const double *u, bool all) {
    for (int k = warp; k < j1 - j0 + 4; k += WARPS64) {
      const int row = j0 - 2 + k;
      if (row < 0 || row >= ny) continue;
      if (all || row < j0 || row >= j1 || lane == 0 || lane == 31) {
        double2 v = in ? __ldcg(reinterpret_cast<const double2 *>(u + g.at(i0, row))) : make_double2(0.0, 0.0);
        if (!has1) v.y = 0.0;
        su[k][lane] = v;
      }
    }
    __syncthreads();
  };
  // the neighbours of a row's cells: `f` holds the rows from `first` on
  auto around = [&](Row64 &o, int row, const double2 (*f)[32], int first) {
    const double2(*r)[32] = f + (row - first);
    o.c = r[0][lane];
    o.s = row == 0 ? o.c : r[-1][lane];
    o.n = row == ny - 1 ? o.c : r[1][lane];
    o.e = __shfl_down_sync(FULL, o.c.x, 1);
    o.w = __shfl_up_sync(FULL, o.c.y, 1);
    if (i0 + 2 >= nx) o.e = o.c.y;
    if (i0 == 0) o.w = o.c.x;
  };
  int iter = sc->iter;
  double error = sc->error;
  double *u = F.u, *un = F.ub;
  unsigned target = 0, set = 0;
  bool checked = false;
  fetch(u, true);
  for (;;) {
    double acc1 = 0.0, acc2 = 0.0;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int row = j0 - 1 + warp + WARPS64 * m;
      if (!made[m]) continue;
      around(q[m], row, su, j0 - 2);
      double2 v = jacobi_row(q[m], has1);
      if (!has1) v.y = 0.0;
      if (owns && own[m]) acc1 = add_change(acc1, v, q[m].c, has1);
      ss[row - j0 + 1][lane] = v;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int row = j0 - 1 + warp + WARPS64 * m;
      if (!own[m]) continue;
      around(q[m], row, ss, j0 - 1);
      double2 v = jacobi_row(q[m], has1);
      if (!has1) v.y = 0.0;
      if (owns) {
        acc2 = add_change(acc2, v, q[m].c, has1);
        put64(un + g.at(i0, row), v, has1);
        su[row - j0 + 2][lane] = v;
      }
    }
    // Pairs start at even counts, so that the sweeps checked (every 50th) are their second.
    checked = (iter + 2) % 50 == 0;
    Digits s1, s2;
    add_lanes(s1, acc1);
    add_lanes(s2, acc2);
    const Digits both = lane < 8 ? s1 : lane < 16 ? s2 : Digits{};
    if (!grid_sum<3>(whole_grid(), S.sum, &sc->bar, A.sums, both, target, set, [&](double e1, double e2, double) {
          const bool met1 = test.met(e1), first = met1 || iter + 1 >= maxiters;
          const bool cv = first ? met1 : !checked && test.met(e2);
          if (lane == 0) {
            S.a = first ? e1 : e2;
            S.first = first;
            S.conv = cv;
            S.done = first || (!checked && (cv || iter + 2 >= maxiters));
          }
        }))
      return;
    error = S.a;
    if (S.first) {  // the first sweep ends it
      ++iter;
      checked = false;
      break;
    }
    iter += 2;
    double *t = u;
    u = un;
    un = t;
    if (!S.done) fetch(u, false);
    if (checked) {  // every 50th sweep r = u0 - A u joins the error (Jacobi.jl:16-21)
      double acc = 0.0;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int row = j0 - 1 + warp + WARPS64 * m;
        if (!own[m]) continue;
        around(q[m], row, su, j0 - 2);
        const double2 r = residual_row(q[m], has1);
        if (owns) {
          put64(F.r + g.at(i0, row), r, has1);
          acc = dadd(acc, dmul(r.x, r.x));
          if (has1) acc = dadd(acc, dmul(r.y, r.y));
        }
      }
      Digits sum;
      add_lanes(sum, acc);
      if (!grid_sum<1>(whole_grid(), S.sum, &sc->bar, A.sums, sum, target, set, [&](double rr) {
            const double e = dadd(error, rr);
            const bool cv = test.met(e);
            if (lane == 0) {
              S.a = e;
              S.conv = cv;
              S.done = cv || iter >= maxiters;
            }
          }))
        return;
      error = S.a;
    }
    if (S.done) break;
  }
  // u, and r .= u, the last sweep's input, with the reflection about it; after
  // a check r's interior holds the residual
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int row = j0 - 1 + warp + WARPS64 * m;
    if (!own[m] || !owns) continue;
    const size_t c = g.at(i0, row);
    const double2 s = ss[row - j0 + 1][lane];
    const double2 v = S.first ? __ldcg(reinterpret_cast<const double2 *>(u + c)) : s;
    const double2 z = S.first ? s : su[row - j0 + 2][lane];
    put64(F.u + c, z, has1);
    if (!checked) put64(F.r + c, v, has1);
    put_faces(F.u, g, c, i0, row, z.x);
    put_faces(F.r, g, c, i0, row, v.x);
    if (has1) {
      put_faces(F.u, g, c + 1, i0 + 1, row, z.y);
      put_faces(F.r, g, c + 1, i0 + 1, row, v.y);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->error = error;
    sc->iter = iter;
    sc->converged = S.conv;
    sc->done = 1;
  }
}

// Rows a block for a deck of the resident kernel, or 0: the fewest FP64
// instructions on a quarter of an SM, with a barrier's time (some 40 of them)
// against one block alone.
int resident_rows(const Geom &g, int blocks) {
  const int strips = (g.nx + STRIP64 - 1) / STRIP64;
  int best = 0, cost = 0;
  for (int rows = 1; rows <= RES_ROWS; ++rows) {
    const long long n = (long long)strips * ((g.ny + rows - 1) / rows);
    if (n > blocks) continue;
    const int c = 14 * ((rows + 5) / 4 + (rows + 3) / 4) + (n > 1 ? 40 : 0);
    if (!best || c < cost) {
      best = rows;
      cost = c;
    }
  }
  return best;
}

}  // namespace
}  // namespace tl

using namespace tl;

// One of the loops from the state its solver has set up; the scalars are read
// back.  One launch.
static int run_loop(tl_ctx *ctx, const void *kernel, int blocks, void *args, size_t smem, double *ms) {
  CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int rc = tl_bar_ready(ctx);
  if (rc) return rc;
  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  void *argv[] = {args};
  CK(cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(WARPS64 * 32), argv, smem, ctx->stream));
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  ctx->launches += 1;
  if ((rc = tl_read_scalars(ctx))) return rc;
  float t = 0.f;
  CK(cudaEventElapsedTime(&t, ctx->ev0, ctx->ev1));
  if (ms) *ms += t;
  return tl_persist_check(ctx);
}

// `which` is TL_GRAPH_CHEBY_EXACT, TL_GRAPH_PPCG_EXACT or TL_GRAPH_JACOBI.
int tl_loop64_run(tl_ctx *ctx, int which, int ninner, double *ms) {
  const int blocks = persist_blocks(ctx->sm_count);
  GridSums *sums = static_cast<GridSums *>(ctx->grid_sums);
  const int rows = which == TL_GRAPH_JACOBI ? resident_rows(ctx->g, blocks) : 0;
  if (rows) {
    Jacobi64 J{ctx->F, ctx->g, sums, (ctx->g.nx + STRIP64 - 1) / STRIP64, rows};
    return run_loop(ctx, (const void *)k_jacobi64_resident, J.strips * ((ctx->g.ny + rows - 1) / rows), &J, 0, ms);
  }
  Loop64 A;
  A.F = ctx->F;
  A.g = ctx->g;
  A.sums = sums;
  A.ninner = ninner;
  const void *kernel = which == TL_GRAPH_CHEBY_EXACT  ? (const void *)k_cheby64
                       : which == TL_GRAPH_PPCG_EXACT ? (const void *)k_ppcg64
                                                      : (const void *)k_jacobi64;
  // a row holds the FP64 pipe for 14 to 20 instructions of 64 cycles; see cg64_tilings for the rule
  const TileCost sweep{0.1, 1200.0, 1500.0, 1150.0, 200.0, 16, 48, 4}, each{0.0, 500.0, 1000.0, 400.0, 150.0, 0, 24, 8};
  A.t = make_tiling(ctx->g.nx, ctx->g.ny, STRIP64, sweep, blocks, WARPS64);
  A.te = make_tiling_on(A.t, ctx->g.nx, ctx->g.ny, 64, each, WARPS64);
  return run_loop(ctx, kernel, A.t.blocks, &A, (size_t)RING64_BYTES * WARPS64, ms);
}
