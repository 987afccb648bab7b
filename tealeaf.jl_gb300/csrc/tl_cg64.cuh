// tl_cg64.cuh -- the fused FP64 CG loop (tealeaf semantics, src/solvers/CG.jl:
// 17-28, 82-104) for persistent kernels: one deck (tl_cg64.cu) or a batch
// (tl_batch.cu).  Per iteration, with a grid
// reduction after each pass:
//     W:  p' = beta p + r,  w = A p',  p'.w,  and u += alpha p of the step before
//     R:  r -= alpha w,  r.r
// u is updated one pass late, where p is read anyway: 96 B per cell and
// iteration instead of 104, and the two passes are nearer balance, W bound by
// the FP64 pipe (9 instructions a cell), R by memory.
//
// 18-21 us an iteration on any deck up to 512^2 went into kernel boundaries
// and the while-node of the graph this replaces.
#pragma once

#include "tl_march.cuh"
#include "tl_ring64.cuh"
#include "tl_solvers.h"

namespace tl {
namespace {

struct Cg64 {
  Fields F;
  Geom g;
  Tiling tw, tr;  // W (strips of 60 columns), R (64)
  GridSums *sums;
  int check;  // the relative test before the first iteration
  int keep;   // every warp has one tile of KEEP_ROWS rows at most: R works on what W left in shared memory
};

// Small decks: with one row a warp, r is still in W's ring and w goes beside it, so
// that R waits for no load and w for no store: 7.2 us an iteration at 64^2 against
// 7.9, 8.4 against 8.9 at 256^2.  With two rows a warp it gained nothing (12.9 both
// ways at 512^2).
constexpr int KEEP_ROWS = 1, KEEP_BYTES = KEEP_ROWS * 512;
constexpr int CG64_SMEM = WARPS64 * (RING64_BYTES + KEEP_BYTES);
// This warp's ring, and where it keeps w.
struct Mem64 {
  unsigned ring, w;
  __device__ __forceinline__ explicit Mem64(const void *smem) {
    const unsigned base = (unsigned)__cvta_generic_to_shared(smem), warp = threadIdx.x >> 5;
    ring = base + warp * RING64_BYTES;
    w = base + WARPS64 * RING64_BYTES + warp * KEEP_BYTES;
  }
};

struct Shared64 {
  SumShared sum;
  double alpha, beta, err, inv_rro;
  int done, conv, sw;
};

// r -= alpha w over this warp's tiles; its share of r.r.
template <bool LATE>
__device__ __forceinline__ Digits r_pass(Grid grid, const Cg64 &A, unsigned ring, bool mirrored, double alpha,
                                         unsigned &handed) {
  constexpr int DEPTH = RING64_BYTES / 1024;
  const int nx = A.g.nx, ny = A.g.ny, lane = threadIdx.x & 31;
  const unsigned slot0 = ring + 16 * lane;
  Digits sum;
  double acc = 0.0;
  TileWalk walk(grid, A.tr, ny, mirrored, &A.F.sc->bar.next_tile, handed);
  handed += walk.requests();
  bool any = false;
  while (walk.valid()) {
    int strip, j0, j1;
    walk.place(strip, j0, j1);
    const unsigned asked = walk.ask();
    const int i0 = strip * 64 + 2 * lane;
    const bool in = i0 < nx, has1 = i0 + 1 < nx;
    const size_t c0 = in ? A.g.at(i0, j0) : (size_t)A.g.hd, step = in ? (size_t)A.g.pitch : 0;
    size_t nxt = c0, c = c0;
    auto issue = [&](int row, unsigned slot) {
      if (row < j1) {
        cp16(slot0 + slot * 1024, A.F.r + nxt, in);
        cp16(slot0 + slot * 1024 + 512, A.F.w + nxt, in);
      }
      nxt += step;
      cp_commit();
    };
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) issue(j0 + d, d);
    if (LATE && any) add_lanes(sum, acc);  // of the tile before
    any = true;
    acc = 0.0;
    unsigned slot = 0, prev = DEPTH - 1;
    for (int j = j0; j < j1; ++j) {
      cp_wait<DEPTH - 2>();
      double2 r = lds2d(slot0 + slot * 1024);
      const double2 w = lds2d(slot0 + slot * 1024 + 512);
      r = make_double2(fma(-alpha, w.x, r.x), fma(-alpha, w.y, r.y));
      if (!has1) r.y = 0.0;
      if (in) {
        acc = fma(r.x, r.x, fma(r.y, r.y, acc));
        put64(A.F.r + c, r, has1);
      }
      c += step;
      issue(j + DEPTH - 1, prev);
      prev = slot;
      slot = slot + 1 == DEPTH ? 0 : slot + 1;
    }
    cp_wait<0>();
    if (!LATE) add_lanes(sum, acc);
    walk.take(asked);
  }
  if (LATE && any) add_lanes(sum, acc);
  return sum;
}

// The same on the one tile (j0 < 0: none) that this warp's W left in shared memory,
// in a ring of `arrays` operands a row.
__device__ __forceinline__ Digits r_kept(const Cg64 &A, const Mem64 &mem, int strip, int j0, int j1, int arrays,
                                         double alpha) {
  const int lane = threadIdx.x & 31;
  Digits sum;
  if (j0 < 0) return sum;
  const int i0 = strip * STRIP64 - 2 + 2 * lane;
  const bool owns = lane >= 1 && lane <= 30 && i0 < A.g.nx, has1 = i0 + 1 < A.g.nx;
  double acc = 0.0;
  for (int j = j0; owns && j < j1; ++j) {
    double2 r = lds2d(mem.ring + 16 * lane + ((j - j0 + 1) * arrays + 1) * 512);
    const double2 w = lds2d(mem.w + 16 * lane + (j - j0) * 512);
    r = make_double2(fma(-alpha, w.x, r.x), fma(-alpha, w.y, r.y));
    if (!has1) r.y = 0.0;
    acc = fma(r.x, r.x, fma(r.y, r.y, acc));
    put64(A.F.r + A.g.at(i0, j), r, has1);
  }
  add_lanes(sum, acc);
  return sum;
}

// HANDED: W's tiles are handed out (and R's, if they are more than the warps).
template <bool KEEP, bool HANDED>
__device__ __forceinline__ bool cg64_loop(Grid grid, const Cg64 &A, Shared64 &S, const Mem64 &mem) {
  const unsigned ring = mem.ring;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool lead = grid.id == 0 && threadIdx.x == 0;
  DevScalars *sc = A.F.sc;
  GridBar *bar = &sc->bar;
  const double bb = sc->bb, eps = sc->eps, epslim = sc->epslim;
  const int maxiters = sc->maxiters, presteps = sc->presteps, errorswitch = sc->errorswitch, rule = sc->switch_rule;
  const bool relative = sc->crit == TL_CRIT_RELATIVE, rooted = relative || rule == 0;
  if (A.check && sqrt(bb > 0 ? ddiv(sc->rro, bb) : sc->rro) < eps) return true;
  const RootTest test(eps, relative ? bb : 1.0);
  double *p = A.F.p, *pn = A.F.pb;
  double rro = sc->rro, alpha = 0.0, beta = 0.0, pw = 0.0;
  int iter = sc->iter;
  bool first = true, mirrored = false;
  unsigned target = 0, set = 0, handed = 0;
  int tile0 = -1, tile1 = -1, tile_strip = 0;  // with `keep`, this warp's tile
  if (KEEP) {
    const TileWalk walk(grid, A.tw, A.g.ny, false, nullptr, 0);
    if (walk.valid()) walk.place(tile_strip, tile0, tile1);
  }
  for (;;) {
    // W
    Ring64 q;
    q.g = A.g;
    q.m = p;
    q.m2 = A.F.r;
    q.kx = A.F.kx;
    q.ky = A.F.ky;
    q.dg = A.F.diag;
    q.own[0] = q.own[1] = A.F.u;
    q.beta = beta;
    q.m_valid = !first;  // the first direction is r
    double acc = 0.0;
    Digits sum;
    auto tile_end = [&]() {
      add_lanes(sum, acc);
      acc = 0.0;
    };
    const int arrays = first ? 5 : 6;
    auto direction = [&](int j, int i0, bool has1, bool owns, const Row64 &o) {
      const double2 w = apply64(o, has1);
      if (owns) {
        const size_t c = A.g.at(i0, j);
        acc = fma(w.y, o.c.y, fma(w.x, o.c.x, acc));
        if (KEEP) sts2d(mem.w + 16 * lane + (j - tile0) * 512, w);
        else put64(A.F.w + c, w, has1);
        put64(pn + c, o.c, has1);
      }
    };
    if (first) {
      ring64<true, 0, HANDED>(grid, q, A.tw, ring, mirrored, &A.F.sc->bar.next_tile, handed, direction, tile_end);
    } else {
      ring64<true, 1, HANDED>(grid, q, A.tw, ring, mirrored, &A.F.sc->bar.next_tile, handed,
                      [&](int j, int i0, bool has1, bool owns, const Row64 &o) {
                        direction(j, i0, has1, owns, o);
                        if (owns)
                          put64(A.F.u + A.g.at(i0, j),
                                make_double2(fma(alpha, o.raw.x, o.own[0].x), fma(alpha, o.raw.y, o.own[0].y)), has1);
                      },
                      tile_end);
    }
    if (!grid_sum<1>(grid, S.sum, bar, A.sums, sum, target, set, [&](double pw) {
          const double a = ddiv(lane == 0 ? rro : 1.0, lane == 0 ? pw : rro);  // and 1/rro for beta, in one division
          if (lane == 0) {
            S.alpha = a;
            S.err = pw;
          } else if (lane == 1) {
            S.inv_rro = a;
          }
          if (lead && iter < maxiters) A.F.cgalpha[iter + 1] = a;  // table holds maxiters + 2 entries
        }))
      return false;
    alpha = S.alpha;
    pw = S.err;
    mirrored = !mirrored && !KEEP;
    {
      double *t = p;
      p = pn;
      pn = t;
    }
    // R
    sum = KEEP ? r_kept(A, mem, tile_strip, tile0, tile1, arrays, alpha) : r_pass<HANDED>(grid, A, ring, mirrored, alpha, handed);
    if (!grid_sum<1>(grid, S.sum, bar, A.sums, sum, target, set, [&](double rrn) {
          // rrn / rro from the reciprocal formed before, with one correction (Markstein's), away from its ends
          double b = rrn * S.inv_rro;
          if (rro > 1e-290 && rro < 1e290) b = fma(fma(-b, rro, rrn), S.inv_rro, b);
          else b = ddiv(rrn, rro);
          const bool conv = rooted ? test.met(rrn) : below(rrn, eps);
          bool sw = false;
          if (!conv && rule == 1) {  // Cheby.jl:25-29, PPCG.jl:27-31
            const int tt = iter + 2;
            sw = errorswitch ? (rrn < epslim) && (tt > CGEIGENITERS) : (tt > presteps) && (rrn < ERROR_SWITCH_MAX);
          }
          if (lane == 0) {
            S.beta = b;
            S.err = rrn;
            S.conv = conv;
            S.sw = sw;
            S.done = conv || sw || iter + 1 >= maxiters;
          }
          if (lead && iter < maxiters) A.F.cgbeta[iter + 1] = b;
        }))
      return false;
    beta = S.beta;
    rro = S.err;
    mirrored = !mirrored && !KEEP;
    first = false;
    ++iter;
    if (S.done) break;
  }
  if (KEEP && tile0 >= 0) {  // the last step's w
    for (int j = tile0; j < tile1; ++j) {
      const int i0 = tile_strip * STRIP64 - 2 + 2 * lane;
      if (lane >= 1 && lane <= 30 && i0 < A.g.nx)
        put64(A.F.w + A.g.at(i0, j), lds2d(mem.w + 16 * lane + (j - tile0) * 512), i0 + 1 < A.g.nx);
    }
  }
  // the last step's u, and p! of the next one (CG.jl:22), with their halo
  const int nx = A.g.nx, ny = A.g.ny, chunks = (nx + 63) / 64;
  const int warps = grid.nb * WARPS64;
  const long long n = (long long)chunks * ny;
  for (long long k = grid.id * WARPS64 + warp; k < n; k += warps) {
    const int j = (int)(k / chunks), i0 = (int)(k % chunks) * 64 + 2 * lane;
    if (i0 >= nx) continue;
    const size_t c = A.g.at(i0, j);
    auto ld = [&](const double *f) { return __ldcg(reinterpret_cast<const double2 *>(f + c)); };
    const double2 pv = ld(p), rv = ld(A.F.r), uv = ld(A.F.u);
    const double2 un = make_double2(fma(alpha, pv.x, uv.x), fma(alpha, pv.y, uv.y));
    const double2 pw = make_double2(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
    put64(A.F.u + c, un, i0 + 1 < nx);
    put64(A.F.p + c, pw, i0 + 1 < nx);
    if (j == 0 || j == ny - 1 || i0 == 0 || i0 + 2 >= nx) {
      put_faces(A.F.u, A.g, c, i0, j, un.x);
      put_faces(A.F.p, A.g, c, i0, j, pw.x);
      if (i0 + 1 < nx) {
        put_faces(A.F.u, A.g, c + 1, i0 + 1, j, un.y);
        put_faces(A.F.p, A.g, c + 1, i0 + 1, j, pw.y);
      }
    }
  }
  if (lead) {
    sc->alpha = alpha;
    sc->beta = beta;
    sc->pw = pw;
    sc->rrn = rro;
    sc->rro = rro;
    sc->error = rro;
    sc->iter = iter;
    sc->first = 0;
    sc->converged = S.conv;
    sc->switched = S.sw;
    sc->done = 1;
  }
  return true;
}

// The loop on one deck by the blocks of `grid`; false when a wait gave up.
__device__ __forceinline__ bool cg64_solve(Grid grid, const Cg64 &A, Shared64 &S, const Mem64 &mem) {
  if (A.keep) return cg64_loop<true, false>(grid, A, S, mem);
  return A.tw.handed ? cg64_loop<false, true>(grid, A, S, mem) : cg64_loop<false, false>(grid, A, S, mem);
}

// Tilings for `blocks` blocks at most.
inline void cg64_tilings(Cg64 &A, int blocks) {
  // A row of W holds the FP64 pipe for 17 x 64 cycles, of R for 4 x 64.  W's
  // shares are even up to 48 rows a warp: there its tiles are the coarser, the
  // better (92 us an iteration at 2048^2 against 110 with tiles handed
  // out); beyond, what the SMs get of HBM differs (326 against 401 at 4096^2).
  const TileCost w{0.25, 1100.0, 1500.0, 1100.0, 200.0, 16, 48, 4}, r{0.0, 300.0, 1000.0, 260.0, 150.0, 0, 24, 8};
  A.tw = make_tiling(A.g.nx, A.g.ny, STRIP64, w, blocks, WARPS64);
  A.tr = make_tiling_on(A.tw, A.g.nx, A.g.ny, 64, r, WARPS64);
  A.keep = !A.tw.handed && A.tw.tiles <= A.tw.warps && A.tw.rows <= KEEP_ROWS;
}

}  // namespace
}  // namespace tl
