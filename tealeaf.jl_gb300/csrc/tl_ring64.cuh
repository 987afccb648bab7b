// tl_ring64.cuh -- the FP64 row marcher of the persistent kernels: every
// five-point pass (CG's direction step, Chebyshev, PPCG's sweeps, Jacobi) over
// the tiles a warp takes, with all operands copied rows ahead into the warp's
// ring in shared memory.
//
// A warp owns strips of 60 columns, two cells a lane in lanes 1..30; lanes 0 and
// 31 hold the neighbouring strips' cells.  What bounds these passes is the FP64
// pipe: an instruction holds it for 64 cycles whatever its active lanes, so a
// value that only the edge lanes need (the other form, 64 columns with edge
// loads) costs as much as one that all need: 2 instructions in 16 per row of
// the CG direction step, against 2 lanes in 32 here.
#pragma once

#include "tl_persist.cuh"

namespace tl {

constexpr int STRIP64 = 60;
constexpr int WARPS64 = 16;          // four a sub-partition: with two, waits on the pipe's results left it 56 % busy (1536^2)
constexpr int RING64_BYTES = 12288;  // ring of one warp: 4 rows of six operands

struct Ring64 {
  Geom g;
  const double *m, *m2;      // the stencil's field, or the two that make it (value = beta m + m2)
  const double *kx, *ky, *dg;
  const double *own[2];      // operands read at the cell alone
  double beta;
  bool m_valid;              // false: m counts as zero
};

// What `body` gets of one row: its two cells' inputs.
struct Row64 {
  double2 c, s, n;     // the field at the cells, and the rows below and above
  double w, e;         // west of the first cell, east of the second
  double2 kx, ky, kyn, dg;
  double kxe;
  double2 own[2], raw; // raw: m itself
};

// diag*c - kx1*e - kx0*w - ky1*n - ky0*s for both cells.
__device__ __forceinline__ double2 apply64(const Row64 &q, bool has1) {
  double a = q.dg.x * q.c.x, b = q.dg.y * q.c.y;
  a = fma(-q.kx.y, has1 ? q.c.y : q.c.x, a);
  b = fma(-q.kxe, q.e, b);
  a = fma(-q.kx.x, q.w, a);
  b = fma(-q.kx.y, q.c.x, b);
  a = fma(-q.kyn.x, q.n.x, a);
  b = fma(-q.kyn.y, q.n.y, b);
  a = fma(-q.ky.x, q.s.x, a);
  b = fma(-q.ky.y, q.s.y, b);
  return make_double2(a, b);
}

// Runs `body(j, i0, has1, row)` for every row of every tile this warp takes, on
// all lanes (body stores and sums on owner lanes only: `owns`), and
// `tile_end()` after each tile; LATE: once the next tile's first rows are on their way
// (CG where tiles are handed out: 326 us an iteration at 4096^2 against 331; on decks
// of a tile a warp it costs more than it hides).  A neighbour across the domain's
// edge is the cell itself; the second cell of a lane that has only one is zero.
template <bool TWO, int NOWN, bool LATE = false, class Body, class TileEnd>
__device__ __forceinline__ void ring64(Grid grid, const Ring64 &A, const Tiling &T, unsigned ring, bool mirrored, unsigned *next,
                                       unsigned &handed, Body &&body, TileEnd &&tile_end) {
  constexpr int NARR = 4 + TWO + NOWN;
  constexpr int DEPTH = RING64_BYTES / (NARR * 512) < 6 ? RING64_BYTES / (NARR * 512) : 6;
  constexpr int O_KX = 512 * (1 + TWO), O_KY = O_KX + 512, O_DG = O_KY + 512, O_OWN = O_DG + 512;
  const int nx = A.g.nx, ny = A.g.ny;
  const int lane = threadIdx.x & 31;
  const unsigned slot0 = ring + 16 * lane;
  TileWalk walk(grid, T, ny, mirrored, next, handed);
  handed += walk.requests();
  bool any = false;
  while (walk.valid()) {
    int strip, j0, j1;
    walk.place(strip, j0, j1);
    const unsigned asked = walk.ask();
    const int i0 = strip * STRIP64 - 2 + 2 * lane;
    const bool in = i0 >= 0 && i0 < nx, has1 = i0 + 1 < nx, inner = i0 + 2 < nx;
    const bool kin = i0 >= 0 && i0 <= nx;  // kx of the first halo column closes the last cell
    const bool owns = in && lane >= 1 && lane <= 30;
    // a copy that reads nothing still needs a 16-byte aligned address: cell 0 of the first row
    const size_t step = kin ? (size_t)A.g.pitch : 0;
    size_t nxt = kin ? (size_t)((long long)A.g.at(i0, 0) + (long long)(j0 - 1) * A.g.pitch) : (size_t)A.g.hd;
    auto issue = [&](int row, unsigned slot) {
      if (row <= j1 && row >= 0) {  // row ny exists: the halo row, read for ky
        const unsigned a = slot0 + slot * (NARR * 512);
        if (row < ny) {
          cp16(a, A.m + nxt, in && A.m_valid);
          if (TWO) cp16(a + 512, A.m2 + nxt, in);
        }
        if (row >= j0) {
          cp16(a + O_KY, A.ky + nxt, in);
          if (row < j1) {
            cp16(a + O_KX, A.kx + nxt, kin);
            cp16(a + O_DG, A.dg + nxt, in);
#pragma unroll
            for (int o = 0; o < NOWN; ++o) cp16(a + O_OWN + 512 * o, A.own[o] + nxt, owns);
          }
        }
      }
      nxt += step;
      cp_commit();
    };
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) issue(j0 - 1 + d, d);
    if (LATE && any) tile_end();
    any = true;
    Row64 q;
    q.s = q.c = make_double2(0.0, 0.0);
    q.ky = q.c;
    unsigned slot = 0, prev = DEPTH - 1;
    for (int row = j0 - 1; row <= j1; ++row) {
      cp_wait<DEPTH - 2>();
      const unsigned a = slot0 + slot * (NARR * 512);
      if (row >= 0 && row < ny) {
        const double2 m = lds2d(a);
        q.n = m;
        if (TWO) {
          const double2 r = lds2d(a + 512);
          q.n = make_double2(fma(A.beta, m.x, r.x), fma(A.beta, m.y, r.y));
        }
        if (!has1) q.n.y = 0.0;
      } else {
        q.n = q.c;
      }
      q.kyn = row >= j0 ? lds2d(a + O_KY) : make_double2(0.0, 0.0);
      const int j = row - 1;
      if (j >= j0) {
        const unsigned b = slot0 + prev * (NARR * 512);
        q.kx = lds2d(b + O_KX);
        q.dg = lds2d(b + O_DG);
        q.raw = lds2d(b);
#pragma unroll
        for (int o = 0; o < NOWN; ++o) q.own[o] = lds2d(b + O_OWN + 512 * o);
        q.kxe = __shfl_down_sync(FULL, q.kx.x, 1);
        q.e = __shfl_down_sync(FULL, q.c.x, 1);
        q.w = __shfl_up_sync(FULL, q.c.y, 1);
        if (!inner) q.e = q.c.y;
        if (i0 == 0) q.w = q.c.x;
        if (j == 0) q.s = q.c;
        body(j, i0, has1, owns, q);
      }
      q.s = q.c;
      q.c = q.n;
      q.ky = q.kyn;
      issue(row + DEPTH - 1, prev);  // its last reader was this trip
      prev = slot;
      slot = slot + 1 == DEPTH ? 0 : slot + 1;
    }
    cp_wait<0>();
    if (!LATE) tile_end();
    walk.take(asked);
  }
  if (LATE && any) tile_end();
}

// Two cells of a row to memory.
__device__ __forceinline__ void put64(double *p, double2 v, bool has1) {
  if (has1) st2(p, v);
  else *p = v.x;
}

}  // namespace tl
