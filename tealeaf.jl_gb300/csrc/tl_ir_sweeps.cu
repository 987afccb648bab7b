// tl_ir_sweeps.cu -- the FP32 Chebyshev and PPCG iterations inside FP64
// refinement (tealeaf semantics, after the presteps' switch), each as one
// persistent kernel with its refinements.
//
// Chebyshev's steps and PPCG's inner sweeps need no sum between them, so one
// pass over the grid takes two: a warp marches up its strip with the first
// step one row ahead of the second, and forms the first step's result one row
// and one lane beyond its own cells as well.  That halves the bytes (a
// Chebyshev step reads and writes 24 B per cell, two in one pass the same 24; a
// PPCG sweep 28) for a tenth more arithmetic, and halves the grid barriers.
// PPCG's update with its first sweep is such a pass too.  The Chebyshev test on
// r.r is made on both steps' sums after each pair.
//
// What bounds the passes: HBM on large grids, the grid barrier on small ones.
#include <cmath>

#include "tl_ir_cg.cuh"

namespace tl {
namespace {

struct IrSweeps {
  Fields F;
  Geom g;
  G32 g32;
  float *r, *x, *p, *pb, *sd, *sdb;
  const float *iw;
  double delta2;
  Tiling t, t64;
  GridSums *sums;
  int ninner;
  double rr;  // PPCG: the true r.r the presteps ended with
};

// What a pass does; w = A m, the second step's primed by 2:
//   STEP_CHEBY   r1 = R - w1; z1 = a1 z + b1 r1; m1 = m + z1;   r2 = R - w2; z2 = a2 z1 + b2 r2; m2 = m1 + z2
//                (m: the correction e, z: p, R: the refinement's residual; Cheby.jl:88-104)
//   STEP_SWEEP   r1 = R - w1; z += m; m1 = a1 m + b1 r1;        r2 = r1 - w2; z += m1; m2 = a2 m1 + b2 r2
//                (m: sd, z: x, R: r; PPCG.jl:74-88)
//   STEP_UPDATE  r1 = R - a1 w1; z += a1 m; m1 = b1 r1 (m: p', b1 = 1/theta; PPCG.jl:64-72), then a sweep
enum { STEP_CHEBY, STEP_SWEEP, STEP_UPDATE };

struct StepArgs {
  const float *m, *R, *z;
  float *mo, *Ro, *zo;
  float a1, b1, a2, b2;
  bool m_valid, z_valid;  // false: zero
  bool store_m, mirrored;
  float down;  // the sums' scale
};

__device__ __forceinline__ float4 axpy4(float a, float4 x, float4 y) {
  return f4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
__device__ __forceinline__ float4 lin4(float a, float4 x, float b, float4 y) {
  return f4(fmaf(a, x.x, b * y.x), fmaf(a, x.y, b * y.y), fmaf(a, x.z, b * y.z), fmaf(a, x.w, b * y.w));
}
__device__ __forceinline__ float4 add4(float4 x, float4 y) { return f4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w); }
__device__ __forceinline__ float dot4(float4 x, float s) {
  return fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, s))));
}

// w = c + the face sums to the four neighbours, as stencil4.
struct Faces4 {
  float4 e;
  float w;  // the west face of the first cell
};
__device__ __forceinline__ Faces4 faces4(const float (&fe)[4], float4 iw) {
  Faces4 k;
  const float ie = __shfl_down_sync(FULL, iw.x, 1);
  k.e = f4(fe[0] * (iw.x + iw.y), fe[1] * (iw.y + iw.z), fe[2] * (iw.z + iw.w), fe[3] * (iw.w + ie));
  k.w = __shfl_up_sync(FULL, k.e.w, 1);
  return k;
}
__device__ __forceinline__ float4 apply4(float4 c, float4 s, float4 n, const Faces4 &k, float4 ks, float4 kn) {
  const float e = __shfl_down_sync(FULL, c.x, 1), w = __shfl_up_sync(FULL, c.w, 1);
  float4 o;
  o.x = fmaf(ks.x, c.x - s.x, fmaf(kn.x, c.x - n.x, fmaf(k.w, c.x - w, fmaf(k.e.x, c.x - c.y, c.x))));
  o.y = fmaf(ks.y, c.y - s.y, fmaf(kn.y, c.y - n.y, fmaf(k.e.x, c.y - c.x, fmaf(k.e.y, c.y - c.z, c.y))));
  o.z = fmaf(ks.z, c.z - s.z, fmaf(kn.z, c.z - n.z, fmaf(k.e.y, c.z - c.y, fmaf(k.e.z, c.z - c.w, c.z))));
  o.w = fmaf(ks.w, c.w - s.w, fmaf(kn.w, c.w - n.w, fmaf(k.e.z, c.w - c.z, fmaf(k.e.w, c.w - e, c.w))));
  return o;
}
__device__ __forceinline__ float4 face_row(float ryh, float4 a, float4 b) {
  return f4(ryh * (a.x + b.x), ryh * (a.y + b.y), ryh * (a.z + b.z), ryh * (a.w + b.w));
}

// One tile's three sums into the pass's.
template <bool HANDED>
__device__ __forceinline__ void tile_sums(PassSums &S, Pair (&acc)[3]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (lane == 0 || lane == 31) acc[d] = Pair{0.f, 0.f};
  add_tile<HANDED>(S, warp_pairs(acc));
}

// One pass of one or two steps; sums r1.r1 and r2.r2 when `sums`.
template <int KIND, int STEPS, bool HANDED>
__device__ __forceinline__ void step_pass(Grid grid, const IrSweeps &A, const StepArgs &q, unsigned ring, float rxh,
                                          float ryh, bool sums, unsigned &handed, PassSums &S) {
  constexpr int DEPTH = RING_BYTES / 2048;
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
    float fe[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) fe[m] = (i0 + m >= 0 && i0 + m + 1 < nx) ? rxh : 0.f;
    const int lo = STEPS == 2 ? j0 - 1 : j0, hi = STEPS == 2 ? j1 + 1 : j1;  // rows of the first step
    // a copy that reads nothing still needs a 16-byte aligned address: cell 0 of the first row
    const size_t col = in ? A.g32.at(i0, 0) : (size_t)A.g32.hd;
    const size_t step = in ? (size_t)A.g32.pitch : 0;
    size_t next = col + (in ? (long long)(lo - 1) * A.g32.pitch : 0);
    auto issue = [&](int row, unsigned slot) {
      if (row <= hi && row >= 0 && row < ny) {
        const unsigned a = slot0 + slot * 2048;
        cp16(a, q.m + next, in && q.m_valid);
        cp16(a + 512, A.iw + next, in);
        if (row >= lo && row < hi) {
          cp16(a + 1024, q.R + next, in);
          if (KIND == STEP_CHEBY || (row >= j0 && row < j1)) cp16(a + 1536, q.z + next, in && q.z_valid);
        }
      }
      next += step;
      cp_commit();
    };
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) issue(lo - 1 + d, d);
    const float4 zero = f4(0, 0, 0, 0);
    float4 ms = zero, mc = zero, ic = zero, k0 = zero, k1 = zero;  // k1: faces below the first step's row, k0: below the second's
    float4 m1s = zero, m1c = zero, r1c = zero, z1c = zero;
    Faces4 kec{zero, 0.f};
    Pair acc[3] = {};
    float ps[2] = {0.f, 0.f};
    int nrow = 0;
    unsigned slot = 0, prev = DEPTH - 1;
    for (int row = lo - 1; row <= hi; ++row) {
      cp_wait<DEPTH - 2>();
      const unsigned a = slot0 + slot * 2048;
      float4 mn = zero, iwn = zero;
      if (row >= 0 && row < ny) {
        mn = lds4(a);
        iwn = lds4(a + 512);
      }
      float4 kn = zero;
      if (row >= lo && row > 0 && row < ny) kn = face_row(ryh, ic, iwn);
      const int j = row - 1;  // the first step's row
      float4 m1 = zero, r1 = zero, z1 = zero;
      Faces4 ke{zero, 0.f};
      if (j >= lo && j < hi && j >= 0 && j < ny) {
        const unsigned b = slot0 + prev * 2048;
        ke = faces4(fe, ic);
        const float4 w = apply4(mc, ms, mn, ke, k1, kn);
        const float4 R = lds4(b + 1024);
        if (KIND == STEP_UPDATE) {
          r1 = axpy4(-q.a1, w, R);
          m1 = f4(r1.x * q.b1, r1.y * q.b1, r1.z * q.b1, r1.w * q.b1);
        } else {
          r1 = f4(R.x - w.x, R.y - w.y, R.z - w.z, R.w - w.w);
        }
        if (KIND == STEP_CHEBY) {
          z1 = lin4(q.a1, lds4(b + 1536), q.b1, r1);
          m1 = add4(mc, z1);
          if (j >= j0 && j < j1) ps[0] = dot4(r1, ps[0]);
          if (STEPS == 2) r1 = R;  // what the second step subtracts from
        } else {
          if (KIND == STEP_SWEEP) m1 = lin4(q.a1, mc, q.b1, r1);
          if (j >= j0 && j < j1) {
            if (STEPS == 1) ps[0] = dot4(r1, ps[0]);
            z1 = lds4(b + 1536);
            z1 = KIND == STEP_UPDATE ? axpy4(q.a1, mc, z1) : add4(z1, mc);
          }
        }
        if (STEPS == 1 && owns) {
          const size_t c = col + (size_t)j * A.g32.pitch;
          if (KIND != STEP_CHEBY) st4(q.Ro + c, r1);
          st4(q.zo + c, z1);
          if (q.store_m) st4(q.mo + c, m1);
        }
      }
      if (STEPS == 2 && j - 1 >= j0 && j - 1 < j1) {
        const float4 w = apply4(m1c, m1s, m1, kec, k0, k1);
        const float4 r2 = f4(r1c.x - w.x, r1c.y - w.y, r1c.z - w.z, r1c.w - w.w);
        float4 z2, m2;
        if (KIND == STEP_CHEBY) {
          z2 = lin4(q.a2, z1c, q.b2, r2);
          m2 = add4(m1c, z2);
        } else {
          z2 = add4(z1c, m1c);
          m2 = lin4(q.a2, m1c, q.b2, r2);
        }
        ps[1] = dot4(r2, ps[1]);
        if (owns) {
          const size_t c = col + (size_t)(j - 1) * A.g32.pitch;
          if (KIND != STEP_CHEBY) st4(q.Ro + c, r2);
          st4(q.zo + c, z2);
          if (q.store_m) st4(q.mo + c, m2);
        }
      }
      if (++nrow == 4) {  // 16 products in FP32, then the pair
        acc[0].add(q.down * ps[0]);
        acc[1].add(q.down * ps[1]);
        ps[0] = ps[1] = 0.f;
        nrow = 0;
      }
      ms = mc;
      mc = mn;
      ic = iwn;
      k0 = k1;
      k1 = kn;
      m1s = m1c;
      m1c = m1;
      r1c = r1;
      z1c = z1;
      kec = ke;
      issue(row + DEPTH - 1, prev);  // its last reader was this trip
      prev = slot;
      slot = slot + 1 == DEPTH ? 0 : slot + 1;
    }
    cp_wait<0>();
    acc[0].add(q.down * ps[0]);
    acc[1].add(q.down * ps[1]);
    if (sums) tile_sums<HANDED>(S, acc);
    if (HANDED) walk.take(asked);
    else walk.step();
  }
}

// p' = beta p + r into `pn`; p'.p' and its face sums (p'.A p' is both together).
template <bool HANDED>
__device__ __forceinline__ void direction_pass(Grid grid, const IrSweeps &A, const float *p, const float *r, float *pn,
                                               float beta, float down, unsigned ring, float rxh, float ryh, bool mirrored,
                                               unsigned &handed, PassSums &S) {
  constexpr int DEPTH = RING_BYTES / 1536;
  const int nx = A.g32.nx, ny = A.g32.ny;
  const int lane = threadIdx.x & 31;
  const unsigned slot0 = ring + 16 * lane;
  TileWalk walk(grid, A.t, ny, mirrored, &A.F.sc->bar.next_tile, handed);
  if (HANDED) handed += walk.requests();
  while (walk.valid()) {
    int strip, j0, j1;
    walk.place(strip, j0, j1);
    const unsigned asked = HANDED ? walk.ask() : 0u;
    const int i0 = strip * STRIP - 4 + 4 * lane;
    const bool in = i0 >= 0 && i0 < nx;
    const bool owns = lane >= 1 && lane <= 30 && i0 < nx;
    float fe[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) fe[m] = (i0 + m >= 0 && i0 + m + 1 < nx) ? rxh : 0.f;
    const size_t col = in ? A.g32.at(i0, 0) : (size_t)A.g32.hd;
    const size_t step = in ? (size_t)A.g32.pitch : 0;
    size_t next = col + (in ? (size_t)j0 * A.g32.pitch : 0);
    const int last = min(j1, ny - 1);
    auto issue = [&](int row, unsigned slot) {
      if (row <= last) {
        const unsigned a = slot0 + slot * 1536;
        cp16(a, p + next, in);
        cp16(a + 512, A.iw + next, in);
        cp16(a + 1024, r + next, in);
      }
      next += step;
      cp_commit();
    };
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) issue(j0 + d, d);
    float4 ps = f4(0, 0, 0, 0), is = ps;
    Pair acc[3] = {};
    float s[2] = {0.f, 0.f};
    int nrow = 0;
    unsigned slot = 0, prev = DEPTH - 1;
    for (int row = j0; row <= last; ++row) {
      cp_wait<DEPTH - 2>();
      const unsigned a = slot0 + slot * 1536;
      const float4 pv = axpy4(beta, lds4(a), lds4(a + 1024)), iw = lds4(a + 512);
      if (row > j0) {
        const float4 k = face_row(ryh, is, iw);
        const float dx = ps.x - pv.x, dy = ps.y - pv.y, dz = ps.z - pv.z, dw = ps.w - pv.w;
        s[1] = fmaf(k.x * dx, dx, fmaf(k.y * dy, dy, fmaf(k.z * dz, dz, fmaf(k.w * dw, dw, s[1]))));
      }
      if (row < j1) {
        const Faces4 k = faces4(fe, iw);
        const float pe = __shfl_down_sync(FULL, pv.x, 1);
        const float dx = pv.x - pv.y, dy = pv.y - pv.z, dz = pv.z - pv.w, dw = pv.w - pe;
        s[1] = fmaf(k.e.x * dx, dx, fmaf(k.e.y * dy, dy, fmaf(k.e.z * dz, dz, fmaf(k.e.w * dw, dw, s[1]))));
        s[0] = dot4(pv, s[0]);
        if (owns) st4(pn + col + (size_t)row * A.g32.pitch, pv);
      }
      if (++nrow == 4) {
        acc[0].add(down * s[0]);
        acc[1].add(down * s[1]);
        s[0] = s[1] = 0.f;
        nrow = 0;
      }
      ps = pv;
      is = iw;
      issue(row + DEPTH - 1, prev);
      prev = slot;
      slot = slot + 1 == DEPTH ? 0 : slot + 1;
    }
    cp_wait<0>();
    acc[0].add(down * s[0]);
    acc[1].add(down * s[1]);
    tile_sums<HANDED>(S, acc);
    if (HANDED) walk.take(asked);
    else walk.step();
  }
}

struct SweepShared {
  SumShared sum;
  double a, b;
  float af;
  Scale scale;
  int done;
};

// u += x on the interior.
__device__ __forceinline__ void fold_correction(Grid grid, const IrSweeps &A, const float *x) {
  const int nx = A.g.nx, lane = threadIdx.x & 31, chunks = (nx + 127) / 128;
  const long long n = (long long)chunks * A.g.ny;
  for (long long w = grid.id * PERSIST_WARPS + (threadIdx.x >> 5); w < n; w += grid.nb * PERSIST_WARPS) {
    const int j = (int)(w / chunks), i0 = (int)(w % chunks) * 128 + 4 * lane;
    if (i0 >= nx) continue;
    add_f32(A.F.u + A.g.at(i0, j), __ldcg(reinterpret_cast<const float4 *>(x + A.g32.at(i0, j))), nx - i0);
  }
}

template <bool HANDED>
__global__ void __launch_bounds__(PERSIST_THREADS, 1) k_cheby32(const IrSweeps A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ SweepShared S;
  const Grid grid = whole_grid();
  const int lane = threadIdx.x & 31;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING_BYTES;
  DevScalars *sc = A.F.sc;
  const float rxh = (float)sc->rxh, ryh = (float)sc->ryh;
  const double eps = sc->eps, bb = sc->bb;
  const int maxiters = sc->maxiters;
  const RootTest test(eps, bb);
  int iter = sc->iter, ci = sc->cheby_iters, nref = 0;
  unsigned target = 0, set = 0, handed = 0;
  bool mirrored = false;
  float *e = A.x, *en = A.pb, *p = A.p, *pn = A.sd;
  double err = sc->error, rr = 0.0;
  if (!ir_residual(grid, A.F, A.g, A.g32, A.t64, A.sums, S.sum, A.r, target, set, handed, rr)) return;
  double rel = bb > 0 ? sqrt(rr / bb) : sqrt(rr);
  while (rel >= eps && iter < maxiters) {
    const double refine_below = A.delta2 * rr;
    bool ev = false;
    Scale scale = scale_of(rr, Scale{});
    for (;;) {
      const bool two = iter + 2 <= maxiters;
      const int i1 = min(ci + 2, maxiters + 1), i2 = min(ci + 3, maxiters + 1);
      StepArgs q;
      q.m = e;
      q.R = A.r;
      q.z = p;
      q.mo = en;
      q.Ro = nullptr;
      q.zo = pn;
      q.a1 = (float)A.F.chebyalpha[i1];
      q.b1 = (float)A.F.chebybeta[i1];
      q.a2 = (float)A.F.chebyalpha[i2];
      q.b2 = (float)A.F.chebybeta[i2];
      q.m_valid = ev;
      q.z_valid = true;
      q.store_m = true;
      q.mirrored = mirrored;
      q.down = scale.down;
      PassSums sums;
      if (two) step_pass<STEP_CHEBY, 2, HANDED>(grid, A, q, ring, rxh, ryh, true, handed, sums);
      else step_pass<STEP_CHEBY, 1, HANDED>(grid, A, q, ring, rxh, ryh, true, handed, sums);
      const int steps = two ? 2 : 1;
      auto fin = [&](double g1, double g2, double) {
        const double g = two ? g2 : g1;
        const bool hit = test.met(g) || below(g, refine_below) || test.met(g1) || below(g1, refine_below);
        if (lane == 0) {
          S.a = g;
          S.scale = scale_of(g, scale);
          S.done = hit || iter + steps >= maxiters;
        }
      };
      if (!grid_sums<HANDED>(grid, S.sum, &sc->bar, A.sums, sums, scale.up, target, set, fin)) return;
      float *t = e;
      e = en;
      en = t;
      t = p;
      p = pn;
      pn = t;
      ev = true;
      mirrored = !mirrored;
      iter += steps;
      ci += steps;
      err = S.a;
      scale = S.scale;
      if (S.done) break;
    }
    fold_correction(grid, A, e);
    if (!grid_barrier(grid, &sc->bar, target)) return;
    if (!ir_residual(grid, A.F, A.g, A.g32, A.t64, A.sums, S.sum, A.r, target, set, handed, rr)) return;
    rel = bb > 0 ? sqrt(rr / bb) : sqrt(rr);
    ++nref;
  }
  export_f32(grid, A.g, A.g32, p, A.F.p);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->red[0] = rr;
    sc->red[1] = rel;
    sc->refinements = nref;
    sc->iter = iter;
    sc->cheby_iters = ci;
    sc->error = err;
    sc->done = 1;
  }
}

template <bool HANDED>
__global__ void __launch_bounds__(PERSIST_THREADS, 1) k_ppcg32(const IrSweeps A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ SweepShared S;
  const Grid grid = whole_grid();
  const int lane = threadIdx.x & 31;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING_BYTES;
  DevScalars *sc = A.F.sc;
  GridBar *bar = &sc->bar;
  const float rxh = (float)sc->rxh, ryh = (float)sc->ryh;
  const double eps = sc->eps, bb = sc->bb;
  const int maxiters = sc->maxiters, n = A.ninner;
  const float rtheta = (float)(1.0 / sc->theta);
  const RootTest test(eps, bb);
  int iter = sc->iter, outer = sc->cheby_iters, nref = 0;
  unsigned target = 0, set = 0, handed = 0;
  bool mirrored = false;
  // p, r and the buffer that is free in between take turns
  float *p = A.p, *r = A.r, *spare = A.pb, *sd = A.sd, *sdn = A.sdb;
  double beta = sc->beta, rr = A.rr, err = sc->error, alpha = 0.0;
  double rel = bb > 0 ? sqrt(rr / bb) : sqrt(rr);
  while (rel >= eps && iter < maxiters) {
    const double refine_below = A.delta2 * rr;
    double gamma = rr;
    Scale scale = scale_of(rr, Scale{});
    bool xv = false;
    for (;;) {
      PassSums sums;
      direction_pass<HANDED>(grid, A, p, r, spare, (float)beta, scale.down, ring, rxh, ryh, mirrored, handed, sums);
      auto step = [&](double pp, double faces, double) {
        const double pw = pp + faces, a = gamma / pw;
        if (lane == 0) {
          S.a = a;
          S.af = (float)a;
        }
      };
      if (!grid_sums<HANDED>(grid, S.sum, bar, A.sums, sums, scale.up, target, set, step)) return;
      mirrored = !mirrored;
      alpha = S.a;
      float *t = p;
      p = spare;
      spare = t;
      // the update with the first sweep, then the others two by two
      sums = PassSums{};
      for (int pp = 1; pp <= n;) {
        const bool update = pp == 1, two = update || pp + 1 <= n;
        const int end = update ? 1 : two ? pp + 1 : pp;  // the last sweep of this pass
        StepArgs q;
        q.m = update ? p : sd;
        q.R = r;
        q.z = A.x;
        q.mo = update ? sd : sdn;
        q.Ro = spare;
        q.zo = A.x;
        q.a1 = update ? S.af : (float)A.F.chebyalpha[pp];
        q.b1 = update ? rtheta : (float)A.F.chebybeta[pp];
        q.a2 = (float)A.F.chebyalpha[end];
        q.b2 = (float)A.F.chebybeta[end];
        q.m_valid = true;
        q.z_valid = xv;
        q.store_m = end < n;  // the last sweep's sd starts nothing
        q.mirrored = mirrored;
        q.down = scale.down;
        const bool last = end == n;
        if (update) step_pass<STEP_UPDATE, 2, HANDED>(grid, A, q, ring, rxh, ryh, last, handed, sums);
        else if (two) step_pass<STEP_SWEEP, 2, HANDED>(grid, A, q, ring, rxh, ryh, last, handed, sums);
        else step_pass<STEP_SWEEP, 1, HANDED>(grid, A, q, ring, rxh, ryh, last, handed, sums);
        mirrored = !mirrored;
        xv = true;
        t = r;
        r = spare;
        spare = t;
        if (!update) {
          t = sd;
          sd = sdn;
          sdn = t;
        }
        if (!last) {
          if (!grid_barrier(grid, bar, target)) return;
        } else {
          auto fin = [&](double g1, double g2, double) {
            const double g = two ? g2 : g1, b = g / gamma;  // PPCG.jl:89-92
            const bool hit = test.met(g) || below(g, refine_below);
            if (lane == 0) {
              S.a = b;
              S.b = g;
              S.scale = scale_of(g, scale);
              S.done = hit || iter + 1 >= maxiters;
            }
          };
          if (!grid_sums<HANDED>(grid, S.sum, bar, A.sums, sums, scale.up, target, set, fin)) return;
        }
        pp = end + 1;
      }
      beta = S.a;
      gamma = err = S.b;
      scale = S.scale;
      ++iter;
      ++outer;
      if (S.done) break;
    }
    fold_correction(grid, A, A.x);
    if (!grid_barrier(grid, bar, target)) return;
    if (!ir_residual(grid, A.F, A.g, A.g32, A.t64, A.sums, S.sum, r, target, set, handed, rr)) return;
    rel = bb > 0 ? sqrt(rr / bb) : sqrt(rr);
    ++nref;
  }
  export_f32(grid, A.g, A.g32, p, A.F.p);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->red[0] = rr;
    sc->red[1] = rel;
    sc->refinements = nref;
    if (nref > 0) {
      sc->iter = iter;
      sc->cheby_iters = outer;
      sc->alpha = alpha;
      sc->beta = beta;
      sc->rro = err;
      sc->error = err;
      sc->first = 0;
      sc->done = 1;
    }
  }
}

// `reps` passes of one kind on the current FP32 fields, coefficients zero: 6 two
// Chebyshev steps, 7 two PPCG sweeps, 8 a CG pass that leaves p and x, 9 one
// that forms two steps' p and x.
__global__ void __launch_bounds__(PERSIST_THREADS, 1) k_bench32(const IrSweeps A, const IrCg C, int kind, int reps) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ SumShared S;
  const Grid grid = whole_grid();
  const unsigned ring = (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING_BYTES;
  GridBar *bar = &A.F.sc->bar;
  const float rxh = (float)A.F.sc->rxh, ryh = (float)A.F.sc->ryh;
  unsigned target = 0, set = 0, handed = 0;
  for (int k = 0; k < reps; ++k) {
    const int odd = k & 1;
    PassSums sums;
    if (kind >= 8) {
      PassArgs q{};
      q.rc = C.r[odd];
      q.rn = C.r[odd ^ 1];
      q.sc = C.s[odd];
      q.sn = C.s[odd ^ 1];
      q.s_valid = q.p_valid = q.x_valid = true;
      q.mirrored = odd;
      q.down = 1.f;
      if (kind == 8) ir_pass<PASS_STEP, true>(grid, C, q, ring, rxh, ryh, handed, sums);
      else ir_pass<PASS_STEP2, true>(grid, C, q, ring, rxh, ryh, handed, sums);
    } else {
      StepArgs q{};
      q.m = kind == 6 ? (odd ? A.pb : A.x) : odd ? A.sdb : A.sd;
      q.mo = kind == 6 ? (odd ? A.x : A.pb) : odd ? A.sd : A.sdb;
      q.R = kind == 6 ? A.r : odd ? A.pb : A.r;
      q.Ro = kind == 6 ? nullptr : odd ? A.r : A.pb;
      q.z = kind == 6 ? (odd ? A.sd : A.p) : A.x;
      q.zo = kind == 6 ? (odd ? A.p : A.sd) : A.x;
      q.m_valid = q.z_valid = q.store_m = true;
      q.mirrored = odd;
      q.down = 1.f;
      if (kind == 6) step_pass<STEP_CHEBY, 2, true>(grid, A, q, ring, rxh, ryh, true, handed, sums);
      else step_pass<STEP_SWEEP, 2, true>(grid, A, q, ring, rxh, ryh, false, handed, sums);
    }
    if (kind == 7) {
      if (!grid_barrier(grid, bar, target)) return;
    } else if (!grid_sums<true>(grid, S, bar, A.sums, sums, 0, target, set, [](double, double, double) {})) {
      return;
    }
  }
}

IrSweeps sweep_args(tl_ctx *ctx, int ninner, double rr) {
  tl_ir_state *ir = ctx->ir;
  IrSweeps A;
  A.F = ctx->F;
  A.g = ctx->g;
  A.g32 = g32_of(ctx);
  A.r = ir->r;
  A.x = ir->x;
  A.p = ir->p;
  A.pb = ir->pb;
  A.sd = ir->sd;
  A.sdb = ir->sdb;
  A.iw = ir->iw;
  A.delta2 = IR_DELTA * IR_DELTA;
  A.ninner = ninner;
  A.rr = rr;
  A.sums = static_cast<GridSums *>(ctx->grid_sums);
  // a row takes both steps' arithmetic; see tl_ir_cg.cuh for the rule
  const TileCost pass{3.0, 450.0, 1500.0, 300.0, 400.0, 16, 24, 8}, resid{1.0, 1200.0, 1500.0, 1100.0, 200.0, 0, 48, 4};
  A.t = make_tiling(ctx->g.nx, ctx->g.ny, STRIP, pass, persist_blocks(ctx->sm_count), PERSIST_WARPS);
  A.t64 = make_tiling_on(A.t, ctx->g.nx, ctx->g.ny, 64, resid, PERSIST_WARPS);
  return A;
}

// `fixed`: the kernel where every warp has its tiles; `handed`: where they are handed out.
int run_sweeps(tl_ctx *ctx, const void *fixed, const void *handed, int ninner, double rr) {
  IrSweeps A = sweep_args(ctx, ninner, rr);
  const void *kernel = A.t.handed ? handed : fixed;
  const size_t smem = (size_t)RING_BYTES * PERSIST_WARPS;
  CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int rc = tl_bar_ready(ctx);
  if (rc) return rc;
  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  void *args[] = {&A};
  CK(cudaLaunchCooperativeKernel(kernel, dim3(A.t.blocks), dim3(PERSIST_THREADS), args, smem, ctx->stream));
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  ctx->launches += 1;
  if ((rc = tl_read_scalars(ctx))) return rc;
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  ctx->last_solve_ms = ms;
  return tl_persist_check(ctx);
}

// p32 = (float) p on the interior, 0 in the halo.
__global__ void k_ir_import_p(Fields F, Geom g, G32 g32, float *p) {
  const long long n = (long long)g.X * g.Y;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int I = (int)(k % g.X), J = (int)(k / g.X);
    const bool interior = I >= g.hd && I < g.X - g.hd && J >= g.hd && J < g.Y - g.hd;
    p[(size_t)I + (size_t)J * g32.pitch] = interior ? (float)F.p[(size_t)I + (size_t)J * g.pitch] : 0.f;
  }
}

}  // namespace
}  // namespace tl

using namespace tl;

// The Chebyshev iteration after its switch, in FP32 inside FP64 refinement
// (tealeaf mode).  On entry the FP64 Chebyshev phase has run its first step
// (the iterate is in ub after an odd count).  The FP32 steps solve for the
// correction of the current refinement with the same coefficient sequence;
// each refinement folds the correction into u, measures the true residual in
// FP64 and restarts the correction from it, so the recurrence continues
// unchanged.  Stops on the relative true residual ||u0 - A u|| / ||u0|| < eps
// or the iteration budget.
int tl_cheby32_run(tl_ctx *ctx, int *refinements, double *rel_out) {
  int rc = tl_read_scalars(ctx);
  if (rc) return rc;
  if (ctx->host_sc->cheby_iters & 1) {
    launch_copy_interior(ctx->stream, ctx->F.u, ctx->F.ub, ctx->g);
    CKL();
  }
  long long blocks = ((long long)ctx->g.X * ctx->g.Y + 255) / 256;
  if (blocks > 152LL * 32) blocks = 152LL * 32;
  k_ir_import_p<<<(int)blocks, 256, 0, ctx->stream>>>(ctx->F, ctx->g, g32_of(ctx), ctx->ir->p);
  CKL();
  if ((rc = run_sweeps(ctx, (const void *)k_cheby32<false>, (const void *)k_cheby32<true>, 0, 0.0))) return rc;
  *refinements = ctx->host_sc->refinements;
  *rel_out = ctx->host_sc->red[1];
  return TL_OK;
}

// The PPCG iteration after its switch, in FP32 inside FP64 refinement
// (tealeaf mode).  On entry the FP32-refined CG presteps have ended at the
// switch (tl_ir_presteps): u holds the iterate, r its true residual in FP64
// and FP32 (r.r in `rr`), p the FP32 search direction, and the device scalars
// theta, beta and the inner coefficients.  The outer steps continue the search
// direction; each refinement folds the correction into u, measures the true
// residual in FP64 and replaces the FP32 residual with it.  Stops on the
// relative true residual ||u0 - A u|| / ||u0|| < eps or the iteration budget.
int tl_ppcg32_run(tl_ctx *ctx, const tl_params *prm, double rr, int *refinements, double *rel_out) {
  int rc = run_sweeps(ctx, (const void *)k_ppcg32<false>, (const void *)k_ppcg32<true>, prm->ppcginnersteps, rr);
  if (rc) return rc;
  *refinements = ctx->host_sc->refinements;
  *rel_out = ctx->host_sc->red[1];
  return TL_OK;
}

// Times one FP32 pass kind (ids as in tl_bench_kernel): per step for the two that
// take two in a pass.
int tl_ir_bench_kernel(tl_ctx *ctx, int kernel, int reps, double *ms_per_launch) {
  if (kernel < 6 || kernel > 9) return TL_ERR_ARG;
  int rc = tl_ensure_ir(ctx);
  if (rc) return rc;
  IrSweeps A = sweep_args(ctx, 0, 0.0);
  IrCg C;
  ir_cg_args(C, ctx, persist_blocks(ctx->sm_count), true);
  const size_t smem = (size_t)RING_BYTES * PERSIST_WARPS;
  CK(cudaFuncSetAttribute(k_bench32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if ((rc = tl_bar_ready(ctx))) return rc;
  CK(cudaEventRecord(ctx->tev0, ctx->stream));
  void *args[] = {&A, &C, &kernel, &reps};
  CK(cudaLaunchCooperativeKernel((const void *)k_bench32, dim3(kernel >= 8 ? C.t.blocks : A.t.blocks),
                                 dim3(PERSIST_THREADS), args, smem, ctx->stream));
  CK(cudaEventRecord(ctx->tev1, ctx->stream));
  if ((rc = tl_read_scalars(ctx)) || (rc = tl_persist_check(ctx))) return rc;
  float t = 0.f;
  CK(cudaEventElapsedTime(&t, ctx->tev0, ctx->tev1));
  *ms_per_launch = t / reps / (kernel <= 7 ? 2 : 1);
  return TL_OK;
}

// The layout of the FP32 CG passes, as tl_get_layout and tl_set_layout show it.
int tl_ir_get_layout(tl_ctx *ctx, int *warps, int *rows, int *blocks) {
  int rc = tl_ensure_ir(ctx);
  if (rc) return rc;
  IrCg C;
  ir_cg_args(C, ctx, persist_blocks(ctx->sm_count), true);
  *warps = ctx->ir->set_warps ? ctx->ir->set_warps : PERSIST_WARPS;
  *rows = C.t.rows;
  *blocks = C.t.blocks;
  return TL_OK;
}

int tl_ir_set_layout(tl_ctx *ctx, int warps, int rows, int blocks) {
  int rc = tl_ensure_ir(ctx);
  if (rc) return rc;
  ctx->ir->set_warps = warps;
  ctx->ir->set_rows = rows;
  ctx->ir->set_blocks = blocks;
  return TL_OK;
}
