// tl_persist.cuh -- pieces of the persistent (cooperative) iteration kernels:
// the grid barrier, thread-private copy rings and the FP32-pair accumulator.
//
// A persistent kernel runs a whole iteration loop in one launch of at most one
// block per SM: a graph with a while-node spends 9 us on each kernel boundary
// of a small deck (18-20 us per CG iteration up to 512^2, whatever the
// deck), a barrier here 1.5 us.  Every block adds the block partials of a
// reduction itself, in the same order, so all blocks hold the same scalars bit
// for bit and take the same decisions without another broadcast.
#pragma once

#include "tl_walk.cuh"

namespace tl {

constexpr int PERSIST_WARPS = 16;                 // warps of a persistent block at most
constexpr int PERSIST_THREADS = 32 * PERSIST_WARPS;
constexpr unsigned BAR_POLLS = 1u << 23;          // a wait gives up after some seconds

// A running sum as an unevaluated pair hi + lo of FP32 numbers (the two-sum of
// Knuth): about 48 significant bits.  One FP64 instruction holds an SM
// sub-partition's FP64 pipe for 64 cycles on this part whatever its active
// lanes, and so does each FP32-to-FP64 conversion; the pair costs 6 (adding an
// FP32 number) to 10 full-rate instructions.
struct Pair {
  float hi, lo;
  __device__ __forceinline__ void add(float v) {
    const float s = __fadd_rn(hi, v);
    const float b = __fsub_rn(s, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(v, b)));
    hi = s;
  }
  __device__ __forceinline__ void add(Pair o) {
    add(o.hi);
    lo = __fadd_rn(lo, o.lo);
  }
};

__device__ __forceinline__ Pair shfl_xor(Pair v, int off) {
  return Pair{__shfl_xor_sync(FULL, v.hi, off), __shfl_xor_sync(FULL, v.lo, off)};
}

// Three sums over a warp at once: lane 0 gets the first, lane 8 the second,
// lane 16 the third.  Halving what a lane carries at each step takes 6 pair
// additions instead of the 15 of three butterflies.
__device__ __forceinline__ Pair warp_pairs(const Pair (&v)[3]) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, q = lane & 8;
  const Pair z{0.f, 0.f};
  Pair a = h ? v[2] : v[0], b = h ? z : v[1];
  a.add(shfl_xor(h ? v[0] : v[2], 16));
  b.add(shfl_xor(h ? v[1] : z, 16));
  Pair c = q ? b : a;
  c.add(shfl_xor(q ? a : b, 8));
  c.add(shfl_xor(c, 4));
  c.add(shfl_xor(c, 2));
  c.add(shfl_xor(c, 1));
  return c;
}

// The blocks that work on one deck: the whole launch, or a batch's group of it.
struct Grid {
  int nb, id;
};
__device__ __forceinline__ Grid whole_grid() { return Grid{(int)gridDim.x, (int)blockIdx.x}; }

// ---- sums over the grid ----------------------------------------------------
// Warps take their tiles in whatever order they come free (the SMs of one GPU
// do not get the same memory bandwidth: at 8192^2 the fast ones waited 110 of
// 400 us for the slow ones with equal shares).  The sums stay the same bit for
// bit all the same: each tile's sum, whose inner order is fixed, is turned
// into a 128-bit whole number of 2^-scale, and whole numbers add up exactly in
// any order, over warps, blocks and the grid.  They also add in 4-cycle
// instructions, where one FP64 addition takes 66.
typedef __int128 Fixed;

// The scale at which a number of the size of `ref` becomes about 2^62: 44 bits
// above it for sums that grow (p.A p against r.r: the operator's eigenvalues),
// 62 below it before anything is rounded off (a million addends, each rounded
// to nearest, are off by some 2^-52 of the sum).
__device__ __forceinline__ int fixed_scale(double ref) {
  return 62 + 1023 - (int)((__double_as_longlong(ref) >> 52) & 0x7ff);
}
// v 2^scale, rounded.  What would reach 2^106 (infinities and NaN
// among it) becomes 2^106: far beyond anything plausible beside 2^62.  A
// warp's sum is cut to it once more (fixed_cut), so that no number of such
// addends wraps round to a plausible sum.  `m` has `bits` bits at most.
constexpr int FIXED_BITS = 106;
__device__ __forceinline__ Fixed fixed_shift(unsigned long long m, int bits, int shift, bool neg) {
  Fixed q;
  if (shift >= 0) q = shift <= FIXED_BITS - bits ? (Fixed)m << shift : (Fixed)(m != 0) << FIXED_BITS;
  else q = shift > -64 ? (Fixed)((m >> -shift) + ((m >> (-shift - 1)) & 1)) : (Fixed)0;
  return neg ? -q : q;
}
__device__ __forceinline__ Fixed fixed_cut(Fixed q) {
  const Fixed most = (Fixed)1 << FIXED_BITS;
  return q > most ? most : q < -most ? -most : q;
}
__device__ __forceinline__ Fixed to_fixed(float v, int scale) {
  const unsigned u = __float_as_uint(v), e = (u >> 23) & 255u;
  const unsigned m = (u & 0x7fffffu) | (e ? 0x800000u : 0u);
  return fixed_shift(e == 255u ? 1u : m, 24, e == 255u ? FIXED_BITS : (int)(e ? e : 1u) - 150 + scale, u >> 31);
}
__device__ __forceinline__ Fixed to_fixed(double v, int scale) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v), e = (u >> 52) & 2047u;
  const unsigned long long m = (u & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull);
  return fixed_shift(e == 2047u ? 1ull : m, 53, e == 2047u ? FIXED_BITS : (int)(e ? e : 1u) - 1075 + scale, u >> 63);
}
// The number a whole number of 2^-scale stands for, cut to 53 bits; NaN for a sum
// that holds something cut to 2^106.
__device__ __forceinline__ double from_fixed(Fixed q, int scale) {
  const bool neg = q < 0;
  unsigned __int128 a = neg ? (unsigned __int128)(-q) : (unsigned __int128)q;
  const unsigned long long hi = (unsigned long long)(a >> 64), lo = (unsigned long long)a;
  if (!(hi | lo)) return 0.0;
  if (hi >> (FIXED_BITS - 64)) return __longlong_as_double(0x7ff8000000000000ll);
  const int top = hi ? 127 - __clzll(hi) : 63 - __clzll(lo);  // of the leading bit
  a = top > 52 ? a >> (top - 52) : a << (52 - top);
  const int e = top - scale + 1023;
  if (e >= 2047) return neg ? -INFINITY : INFINITY;
  if (e <= 0) return 0.0;  // below the normal numbers: nothing of the sum is left
  return __longlong_as_double((long long)((unsigned long long)a & 0xfffffffffffffull) | ((long long)e << 52) |
                              ((long long)neg << 63));
}
__device__ __forceinline__ Fixed shfl_xor(Fixed v, int off) {
  const unsigned __int128 u = (unsigned __int128)v;
  unsigned long long lo = (unsigned long long)u, hi = (unsigned long long)(u >> 64);
  lo = __shfl_xor_sync(FULL, lo, off);
  hi = __shfl_xor_sync(FULL, hi, off);
  return (Fixed)(((unsigned __int128)hi << 64) | lo);
}
__device__ __forceinline__ Fixed shfl(Fixed v, int lane) {
  const unsigned __int128 u = (unsigned __int128)v;
  unsigned long long lo = (unsigned long long)u, hi = (unsigned long long)(u >> 64);
  lo = __shfl_sync(FULL, lo, lane);
  hi = __shfl_sync(FULL, hi, lane);
  return (Fixed)(((unsigned __int128)hi << 64) | lo);
}

// A persistent launch's block partials in global memory, two sets in turn (a
// block may already be at its next sum while another still reads this one).
// Each block adds up all partials itself: adding them into one place with
// atomics instead made an iteration 2.7 us longer (152 blocks on one line).
constexpr int PERSIST_MAX_BLOCKS = 160;
// The partials of one sum lie side by side: what the blocks' loads cost is the
// 32-byte sectors that all of them want at once (three sums of 152 blocks, 64
// bytes a block: 3.2 us a reduction against 3.0).
struct GridSums {
  Fixed part[2][3][PERSIST_MAX_BLOCKS];
  Pair pair[2][PERSIST_MAX_BLOCKS][4];  // [.][.][3] pads a block to 32 bytes
};

__device__ __forceinline__ Fixed ldcg_fixed(const Fixed *p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(p));
  return (Fixed)(((unsigned __int128)v.y << 64) | v.x);
}
__device__ __forceinline__ void stcg_fixed(Fixed *p, Fixed v) {
  const unsigned __int128 u = (unsigned __int128)v;
  __stcg(reinterpret_cast<ulonglong2 *>(p), make_ulonglong2((unsigned long long)u, (unsigned long long)(u >> 64)));
}

// A block's arrival at a barrier over the blocks of a cooperative launch and its
// wait for `target` arrivals in all, by one whole warp.  False when the wait
// gave up: the kernel returns at once, every block by its own limit.  What the
// block wrote before its last block barrier, and this warp before the call, is
// visible to every block after its wait.  All lanes wait, on one load: where
// lane 0 alone waited, the compiler ran all that follows once for it and once
// for the others (3 us a sum) and moved the others' loads ahead of the wait.
// Acquiring loads, where plain ones with a fence after them took 0.25 to 0.35 us
// more.
__device__ __forceinline__ bool grid_arrive_wait(GridBar *g, unsigned target) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g->count) : "memory");
  unsigned n = 0;
  bool there;
  do {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&g->count) : "memory");
    there = __all_sync(FULL, (int)(v - target) >= 0);
  } while (!there && ++n < BAR_POLLS);
  if (!there && (threadIdx.x & 31) == 0) atomicExch(&g->fail, 1u);
  return there;
}

// The barrier for whole blocks; `target` counts the arrivals expected so far on
// every thread (start at 0).
__device__ __forceinline__ bool grid_barrier(Grid G, GridBar *g, unsigned &target) {
  __shared__ int ok;
  __syncthreads();
  if (G.nb == 1) return true;
  target += G.nb;
  if (threadIdx.x < 32) ok = grid_arrive_wait(g, target);
  __syncthreads();
  return ok != 0;
}

// Non-negative doubles in integer order: a compare on the FP64 pipe takes 64 cycles.
__device__ __forceinline__ bool below(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// A convergence test sqrt(e) < eps with e = error / bb (bb 1 for the absolute
// test): what lies above `limit` fails it whatever its rounding, so that most
// trips need no root and no division.  A limit that is not a normal number
// decides nothing.
struct RootTest {
  double eps, bb, limit;
  bool usable;
  __device__ __forceinline__ RootTest(double eps, double bb) : eps(eps), bb(bb), limit(eps * eps * bb * (1.0 + 1e-9)) {
    usable = limit > 1e-290 && limit < 1e290;
  }
  __device__ __forceinline__ bool met(double error) const {
    if (usable && below(limit, error)) return false;
    return sqrt(bb == 1.0 ? error : error / bb) < eps;
  }
};

struct SumShared {
  Fixed warp[PERSIST_WARPS][3];
  Pair pair[PERSIST_WARPS][4];  // [.][3] pads a row to 32 bytes
  int ok;
};

// Sums over the grid and what follows from them: `fin(totals...)` on warp 0, and
// the block meets.  One block barrier before the grid's, one after `fin`.
// `set` counts the calls of a launch; target as in grid_barrier.
// Between reading and writing shared scalars `fin` needs a warp barrier.
//
// One sum: each warp's share in lane 0, in whole numbers of 2^-scale.
template <class Fin>
__device__ __forceinline__ bool grid_sum1(Grid grid, SumShared &S, GridBar *bar, GridSums *G, Fixed v, int scale, unsigned &target,
                                          unsigned &set, Fin &&fin) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = grid.nb, nw = blockDim.x >> 5;
  target += nb;
  if (lane == 0) S.warp[warp][0] = fixed_cut(v);
  __syncthreads();
  if (warp == 0) {
    Fixed t = lane < nw ? S.warp[lane][0] : (Fixed)0;
    for (int off = nw >> 1; off >= 1; off >>= 1) t += shfl_xor(t, off);
    if (nb > 1) {
      Fixed *part = G->part[set & 1][0];
      if (lane == 0) stcg_fixed(part + grid.id, t);
      S.ok = grid_arrive_wait(bar, target);
      Fixed q[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) q[m] = lane + 32 * m < nb ? ldcg_fixed(part + lane + 32 * m) : (Fixed)0;
      t = q[0] + q[1] + q[2] + q[3] + q[4];
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) t += shfl_xor(t, off);
    }
    fin(from_fixed(shfl(t, 0), scale));
  }
  ++set;
  __syncthreads();
  return nb == 1 || S.ok != 0;
}

// Three sums, each warp's share in lanes 0, 8 and 16.  Two forms: `v`, whole
// numbers, for tiles taken in any order; `w`, pairs, which are cheaper to form
// and to add (1.3 us of an iteration of 7.9 at 256^2), where every warp has its
// one fixed tile.
template <bool FIXED, class Fin>
__device__ __forceinline__ bool grid_sum3(Grid grid, SumShared &S, GridBar *bar, GridSums *G, Fixed v, int scale, Pair w,
                                          unsigned &target, unsigned &set, Fin &&fin) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = grid.nb, nw = blockDim.x >> 5;
  target += nb;
  if ((lane & 7) == 0 && lane < 24) {
    if (FIXED) S.warp[warp][lane >> 3] = fixed_cut(v);
    else S.pair[warp][lane >> 3] = w;
  }
  __syncthreads();
  if (warp == 0) {
    const int d = lane < 24 ? lane >> 3 : 2, c = lane & 7;
    double tot;
    if (FIXED) {
      Fixed t = c < nw ? S.warp[c][d] : (Fixed)0;
      if (nw > 8) t += S.warp[c + 8][d];
      t += shfl_xor(t, 4);
      t += shfl_xor(t, 2);
      t += shfl_xor(t, 1);
      if (nb > 1) {
        Fixed(*part)[PERSIST_MAX_BLOCKS] = G->part[set & 1];
        if (lane < 24 && c == 0) stcg_fixed(&part[d][grid.id], t);
        S.ok = grid_arrive_wait(bar, target);
        Fixed q[3][5], x[3];
#pragma unroll
        for (int e = 0; e < 3; ++e)
#pragma unroll
          for (int m = 0; m < 5; ++m) q[e][m] = lane + 32 * m < nb ? ldcg_fixed(&part[e][lane + 32 * m]) : (Fixed)0;
#pragma unroll
        for (int e = 0; e < 3; ++e) x[e] = q[e][0] + q[e][1] + q[e][2] + q[e][3] + q[e][4];
        // over the warp: lanes 0..7 end with the first sum, 8..15 the second, the rest the third
        const bool up = lane & 16;
        const Fixed a = shfl_xor(up ? x[0] : x[2], 16), b = shfl_xor(x[1], 16);
        x[0] = up ? x[2] + a : x[0] + a;
        x[1] = up ? (Fixed)0 : x[1] + b;
        const bool second = !up && (lane & 8);
        const Fixed f = shfl_xor(second || up ? x[0] : x[1], 8);
        t = (second ? x[1] : x[0]) + f;
        t += shfl_xor(t, 4);
        t += shfl_xor(t, 2);
        t += shfl_xor(t, 1);
      }
      tot = from_fixed(t, scale);
    } else {
      Pair q[3] = {};
      if (lane < nw) {
#pragma unroll
        for (int m = 0; m < 3; ++m) q[m] = S.pair[lane][m];
      }
      Pair t = warp_pairs(q);
      if (nb > 1) {
        Pair(*part)[4] = G->pair[set & 1];
        if (lane < 24 && c == 0) __stcg(reinterpret_cast<float2 *>(&part[grid.id][d]), make_float2(t.hi, t.lo));
        S.ok = grid_arrive_wait(bar, target);
        float4 ab[5];
        float2 e[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          const int k = lane + 32 * m;
          ab[m] = k < nb ? __ldcg(reinterpret_cast<const float4 *>(&part[k][0])) : make_float4(0.f, 0.f, 0.f, 0.f);
          e[m] = k < nb ? __ldcg(reinterpret_cast<const float2 *>(&part[k][2])) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) q[m] = Pair{0.f, 0.f};
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          q[0].add(Pair{ab[m].x, ab[m].y});
          q[1].add(Pair{ab[m].z, ab[m].w});
          q[2].add(Pair{e[m].x, e[m].y});
        }
        t = warp_pairs(q);
      }
      tot = (double)t.hi + (double)t.lo;
    }
    fin(__shfl_sync(FULL, tot, 0), __shfl_sync(FULL, tot, 8), __shfl_sync(FULL, tot, 16));
  }
  ++set;
  __syncthreads();
  return nb == 1 || S.ok != 0;
}

// Adds a warp's lanes, in every lane.
__device__ __forceinline__ Fixed warp_fixed(Fixed v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v += shfl_xor(v, off);
  return v;
}

// Copies into a ring of shared memory where every thread reads back only what
// it copied itself: no barrier, and rows far ahead of their use cost no
// registers.  The copies go past L1 (.cg), so they read what other SMs wrote
// before the last grid barrier.  `pred` false fills with zeros and reads nothing.
__device__ __forceinline__ void cp16(unsigned smem, const void *g, bool pred) {
  const int n = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(g), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float4 lds4(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts2d(unsigned a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ double2 lds2d(unsigned a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}

// How a persistent kernel shares an nx x ny grid: warp tiles of `cols` columns,
// numbered along a row band first, bands of `rows` rows up to row `split` and of
// `rows2` from there.  Fewer tiles than warps are spread over the blocks, one
// warp of each after another; otherwise a block's warps start on neighbouring
// strips of the same rows.  After its first tile a warp takes every (number of
// warps)th one, or, with `handed`, the next that is free: the SMs of one GPU do
// not get the same memory bandwidth (with equal shares the fast ones waited 110
// of 400 us for the slow ones at 8192^2, FP32 CG).  The short bands come last, so
// that the warps finish together.
struct Tiling {
  int ntx, rows, split, rows2;
  int tiles1, tiles, blocks, warps;
  bool handed;
};

struct TileWalk {
  const Tiling &T;
  int ny;
  bool mirrored;  // rows counted from the top: the next pass begins where this one ends, in L2
  int t;
  unsigned *next;
  unsigned base;
  __device__ __forceinline__ TileWalk(Grid grid, const Tiling &T, int ny, bool mirrored, unsigned *next, unsigned base)
      : T(T), ny(ny), mirrored(mirrored), next(next), base(base) {
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    t = T.tiles < T.warps ? warp * grid.nb + grid.id : grid.id * nw + warp;
  }
  __device__ __forceinline__ bool valid() const { return t < T.tiles; }
  // strip, and rows [j0, j1)
  __device__ __forceinline__ void place(int &strip, int &j0, int &j1) const {
    const bool tail = t >= T.tiles1;
    const int u = tail ? t - T.tiles1 : t, band = u / T.ntx;
    strip = u - band * T.ntx;
    j0 = tail ? T.split + band * T.rows2 : band * T.rows;
    j1 = tail ? min(j0 + T.rows2, ny) : min(j0 + T.rows, T.split);
    if (mirrored) {
      const int k = ny - j1;
      j1 = ny - j0;
      j0 = k;
    }
  }
  // asked for while the current tile is still ahead, so that its latency is hidden
  __device__ __forceinline__ unsigned ask() const {
    unsigned v = 0;
    if (T.handed && (threadIdx.x & 31) == 0) v = atomicAdd(next, 1u);
    return v;
  }
  __device__ __forceinline__ void take(unsigned asked) {
    t = T.handed ? T.warps + (int)(__shfl_sync(FULL, asked, 0) - base) : t + T.warps;
  }
  // requests a whole pass makes: each warp asks once for each of its tiles
  __device__ __forceinline__ unsigned requests() const { return T.handed ? (unsigned)T.tiles : 0u; }
};

inline int persist_blocks(int sm_count) { return sm_count < PERSIST_MAX_BLOCKS ? sm_count : PERSIST_MAX_BLOCKS; }

// The shape.  Up to `hand_from` strip rows a warp: the rows that make the slowest
// SM's pass shortest, in equal shares.  Beyond: tall bands, whose overlap is
// small, for the first three quarters and bands of `rows2` for the rest, handed
// out.  A tile takes `lat` cycles a row and `lat0` besides when its warp runs
// alone, `issue` and `issue0` of a sub-partition's issue (or FP64) slots; `extra`
// rows overlap the next tile.  A deck of at most `solo` strip rows runs on one
// block, which needs no grid barrier: a row a warp (28^2 by FP64 CG: 8.1 us an
// iteration spread over blocks, 10.6 with two rows a warp on one).
struct TileCost {
  double extra, lat, lat0, issue, issue0;
  int solo, hand_from, rows2;
};
inline Tiling make_tiling(int nx, int ny, int cols, const TileCost &c, int max_blocks, int block_warps) {
  Tiling t;
  t.ntx = (nx + cols - 1) / cols;
  const long long strip_rows = (long long)t.ntx * ny;
  const int cap = strip_rows <= c.solo ? 1 : max_blocks;
  const long long warps = (long long)cap * block_warps;
  t.rows2 = c.rows2;
  t.handed = strip_rows > c.hand_from * warps;
  if (t.handed) {
    t.rows = strip_rows > 128 * warps ? 32 : 16;
    t.split = (int)(0.75 * ny) / t.rows * t.rows;
  } else {
    double best = -1.0;
    t.rows = 1;
    for (int rows = 1; rows <= (ny < 64 ? ny : 64); ++rows) {
      const long long tiles = (long long)t.ntx * ((ny + rows - 1) / rows);
      const long long per_block = (tiles + cap - 1) / cap;
      const long long rounds = (per_block + block_warps - 1) / block_warps;
      const double lat = rounds * ((rows + c.extra) * c.lat + c.lat0);
      const double issue = (double)((per_block + 3) / 4) * ((rows + c.extra) * c.issue + c.issue0);
      const double cost = lat > issue ? lat : issue;
      if (best < 0 || cost < best) {
        best = cost;
        t.rows = rows;
      }
    }
    t.split = ny;
  }
  t.tiles1 = t.ntx * ((t.split + t.rows - 1) / t.rows);
  t.tiles = t.tiles1 + t.ntx * ((ny - t.split + t.rows2 - 1) / t.rows2);
  t.blocks = t.tiles < cap ? t.tiles : cap;
  t.warps = t.blocks * block_warps;
  return t;
}

// The same grid of blocks for another pass.
inline Tiling make_tiling_on(const Tiling &first, int nx, int ny, int cols, const TileCost &c, int block_warps) {
  Tiling t = make_tiling(nx, ny, cols, c, first.blocks, block_warps);
  t.blocks = first.blocks;
  t.warps = first.warps;
  if (t.handed && t.tiles <= t.warps) t.handed = false;
  return t;
}

}  // namespace tl
