// tl_persist.cuh -- pieces of the persistent (cooperative) iteration kernels:
// the grid barrier, the sums over the grid and thread-private copy rings.
//
// A persistent kernel runs a whole iteration loop in one launch of at most one
// block per SM: a graph with a while-node spends 9 us on each kernel boundary
// of a small deck (18-20 us per CG iteration up to 512^2, whatever the
// deck), a barrier here takes 1.2 us over 152 blocks (0.9 over two), with a sum of
// digits 2.6, with three 3.0, with three sums of pairs 2.1.  Every block adds the
// block partials of a reduction itself, so all blocks hold the same scalars bit for
// bit and take the same decisions without another broadcast.
#pragma once

#include "tl_walk.cuh"

namespace tl {

constexpr int PERSIST_WARPS = 16;                 // warps of a persistent block
constexpr int PERSIST_THREADS = 32 * PERSIST_WARPS;
constexpr unsigned BAR_POLLS = 1u << 23;          // a wait gives up after 1.3 s (314 cycles a poll)

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
// bit all the same.  A number is cut into digits of 25 bits whose places are the
// same for all doubles (digit b counts 2^(25 b - 1074)); a sum keeps the digits of
// the four highest places that any addend has reached, each as a whole number of
// its own, with no carries between them.  What an addend puts into a place does
// not depend on the others, nor does the highest place, so neither does the sum
// on the order, over warps, blocks and the grid.  Whole numbers also add
// in 4-cycle instructions, where one FP64 addition takes 66.
//
// The places come from the addends themselves, not from an earlier sum: whatever
// a step did to the sum, the highest addend is held to its last bit and every
// other one to 2^-75 of it at least (2^22 addends, all cut the same way, are off by
// 2^-53).  There is room for 2^27 addends; a deck of 2^31 cells has fewer than 10^8.
constexpr int DIGIT = 25, DIGITS = 4;
constexpr int TOP_MIN = 2;  // of zero and the smallest doubles
// Infinities and NaN: a place above all others, in which digit 0 counts what
// holds +Inf, digit 2 what holds -Inf, NaN being both, so that none cancels another.
constexpr int TOP_SPECIAL = 100;

typedef __int128 Whole;

// +-m 2^(at - 1074)
struct Addend {
  unsigned long long m;
  int at, top;  // top: the place of its highest digit
  bool neg;
};
__device__ __forceinline__ Addend addend(double v) {
  const unsigned hi = (unsigned)__double2hiint(v);
  const int e = (int)(hi >> 20) & 2047;
  Addend a;
  a.m = ((unsigned long long)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | (unsigned)__double2loint(v);
  a.at = max(e, 1) - 1;
  a.top = e == 2047 ? TOP_SPECIAL : (a.at + 52) / DIGIT;
  a.neg = hi >> 31;
  return a;
}
// Its four digits up to place `top`, at or above its own.
__device__ __forceinline__ void digits(const Addend &a, int top, int (&d)[DIGITS]) {
  constexpr unsigned ONES = (1u << DIGIT) - 1;
  const int s = a.at - (top - (DIGITS - 1)) * DIGIT, left = min(max(s, 0), 47);  // more for a zero alone
  const unsigned long long m = a.m >> min(max(-s, 0), 63), lo = m << left, hi = (m >> 1) >> (63 - left);
  d[0] = (int)((unsigned)lo & ONES);
  d[1] = (int)((unsigned)(lo >> DIGIT) & ONES);
  d[2] = (int)(((unsigned)(lo >> 2 * DIGIT) | ((unsigned)hi << (64 - 2 * DIGIT))) & ONES);
  d[3] = (int)((unsigned)(hi >> (3 * DIGIT - 64)) & ONES);
#pragma unroll
  for (int k = 0; k < DIGITS; ++k) d[k] = a.neg ? -d[k] : d[k];
}
// Whether a number counts in digit k of the special place.
__device__ __forceinline__ bool counts(bool special, bool nan, bool neg, int k) {
  return special && (k == 0 ? nan || !neg : k == 2 && (nan || neg));
}
__device__ __forceinline__ int pick(const int (&d)[DIGITS], int k) {
  return k & 2 ? (k & 1 ? d[3] : d[2]) : (k & 1 ? d[1] : d[0]);
}

// A warp's share of a sum: each lane holds digit (lane & 3).
struct Digits {
  int top = TOP_MIN;
  long long d = 0;
};
// The digits counted from a higher top: those below the four are dropped.
__device__ __forceinline__ void raise_top(Digits &s, int top) {
  const int k = (threadIdx.x & 3) + top - s.top;
  const long long v = __shfl_sync(FULL, s.d, (threadIdx.x & 28) | (k & 3));
  s.d = k < DIGITS ? v : 0;
  s.top = top;
}
// Adds one number of each lane.
__device__ __forceinline__ void add_lanes(Digits &s, double v) {
  const Addend a = addend(v);
  const int top = max(s.top, __reduce_max_sync(FULL, a.top)), k = threadIdx.x & 3;
  if (top != s.top) raise_top(s, top);
  if (top == TOP_SPECIAL) {
    const bool special = a.top == TOP_SPECIAL, nan = a.m & 0xfffffffffffffull;
    const bool plus = __any_sync(FULL, counts(special, nan, a.neg, 0)), minus = __any_sync(FULL, counts(special, nan, a.neg, 2));
    s.d += k == 0 ? plus : k == 2 && minus;
    return;
  }
  int d[DIGITS];
  digits(a, top, d);
#pragma unroll
  for (int q = 0; q < DIGITS; ++q) d[q] = __reduce_add_sync(FULL, d[q]);
  s.d += pick(d, k);
}
// Adds a pair to each of the warp's sums: eight lanes a sum, its pair in their first.
// Both numbers go into one integer, cut 52 bits below the larger one's leading bit, of
// which each lane takes its digit.
__device__ __forceinline__ void add_pairs(Digits &s, Pair v) {
  const int k = threadIdx.x & 3, first = threadIdx.x & 24;
  const unsigned u[2] = {__float_as_uint(__shfl_sync(FULL, v.hi, first)), __float_as_uint(__shfl_sync(FULL, v.lo, first))};
  const int e[2] = {(int)(u[0] >> 23) & 255, (int)(u[1] >> 23) & 255}, most = max(max(e[0], e[1]), 1);
  long long m = 0;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const unsigned long long x = ((unsigned long long)((u[q] & 0x7fffffu) | (e[q] ? 0x800000u : 0u)) << 29) >>
                                 min(most - max(e[q], 1), 63);
    m += u[q] >> 31 ? -(long long)x : (long long)x;
  }
  const int at = most + 895;  // below 2^54, it counts 2^(at - 1074)
  const int top = max(s.top, most == 255 ? TOP_SPECIAL : m ? (at + 53) / DIGIT : TOP_MIN);
  if (__any_sync(FULL, top != s.top)) raise_top(s, top);
  if (top == TOP_SPECIAL) {
    bool count = false;
#pragma unroll
    for (int q = 0; q < 2; ++q) count = count || counts(e[q] == 255, u[q] & 0x7fffffu, u[q] >> 31, k);
    s.d += count;
  } else {
    const unsigned long long a = m < 0 ? -m : m;
    const int right = (top - (DIGITS - 1) + k) * DIGIT - at;
    const int d = (int)((unsigned)(right >= 0 ? a >> min(right, 63) : a << min(-right, 63)) & ((1u << DIGIT) - 1));
    s.d += m < 0 ? -d : d;
  }
}

// The four digits as one whole number.
__device__ __forceinline__ Whole join(long long d0, long long d1, long long d2, long long d3) {
  return (((((Whole)d3 << DIGIT) + d2) << DIGIT) + d1 << DIGIT) + d0;
}
// The double nearest to it.
__device__ __forceinline__ double to_double(Whole q, int top) {
  const bool neg = q < 0;
  const unsigned __int128 a = neg ? -(unsigned __int128)q : (unsigned __int128)q;
  const unsigned long long h = (unsigned long long)(a >> 64), l = (unsigned long long)a, w = h ? h : l;
  const int c = __clzll(w);
  const unsigned long long hi = (w << c) | (h ? (l >> 1) >> (63 - c) : 0ull);  // the leading bit at the top
  const int e = (h ? 127 : 63) - c + (top - (DIGITS - 1)) * DIGIT - 51;        // exponent field
  unsigned long long m = ((unsigned long long)e << 52) + (hi >> 11) - (1ull << 52) + ((hi >> 10) & 1);
  if (top == TOP_SPECIAL || !w || e < 1 || e >= 2047) {
    if (top == TOP_SPECIAL) {
      const bool plus = l & ((1ull << 2 * DIGIT) - 1), minus = a >> 2 * DIGIT;
      return plus && minus ? __longlong_as_double(0x7ff8000000000000ll) : plus ? INFINITY : -INFINITY;
    }
    if (!w) return 0.0;
    if (e >= 2047) return neg ? -INFINITY : INFINITY;
    const int below = min(12 - e, 63);  // below the normal numbers
    m = (hi >> below) + ((hi >> (below - 1)) & 1);
  }
  return __longlong_as_double((long long)(m | ((unsigned long long)neg << 63)));
}

// A persistent launch's block partials in global memory, two sets in turn (a
// block may already be at its next sum while another still reads this one).
// Each block adds up all partials itself: adding them into one place with
// atomics instead made an iteration 2.7 us longer (152 blocks on one line).
constexpr int PERSIST_MAX_BLOCKS = 160;
// The partials of one sum lie side by side, a block's in one 32-byte sector: what the
// blocks' loads cost is the sectors that all of them want at once.  A word holds a
// digit above the 7 bits of its top.
struct GridSums {
  long long part[2][3][PERSIST_MAX_BLOCKS][DIGITS];
  Pair pair[2][PERSIST_MAX_BLOCKS][4];  // [.][.][3] pads a block to 32 bytes
};

// A block's arrival at a barrier over the blocks of a cooperative launch and its
// wait for `target` arrivals in all, by one whole warp.  False when the wait
// gave up: the kernel returns at once, every block by its own limit.  What the
// block wrote before its last block barrier, and this warp before the call, is
// visible to every block after its wait.  All lanes wait, on one load: where
// lane 0 alone waited, the compiler ran all that follows once for it and once
// for the others (3 us a sum) and moved the others' loads ahead of the wait.
// Acquiring loads, where plain ones with a fence after them took 0.25 to 0.35 us
// more.  `busy`: a counter that whoever is waited for moves on; the limit counts
// from its last change.
__device__ __forceinline__ bool grid_arrive_wait(GridBar *g, unsigned target, const unsigned *busy = nullptr) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g->count) : "memory");
  unsigned n = 0, last = 0;
  bool there;
  do {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&g->count) : "memory");
    there = __all_sync(FULL, (int)(v - target) >= 0);
    if (busy && (n & 1023u) == 1023u) {
      const unsigned now = __shfl_sync(FULL, *reinterpret_cast<const volatile unsigned *>(busy), 0);
      if (now != last) n = 0;
      last = now;
    }
  } while (!there && ++n < BAR_POLLS);
  if (!there && (threadIdx.x & 31) == 0) atomicExch(&g->fail, 1u);
  return there;
}

// The barrier for whole blocks; `target` counts the arrivals expected so far on
// every thread (start at 0).
__device__ __forceinline__ bool grid_barrier(Grid G, GridBar *g, unsigned &target, const unsigned *busy = nullptr) {
  __shared__ int ok;
  __syncthreads();
  if (G.nb == 1) return true;
  target += G.nb;
  if (threadIdx.x < 32) ok = grid_arrive_wait(g, target, busy);
  __syncthreads();
  return ok != 0;
}

// a < b for an `a` that is not negative, in integer order: a compare on the FP64 pipe
// takes 64 cycles.  Nothing is below NaN or a negative b, nor is NaN below anything.
__device__ __forceinline__ bool below(double a, double b) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(a), y = (unsigned long long)__double_as_longlong(b);
  return x < y && y <= 0x7ff0000000000000ull;
}

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
  int top[3][PERSIST_WARPS];
  long long digit[3][PERSIST_WARPS][DIGITS];
  Pair pair[PERSIST_WARPS][4];  // [.][3] pads a row to 32 bytes
  int ok;
};

// The digits (lane & 3) of sum `e` of every LANESth warp from the jth on, added up at
// the highest top of the block's.
template <int LANES, class Highest>
__device__ __forceinline__ long long gather_digits(const SumShared &S, int e, int j, int &top, Highest &&highest) {
  constexpr int N = PERSIST_WARPS / LANES;
  const int k = threadIdx.x & 3;
  int t[N];
  top = TOP_MIN;
#pragma unroll
  for (int m = 0; m < N; ++m) top = max(top, t[m] = S.top[e][j + LANES * m]);
  top = highest(top);
  long long d = 0;
#pragma unroll
  for (int m = 0; m < N; ++m) {
    const int at = k + top - t[m];
    const long long x = S.digit[e][j + LANES * m][at & 3];
    d += at < DIGITS ? x : 0;
  }
  return d;
}
// The block's digits of the one sum, in every lane; of the three, eight lanes each.
__device__ __forceinline__ long long block_digits1(const SumShared &S, int &top) {
  long long d = gather_digits<8>(S, 0, (threadIdx.x & 31) >> 2, top, [](int t) { return __reduce_max_sync(FULL, t); });
#pragma unroll
  for (int off = 16; off >= DIGITS; off >>= 1) d += __shfl_xor_sync(FULL, d, off);
  return d;
}
__device__ __forceinline__ long long block_digits3(const SumShared &S, int &top) {
  const int lane = threadIdx.x & 31;
  const long long d = gather_digits<2>(S, lane < 24 ? lane >> 3 : 2, (lane & 7) >> 2, top,
                                       [](int t) { return max(t, __shfl_xor_sync(FULL, t, DIGITS)); });
  return d + __shfl_xor_sync(FULL, d, DIGITS);
}
__device__ __forceinline__ Whole join_lanes(long long d, int first) {
  const long long d0 = __shfl_sync(FULL, d, first), d1 = __shfl_sync(FULL, d, first + 1), d2 = __shfl_sync(FULL, d, first + 2),
                  d3 = __shfl_sync(FULL, d, first + 3);
  return join(d0, d1, d2, d3);
}

// The blocks' partials of N sums, each warp's eight (and eight of the blocks past 128)
// added up where its own digits were.  The whole block does it: one warp took
// 800 cycles a sum, with the digits joined into 16 bytes, 1100 with them in 32.
template <int N>
__device__ __forceinline__ void spread_partials(SumShared &S, const long long (*part)[PERSIST_MAX_BLOCKS][DIGITS], int nb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = 8 * warp + (lane >> 2);
  long long w[N][2];
#pragma unroll
  for (int e = 0; e < N; ++e)
#pragma unroll
    for (int m = 0; m < 2; ++m) w[e][m] = b + 128 * m < nb ? __ldcg(&part[e][b + 128 * m][lane & 3]) : (long long)TOP_MIN;
#pragma unroll
  for (int e = 0; e < N; ++e) {
    Digits s{(int)w[e][0] & 127, w[e][0] >> 7}, t{(int)w[e][1] & 127, w[e][1] >> 7};
    const int top = __reduce_max_sync(FULL, max(s.top, t.top));
    raise_top(s, top);
    raise_top(t, top);
    long long d = s.d + t.d;
#pragma unroll
    for (int off = 16; off >= DIGITS; off >>= 1) d += __shfl_xor_sync(FULL, d, off);
    if (lane < DIGITS) S.digit[e][warp][lane] = d;
    if (lane == 0) S.top[e][warp] = top;
  }
}

// A deck on one block has no barrier; its sums move the counter on all the same, for
// those that wait for the deck (tl_batch.cu).
__device__ __forceinline__ void count_alone(GridBar *bar) {
  if (threadIdx.x == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(&bar->count) : "memory");
}

// Sums over the grid and what follows from them: `fin(totals...)` on warp 0, and
// the block meets.  One block barrier before the grid's, two between it and `fin`,
// one after.  `set` counts the calls of a launch; target as in grid_barrier.
// Between reading and writing shared scalars `fin` needs a warp barrier.
//
// N = 1: each warp's digits of one sum.  N = 3: of three, the first in its lanes 0..7,
// the second and third in the next eights.
template <int N, class Fin>
__device__ __forceinline__ bool grid_sum(Grid grid, SumShared &S, GridBar *bar, GridSums *G, const Digits &v, unsigned &target,
                                         unsigned &set, Fin &&fin) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = grid.nb, e = lane >> 3, k = lane & 7;
  const bool holds = e < N && k < DIGITS;
  target += nb;
  if (holds) {
    S.digit[e][warp][k] = v.d;
    if (k == 0) S.top[e][warp] = v.top;
  }
  __syncthreads();
  int top;
  auto block_digits = [&]() { return N == 1 ? block_digits1(S, top) : block_digits3(S, top); };
  if (nb > 1) {
    long long(*part)[PERSIST_MAX_BLOCKS][DIGITS] = G->part[set & 1];
    if (warp == 0) {
      const long long d = block_digits();
      if (holds) __stcg(&part[e][grid.id][k], (d << 7) | top);
      S.ok = grid_arrive_wait(bar, target);
    }
    __syncthreads();
    spread_partials<N>(S, part, nb);
    __syncthreads();
  } else {
    count_alone(bar);
  }
  if (warp == 0) {
    const Whole q = join_lanes(block_digits(), N == 1 ? 0 : lane & 24);
    const double tot = to_double(q, top);
    if constexpr (N == 1) fin(tot);
    else fin(__shfl_sync(FULL, tot, 0), __shfl_sync(FULL, tot, 8), __shfl_sync(FULL, tot, 16));
  }
  ++set;
  __syncthreads();
  return nb == 1 || S.ok != 0;
}

// Three sums of pairs, each warp's share in lanes 0, 8 and 16: cheaper to form and
// to add (2.1 us over 152 blocks against 3.0), where the warps' tiles are fixed.
template <class Fin>
__device__ __forceinline__ bool grid_sum_pairs(Grid grid, SumShared &S, GridBar *bar, GridSums *G, Pair w, unsigned &target,
                                               unsigned &set, Fin &&fin) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = grid.nb, nw = blockDim.x >> 5;
  target += nb;
  if ((lane & 7) == 0 && lane < 24) S.pair[warp][lane >> 3] = w;
  __syncthreads();
  if (warp == 0) {
    Pair q[3] = {};
    if (lane < nw) {
#pragma unroll
      for (int m = 0; m < 3; ++m) q[m] = S.pair[lane][m];
    }
    Pair t = warp_pairs(q);
    if (nb > 1) {
      Pair(*part)[4] = G->pair[set & 1];
      if (lane < 24 && (lane & 7) == 0)
        __stcg(reinterpret_cast<float2 *>(&part[grid.id][lane >> 3]), make_float2(t.hi, t.lo));
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
    } else {
      count_alone(bar);
    }
    const double tot = (double)t.hi + (double)t.lo;
    fin(__shfl_sync(FULL, tot, 0), __shfl_sync(FULL, tot, 8), __shfl_sync(FULL, tot, 16));
  }
  ++set;
  __syncthreads();
  return nb == 1 || S.ok != 0;
}

// The FP32 passes add up 16 products in FP32, as far as those go (3.4e38), and the pairs
// of a tile, a warp or the whole grid beyond that: `down` is a power of two that
// brings them to about 1 where the last r.r was `ref`, and the total gets 2^up back, both
// exactly.  r.r may grow by 2^127 in a step, or fall by 2^100 and keep its bits.
struct Scale {
  float down = 1.f;
  int up = 0;
};
__device__ __forceinline__ Scale scale_of(double ref, Scale last) {
  const int e = (__double2hiint(ref) >> 20) & 2047, c = min(max(e, 1023 - 120), 1023 + 120);
  if (e == 0 || e == 2047) return last;  // nothing to go by
  Scale s;
  s.down = __int_as_float((127 + 1023 - c) << 23);
  s.up = c - 1023;
  return s;
}
// v 2^up, for what a sum of FP32 numbers can be.
__device__ __forceinline__ double scaled_up(double v, int up) {
  const int hi = __double2hiint(v), e = (hi >> 20) & 2047;
  return e == 0 || e == 2047 ? v : __hiloint2double(hi + up * (1 << 20), __double2loint(v));
}

// A warp's share of three sums over its tiles, in either form.
struct PassSums {
  Digits d;
  Pair w{0.f, 0.f};
};
template <bool HANDED>
__device__ __forceinline__ void add_tile(PassSums &s, Pair tile) {
  if (HANDED) add_pairs(s.d, tile);
  else s.w.add(tile);
}
template <bool HANDED, class Fin>
__device__ __forceinline__ bool grid_sums(Grid grid, SumShared &S, GridBar *bar, GridSums *G, const PassSums &v, int up,
                                          unsigned &target, unsigned &set, Fin &&fin) {
  auto scaled = [&](double a, double b, double c) { fin(scaled_up(a, up), scaled_up(b, up), scaled_up(c, up)); };
  if constexpr (HANDED) return grid_sum<3>(grid, S, bar, G, v.d, target, set, scaled);
  else return grid_sum_pairs(grid, S, bar, G, v.w, target, set, scaled);
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
  // the same where it is known that none are handed out
  __device__ __forceinline__ void step() { t += T.warps; }
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
// block, which needs no grid barrier: a row a warp (28^2 by FP64 CG: 7.4 us an
// iteration spread over blocks, 10.2 with two rows a warp on one).
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
