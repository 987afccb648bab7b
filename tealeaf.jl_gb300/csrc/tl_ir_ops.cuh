// tl_ir_ops.cuh -- the FP32 buffers of the refinement path, shared by the
// single-deck solves and the batch.  A solve starts (tl_start.cu) from the FP32
// residual and the inverse weights iw = 1/w over the whole array (w = rho for
// conductivity, 1/rho for its reciprocal: CG.jl:57-60), with rx/2, ry/2, so that
// Kx = rx (w_l + w_c) / (2 w_l w_c) = rx/2 (iw_l + iw_c) (CG.jl:62-67).
//
// FP32 arrays are pitched like the FP64 fields, 32 floats per pitch unit, first
// interior cell of each row 128-byte aligned; a lane owns 4 consecutive cells
// (one float4).
#pragma once

#include "tl_solvers.h"
#include "tl_walk.cuh"

struct tl_ir_state {
  float *buf = nullptr;
  long long pitch = 0, lead = 0, stride = 0;
  // CG: p, x; r in r / pb and s in sd / sdb by turns.  Chebyshev: the correction
  // in x / pb, p in p / sd.  PPCG: x; p and r take turns in p, pb and r; sd / sdb
  float *p = nullptr, *pb = nullptr, *r = nullptr, *x = nullptr;
  float *sd = nullptr, *sdb = nullptr;
  float *iw = nullptr;  // 1 / w (w = rho or 1/rho, CG.jl:57-60), halo included
  // tl_set_layout of the FP32 CG passes (kernels 8 and 9): 0 by rule
  int set_warps = 0, set_rows = 0, set_blocks = 0;
};

namespace tl {
namespace {

constexpr double IR_DELTA = 0.1;  // refine when ||r32|| < delta * ||r at the last refinement||

struct G32 {
  int nx, ny, hd, X, Y;
  long long pitch;
  __host__ __device__ __forceinline__ size_t at(int i, int j) const {
    return (size_t)(hd + i) + (size_t)(hd + j) * (size_t)pitch;
  }
};

__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float comp(const float4 &v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

G32 g32_of(tl_ctx *ctx) {
  G32 g;
  g.nx = ctx->g.nx;
  g.ny = ctx->g.ny;
  g.hd = ctx->g.hd;
  g.X = ctx->g.X;
  g.Y = ctx->g.Y;
  g.pitch = ctx->ir->pitch;
  return g;
}

}  // namespace
}  // namespace tl
