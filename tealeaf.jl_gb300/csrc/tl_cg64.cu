// tl_cg64.cu -- the fused FP64 CG loop on one deck, one cooperative launch.
#include "tl_cg64.cuh"

namespace tl {
namespace {

__global__ void __launch_bounds__(WARPS64 * 32, 1) k_cg64(const Cg64 A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ Shared64 S;
  cg64_solve(whole_grid(), A, S, Mem64(ring_mem));
}

}  // namespace
}  // namespace tl

using namespace tl;

// The fused CG loop from the state tl_solve_start left (p = r, r.r in rro), to
// the solver's test, the presteps' switch or the iteration budget, with the last
// step's p! and the halo of u and p; the scalars are read back.  One launch.
int tl_cg64_run(tl_ctx *ctx, int check, double *ms) {
  Cg64 A;
  A.F = ctx->F;
  A.g = ctx->g;
  A.sums = static_cast<GridSums *>(ctx->grid_sums);
  A.check = check;
  cg64_tilings(A, persist_blocks(ctx->sm_count));
  const size_t smem = CG64_SMEM;
  CK(cudaFuncSetAttribute(k_cg64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int rc = tl_bar_ready(ctx);
  if (rc) return rc;
  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  void *args[] = {&A};
  CK(cudaLaunchCooperativeKernel((const void *)k_cg64, dim3(A.tw.blocks), dim3(WARPS64 * 32), args, smem, ctx->stream));
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  ctx->launches += 1;
  if ((rc = tl_read_scalars(ctx))) return rc;
  float t = 0.f;
  CK(cudaEventElapsedTime(&t, ctx->ev0, ctx->ev1));
  if (ms) *ms += t;
  return tl_persist_check(ctx);
}
