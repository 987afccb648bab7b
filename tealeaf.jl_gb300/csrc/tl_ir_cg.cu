// tl_ir_cg.cu -- the FP32-refined CG solve of one deck, one cooperative launch.
#include "tl_ir_cg.cuh"

namespace tl {
namespace {

__global__ void __launch_bounds__(PERSIST_THREADS, 1) k_ir_cg(const IrCg A) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ Shared S;
  ir_solve(whole_grid(), A, S, (unsigned)__cvta_generic_to_shared(ring_mem) + (threadIdx.x >> 5) * RING_BYTES);
}

}  // namespace
}  // namespace tl

using namespace tl;

// Runs the FP32-refined CG loop on the state that tl_solve_start (or the warm start
// after it) left, to the relative true residual, the iteration budget or the
// presteps' switch; the scalars are read back.  One launch.
int tl_ir_cg_run(tl_ctx *ctx) {
  IrCg A;
  ir_cg_args(A, ctx, persist_blocks(ctx->sm_count), true);
  CK(cudaFuncSetAttribute(k_ir_cg, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES * PERSIST_WARPS));
  int rc = tl_bar_ready(ctx);
  if (rc) return rc;
  CK(cudaEventRecord(ctx->ev0, ctx->stream));
  void *args[] = {&A};
  CK(cudaLaunchCooperativeKernel((const void *)k_ir_cg, dim3(A.t.blocks), dim3(PERSIST_THREADS), args,
                                 RING_BYTES * PERSIST_WARPS, ctx->stream));
  CK(cudaEventRecord(ctx->ev1, ctx->stream));
  ctx->launches += 1;
  if ((rc = tl_read_scalars(ctx))) return rc;
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  ctx->last_solve_ms += ms;
  return tl_persist_check(ctx);
}
