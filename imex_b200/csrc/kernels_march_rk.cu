// The row-marching pressure solves of the Redlich-Kwong gas.  Multiply-adds stay uncontracted here, as in
// the tile kernels and in the stage's EOS: the solves wait on the inversions' divisions and square roots,
// and contracted they gained nothing (a step of the 768^2 random field 6763 us against 6765, its Newton
// solves 408 us each against 410).
#include "march_solve.cuh"

namespace imex {
namespace march {

imex_status gmres_solve_rk(imex_ctx* ctx, bool jac, int fam, double* x, const double* b, const Scratch* scratch) {
  return solve<PressureRow<double, true>>(ctx, jac, fam, IMEX_MIXED_PRESSURE, x, b, scratch);
}
imex_status newton_solve_rk(imex_ctx* ctx, double* p, const double* b, int keys) {
  return is_mixed(ctx, IMEX_MIXED_PRESSURE) ? newton_one<float, true>(ctx, p, b, keys)
                                            : newton_one<double, true>(ctx, p, b, keys);
}
imex_status batch_newton_rk(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members) {
  return is_mixed(members[0], IMEX_MIXED_PRESSURE) ? add_newtons<float, true>(plan, members)
                                                   : add_newtons<double, true>(plan, members);
}

}  // namespace march

// this translation unit's EOS iteration-cap flag
imex_status eos_flag_march_enqueue(imex_ctx* ctx, int* host_flag) {
  return cuda_check(ctx, cudaMemcpyFromSymbolAsync(host_flag, d_eos_flag, sizeof(int), 0, cudaMemcpyDeviceToHost,
                                                   ctx->stream),
                    "eos flag");
}
imex_status eos_flag_march_clear(imex_ctx* ctx) {
  static const int zero = 0;
  cudaError_t e = cudaMemcpyToSymbolAsync(d_eos_flag, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  return cuda_check(ctx, e, "eos flag reset");
}

}  // namespace imex
