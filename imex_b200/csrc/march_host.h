// Host interface of the row-marching solver kernels (kernels_march.cu).
#pragma once

#include <vector>

#include "imex_internal.h"

namespace imex {
namespace march {

// work arrays of a solve that must not use the context's (imex_gmres_noalloc)
struct Scratch {
  double *V, *AV, *partial;
  SyncState* sync;
};
// whether the solve of `op` (imex_op) under this context's configuration can run here (and does, in an ensemble)
bool supports(const imex_ctx* ctx, int op);
// whether one context's solve does; fp64: whatever the configuration's precision (imex_gmres_noalloc)
bool takes(const imex_ctx* ctx, int op, bool fp64 = false);
imex_status gmres_solve(imex_ctx* ctx, int op, int fam, double* x, const double* b, const Scratch* scratch = nullptr);
imex_status newton_solve(imex_ctx* ctx, double* p, const double* b, int keys);
// whether the batched solve of these members does
bool takes(const std::vector<imex_ctx*>& members, int op);
// the batched solve of every member; nested: the nested Newton instead of the linear pressure solve
imex_status batch_build(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members, int op, bool nested);
// the same for the Redlich-Kwong gas's pressure solves (kernels_march_rk.cu)
imex_status gmres_solve_rk(imex_ctx* ctx, bool jac, int fam, double* x, const double* b, const Scratch* scratch);
imex_status newton_solve_rk(imex_ctx* ctx, double* p, const double* b, int keys);
imex_status batch_newton_rk(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members);
// doubles of partial sums a solve with Scratch needs
size_t scratch_partials(imex_ctx* ctx);

}  // namespace march
}  // namespace imex
