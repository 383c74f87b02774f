// The row-marching solves of the ideal gas (pressure), the energy formula and the magnetic
// systems, and the choice between them and the tile kernels.  Multiply-adds are contracted in
// this file (build.py): a solve's rounding stays below its tolerance either way.
#include "march_solve.cuh"

namespace imex {
namespace march {
namespace {

// Every block runs `iters` pass ends over the launched blocks and `phantom` others that were never
// launched; the first block, whose verdict is the launch's as in a solve, comes `late` cycles after
// the rest to the last of them.  *gave_up: blocks that did not get through with the right sum.
constexpr int kSelfWarps = 8;
__global__ void __launch_bounds__(32 * kSelfWarps, 1)
    k_pass_end_selftest(SyncState* sync, double* partial, DevStats* st, int phantom, int iters, long long late,
                        long long limit, long long* cycles, int* gave_up) {
  __shared__ Shared S;
  Sync y{sync, ld_relaxed(&sync->epoch), 0ull, limit, (int)gridDim.x + phantom, (int)blockIdx.x, partial};
  const long long t0 = clock64();
  bool ok = true;
  for (int k = 0; ok && k < iters; ++k) {
    if (blockIdx.x == 0 && k + 1 == iters) {
      const long long t1 = clock64();
      while (clock64() - t1 < late) {
      }
    }
    acc_clear(S);
    if ((threadIdx.x & 31) == 0) S.acc[threadIdx.x >> 5][0] = 1.0;
    ok = pass_end<kSelfWarps>(y, S, 1) && S.red[0] == (double)(kSelfWarps * y.nblk);
  }
  if (threadIdx.x != 0) return;
  if (!ok) atomicAdd(gave_up, 1);
  if (blockIdx.x != 0) return;
  *cycles = clock64() - t0;
  if (!ok) atomicMax(&st->status, (int)IMEX_ERR_SYNC);
  else if (y.seq > 0) st_relaxed(&sync->epoch, y.base + y.seq * (unsigned long long)y.nblk);
}

}  // namespace

// The B form's operator in the mixed form: its FP32 rows need half the registers and half the ring,
// which leaves room for twelve warps instead of eight (the FP64 refinement passes, a few per solve,
// spill 260 bytes), and its ring of twelve vectors makes loads ahead past it cost more registers than
// they hide.  A pass waits on its own chain of loads and arithmetic, so warps count.  Whole step of
// the 1024^2 random field, us, by warps / FP64 vectors in the ring / loaded ahead: 8/8/5 7870, 12/5/5
// 7702, 12/5/0 7423, 12/6/0 7287, 12/7/0 7819 (too little L1 left), 16/4/0 7580, 10/6/5 8244.
// The FP64 solve keeps eight warps: it needs their 255 registers.
using MagBMixed = MagBRow<double, 12, 6, 0>;
// The solves that run here: the fast arithmetic (the exact one keeps the reference's operation
// order, which the face forms do not), global dissipation (the energy operator has none) and,
// in the A form, periodic boundaries (an open tile extrapolates A past the edge).  The other
// configurations keep the tile kernels.
bool supports(const imex_ctx* ctx, int op) {
  const DevParams& P = ctx->P;
  if (!P.fast) return false;
  if (op == IMEX_OP_ENERGY) return true;
  if (op == IMEX_OP_MAGNETIC_A) return P.GLF && !P.xclamp && !P.yclamp;
  return P.GLF != 0;
}
// The FP64 A form of one small context stays with the tile kernels: a task marches four halo rows beside
// its two to five, and a pass lasts as long as a task.  us per solve, tile / marching: 64^2 169 / 200, 128^2 154 /
// 162, 251 x 173 116 / 118, 320^2 138 / 138, 512^2 161 / 127.  The mixed form and ensembles are
// faster here at every size.
constexpr size_t kMarchA = 100000;
bool takes(const imex_ctx* ctx, int op, bool fp64) {
  if (!supports(ctx, op)) return false;
  return op != IMEX_OP_MAGNETIC_A || ctx->N >= kMarchA || (!fp64 && is_mixed(ctx, IMEX_MIXED_MAGNETIC));
}
// Members nearly as many as blocks get one block each here, and the FP64 magnetic solve of one of 32^2 to 64^2
// cells in one block takes longer than on four tile blocks per SM.  Ensemble steps, ms, B form, tile / marching
// magnetic solves: 80 members of sides 8 to 60 1.29 / 1.36, 80 of 32 to 64 1.64 / 1.83, 148 of 8 to 60 1.92 / 1.99 (A
// form 1.76 / 2.08, 2.12 / 2.44, 2.53 / 2.73); 80 of 8 to 24 1.00 / 0.98, 200 of 32 to 64 3.72 / 3.48, 40 of 16 to 64 and
// the mixed form faster here.
bool takes(const std::vector<imex_ctx*>& members, int op) {
  imex_ctx* c0 = members[0];
  if (!supports(c0, op)) return false;
  if (op != IMEX_OP_MAGNETIC_A && op != IMEX_OP_MAGNETIC_B) return true;
  if (is_mixed(c0, op == IMEX_OP_MAGNETIC_A ? IMEX_MIXED_MAGNETIC : IMEX_MIXED_MAGNETIC | IMEX_MIXED_MAGNETIC_B)) return true;
  const size_t n = members.size(), sms = (size_t)c0->num_sms;
  size_t largest = 0;
  for (const imex_ctx* m : members) largest = std::max(largest, m->N);
  return 2 * n <= sms || n > sms || largest <= 24 * 24 || largest > 64 * 64;
}
imex_status gmres_solve(imex_ctx* ctx, int op, int fam, double* x, const double* b, const Scratch* scratch) {
  const bool rk = ctx->P.eos_type != IMEX_IDEAL_GAS;
  if (op == IMEX_OP_PRESSURE_L || op == IMEX_OP_PRESSURE_J) {
    const bool jac = op == IMEX_OP_PRESSURE_J;
    return rk ? gmres_solve_rk(ctx, jac, fam, x, b, scratch)
              : solve<PressureRow<double, false>>(ctx, jac, fam, IMEX_MIXED_PRESSURE, x, b, scratch);
  }
  if (op == IMEX_OP_ENERGY) return solve<EnergyRow<double>>(ctx, false, fam, IMEX_MIXED_PRESSURE, x, b, scratch);
  if (op == IMEX_OP_MAGNETIC_B)
    return solve<MagBRow<double>, MagBMixed>(ctx, false, fam, IMEX_MIXED_MAGNETIC | IMEX_MIXED_MAGNETIC_B, x, b, scratch);
  return solve<MagARow<double>>(ctx, false, fam, IMEX_MIXED_MAGNETIC, x, b, scratch);
}
imex_status newton_solve(imex_ctx* ctx, double* p, const double* b, int keys) {
  if (ctx->P.eos_type != IMEX_IDEAL_GAS) return newton_solve_rk(ctx, p, b, keys);
  return is_mixed(ctx, IMEX_MIXED_PRESSURE) ? newton_one<float, false>(ctx, p, b, keys)
                                            : newton_one<double, false>(ctx, p, b, keys);
}
imex_status batch_build(BatchSolvePlan* plan, const std::vector<imex_ctx*>& members, int op, bool nested) {
  imex_ctx* c0 = members[0];
  if (op == IMEX_OP_MAGNETIC_A)
    return add_solves<MagARow<double>>(plan, members, IMEX_MIXED_MAGNETIC, F_GMRES_MAG_A, magnetic_system);
  if (op == IMEX_OP_MAGNETIC_B)
    return add_solves<MagBRow<double>, MagBMixed>(plan, members, IMEX_MIXED_MAGNETIC | IMEX_MIXED_MAGNETIC_B, F_GMRES_MAG_B,
                                       magnetic_system);
  if (op == IMEX_OP_ENERGY)
    return add_solves<EnergyRow<double>>(plan, members, IMEX_MIXED_PRESSURE, F_GMRES_ENERGY, energy_system);
  if (!nested)
    return add_solves<PressureRow<double, false>>(plan, members, IMEX_MIXED_PRESSURE, F_NEWTON, pressure_system);
  if (c0->P.eos_type != IMEX_IDEAL_GAS) return batch_newton_rk(plan, members);
  return is_mixed(c0, IMEX_MIXED_PRESSURE) ? add_newtons<float, false>(plan, members)
                                           : add_newtons<double, false>(plan, members);
}
size_t scratch_partials(imex_ctx* ctx) {
  return (size_t)2 * (ctx->num_sms < kMaxBlocks ? ctx->num_sms : kMaxBlocks) * kSlots;
}

}  // namespace march

imex_status run_pass_end_selftest(imex_ctx* ctx, int iterations, int phantom_blocks, double late_s, double timeout_s,
                                  double* us, int* gave_up, int* blocks) {
  const int nb = ctx->num_sms < kMaxBlocks ? ctx->num_sms : kMaxBlocks;
  if (2LL * (nb + phantom_blocks) * march::kSlots > ctx->partial_len)
    return set_error(ctx, IMEX_ERR_INVALID, "pass-end self-test: too many phantom blocks");
  const double khz = ctx->clock_khz > 0 ? (double)ctx->clock_khz : 2.0e6;
  long long late = (long long)(late_s * khz * 1e3), limit = (long long)(timeout_s * khz * 1e3) + 1;
  long long* cycles = reinterpret_cast<long long*>(ctx->red);
  int* count = reinterpret_cast<int*>(ctx->red + 1);
  cudaError_t e = cudaMemsetAsync(ctx->red, 0, 2 * sizeof(double), ctx->stream);
  if (e != cudaSuccess) return cuda_check(ctx, e, "pass-end self-test");
  void* params[] = {(void*)&ctx->sync, (void*)&ctx->partial, (void*)&ctx->st, (void*)&phantom_blocks, (void*)&iterations,
                    (void*)&late,      (void*)&limit,        (void*)&cycles,  (void*)&count};
  e = cudaLaunchCooperativeKernel((const void*)march::k_pass_end_selftest, dim3(nb), dim3(32 * march::kSelfWarps), params, 0,
                                  ctx->stream);
  if (e != cudaSuccess) return cuda_check(ctx, e, "pass-end self-test launch");
  ctx->kernel_launches += 1;
  double h[2] = {0.0, 0.0};
  e = cudaMemcpyAsync(h, ctx->red, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_check(ctx, e, "pass-end self-test");
  long long spent = 0;
  int out = 0;
  std::memcpy(&spent, &h[0], sizeof(spent));
  std::memcpy(&out, &h[1], sizeof(out));
  if (us) *us = iterations > 0 ? (double)spent / iterations / (khz * 1e-3) : 0.0;
  if (gave_up) *gave_up = out;
  if (blocks) *blocks = nb;
  return IMEX_OK;
}

}  // namespace imex
