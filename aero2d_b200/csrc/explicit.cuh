// Launchers of the explicit RK4 + residual-smoothing kernels.
#pragma once
#include <cuda_runtime.h>

#include "batch.cuh"

namespace a2d {

// fp32: the explicit iteration's FP32 form (compute in FP32, values kept in the FP64 arrays)
// (and U copied to U0)
void launch_local_dt(const Batch& b, const double* U, double* U0, double* dt, double cfl, bool fp32, cudaStream_t s);
// one case's local time steps from primitives in the reference layout W[4][ni][nc] -> dt[ni][nc]
void launch_local_dt_prim(const GridDev& g, const double* W, double* dt, double cfl, cudaStream_t s);
// smoothing along i and j in one kernel: out = U0 - a (dt / vol) smoothed(R), or with U0 null the
// smoothed R; tab: the tables that launch_irs_table made for the plan's smoothing coefficient e
struct IrsArgs {
  const double* R = nullptr;
  const double* U0 = nullptr;
  const double* dt = nullptr;
  double* out = nullptr;
  const double* tab = nullptr;
  double e = 0.0, a = 0.0;
  int max_ni = 0;
  size_t smem = 0;          // the largest irs_smem_bytes of the cases
};
constexpr size_t kIrsMaxSmem = 227 * 1024;   // past it (lines of hundreds of rows): the kernels below
void launch_irs_fused(const Batch& b, const IrsArgs& p, bool fp32, cudaStream_t s);
void launch_irs_table(const Batch& b, double* tab, double e, bool fp32, cudaStream_t s);
size_t irs_table_entries(int ni, int nc);
size_t irs_smem_bytes(int ni, int nc, double e, bool fp32);
cudaError_t irs_init();
// R (in) -> tmp (out, smoothed along i then j)
void launch_irs(const Batch& b, double* R, double* tmp, double e, int max_ni, int max_nc, bool fp32,
                cudaStream_t s);
void launch_rk_stage(const Batch& b, const double* U0, const double* R, const double* dt, double* U, double a,
                     bool rest, bool fp32, cudaStream_t s);
void launch_rk_res(const Batch& b, const double* U0, const double* U, const double* dt, double* tpart,
                   cudaStream_t s);
void launch_rk_finish(const Batch& b, const double* tpart, const double* coef, double* res, double* circ,
                      cudaStream_t s);

// FAS multigrid transfers between a batch and its coarse batch (same cases, ni/2 x nc/2)
void launch_add_forcing(const Batch& b, double* R, const double* P, cudaStream_t s);
void launch_fas_restrict(const Batch& fine, const Batch& coarse, const double* Uf, double* Uc, double* Uc0,
                         cudaStream_t s);
void launch_fas_forcing(const Batch& fine, const Batch& coarse, const double* Rf, double* Pc, cudaStream_t s);
void launch_fas_prolong(const Batch& fine, const Batch& coarse, double* Uf, const double* Uc, const double* Uc0,
                        cudaStream_t s);

}  // namespace a2d
