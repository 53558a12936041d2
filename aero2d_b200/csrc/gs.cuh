// Argument blocks and launchers of the Gram-Schmidt kernels (gs.cu).
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "batch.cuh"

namespace a2d {

constexpr int kHStride = kMaxRestart + 2;   // per-case stride of coefficient arrays
constexpr int kGsRows = 8;                  // rows of a chunk (gs.cu)

template <typename TB>
struct GsArgs {
  const double* w = nullptr;      // vector being orthogonalised
  const TB* V = nullptr;          // raw basis, vector q at V + q * vstride
  size_t vstride = 0;
  int nq = 0;                     // basis vectors taken (at most kMaxRestart)
  double* part = nullptr;         // pass 1, 2: partials [chunk][pstride], slot q; pass 1 also w . w in slot nq
  int pstride = 0;
  // pass 2 and 3: the partials of the pass before, which every CTA reduces over its case's chunks
  // itself into h_q = scale_q * sum; the case's first CTA stores h in fold_h (and, with
  // fold_wn0, the norm of w from slot nq).  Pass 3 subtracts with h1 + h
  const double* fold_part = nullptr;
  double* fold_h = nullptr;
  double* fold_wn0 = nullptr;
  const double* h1 = nullptr;     // [case][kHStride] coefficients of pass 1
  const double* scale = nullptr;  // [q][case] scale of raw basis vector q
  TB* Vout = nullptr;             // pass 3 / start: raw basis vector written
  double* part_norm = nullptr;    // pass 3, start: squared norm per chunk
  uint32_t need = 0;
};

struct GsCloseArgs {
  const double* part_norm = nullptr;
  const double* wn0 = nullptr;
  const double* h1 = nullptr;
  const double* h2 = nullptr;
  double* H = nullptr;            // [case][kMaxRestart][kMaxRestart+1], column k = step k
  double* scale = nullptr;        // [q][case]; k = -1 writes row 0
  CaseCtl* ctl = nullptr;
  uint32_t* live = nullptr;
  int k = -1;
  uint32_t need = 0;
};

template <typename TB> void launch_gs_dots(const Batch& b, const GsArgs<TB>& a, cudaStream_t s);
template <typename TB> void launch_gs_project(const Batch& b, const GsArgs<TB>& a, cudaStream_t s);
template <typename TB> void launch_gs_finish(const Batch& b, const GsArgs<TB>& a, cudaStream_t s);
template <typename TB> void launch_gs_start(const Batch& b, const GsArgs<TB>& a, cudaStream_t s);
void launch_gs_close(const Batch& b, const GsCloseArgs& a, cudaStream_t s);
// A whole Arnoldi step (passes 1 to 3 and the close) in one launch, a cluster per case: the most
// vectors, up to nq, that a case of max_chunks chunks takes with clusters of `cluster` CTAs while
// every case's runs at once (0: none), and the launch
int gs_case_vectors(int ncases, int cluster, int max_chunks, int nq);
void launch_gs_case(const Batch& b, const GsArgs<__nv_bfloat16>& a, const GsCloseArgs& c, uint32_t* err, int cluster,
                    int max_chunks, cudaStream_t s);
// raises the dynamic shared-memory limit of the passes (host, once per device)
cudaError_t gs_init();

}  // namespace a2d
