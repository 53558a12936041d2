// Host runtime of the Euler path: batch plans, workspace layout, the
// pseudo-transient Newton step as a sequence of kernels (replayed as one CUDA
// graph), the explicit RK iteration, and the extern "C" entry points declared
// in include/aero2d_b200.h.
//
// A plan owns no device memory: every device array lives in the caller's
// workspace, carved at bind time.  The Newton loop's per-case bookkeeping
// (rollback, freeze, SER CFL, convergence test, aero2d/implicit.py:216-244)
// runs on the device, so the host synchronises once per step only to learn
// whether any case is still live.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include "aero2d_b200.h"
#include "batch.cuh"
#include "explicit.cuh"
#include "kernels.cuh"
#include "launch.cuh"

#include <nvtx3/nvToolsExt.h>
#include "gs.cuh"
#include "krylov.cuh"
#include "physics.cuh"

namespace a2d {

thread_local std::string g_last_error;

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

#define A2D_CK(call)                                                                   \
  do {                                                                                 \
    cudaError_t e_ = (call);                                                           \
    if (e_ != cudaSuccess)                                                             \
      return fail(A2D_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));  \
  } while (0)

struct Carve {
  size_t off = 0;
  size_t take(size_t bytes) {
    off = (off + 255) & ~size_t(255);
    const size_t o = off;
    off += bytes;
    return o;
  }
};

static size_t metrics_total_bytes(int ni, int nc) {
  return metrics_float_offset(ni, nc) + metrics_floats(ni, nc) * 4;
}

// Krylov basis storage of the mixed path: BF16 (the basis is the raw,
// unnormalised Arnoldi vectors with FP64 scales; Gram-Schmidt, the Hessenberg
// matrix and the update are FP64)
using Basis16 = __nv_bfloat16;

enum VecSlot { kU = 0, kR, kVin, kJV, kDU, kB, kX0, kT, kRr, kZ, kW, kPA, kPB, kU0, kPE, kPD, kNumVec };

}  // namespace a2d

using namespace a2d;

// the most 16x4 tiles that one wave of the FP64 and of the FP32 stencils takes: 2 and 4 CTAs on
// each of 148 SMs (tile_stencil)
constexpr int kFineTiles64 = 2 * 148, kFineTiles32 = 4 * 148;

struct a2d_plan {
  a2d_params p{};
  int ncases = 0;
  int m = 0;               // GMRES restart
  int max_ni = 0, max_nc = 0;
  std::vector<CaseDev> cases;
  std::vector<Tile> tiles;
  std::vector<Tile> jtiles;    // tiles of the FP32 linearised stencil, in the shape jvp_tile
  // tuning knobs (a2d_plan_set_tuning); the defaults are the fastest measured on a B200 on
  // the batch shapes timed (64, 4 x 16 and 8 cases of 256 x 64); FP64 plans start with the
  // lanes sweep
  int jvp_tile = kTile32x16;
  int sweep_variant = kSweepHalves;
  int max_jtiles = 0;          // the most tiles any JVP tile shape needs (workspace room)
  std::vector<Chunk> chunks;
  std::vector<Group> groups;
  std::vector<long long> cp_off;
  // cases by line-group count, and those that the one-launch preconditioner (lines.cu) cannot take
  // apart: a launch per class that `one` is set for; line_cases holds the case indices
  // class after class, rest_groups the line groups of all other classes, which the per-sweep
  // kernels take together (both set at bind, choose_lines)
  struct LineClass {
    int groups, rows, first, count;
    bool fits, one;
  };
  std::vector<LineClass> line_classes;
  std::vector<int> line_cases;
  int gs_cluster = 0, gs_vectors = 0, max_chunks = 0;   // Arnoldi steps in one launch: cluster size, up to this step
  std::vector<Group> rest_groups;
  size_t o_rgroups = 0;
  // smoothing tables (explicit.cu), a shape's once, of the cases whose shape fits the fused kernel;
  // irs_rest: cases that it does not fit
  size_t irs_entries = 0, irs_smem = 0, o_irs = 0;
  bool irs_rest = false;
  size_t o_lcases = 0, o_E0 = 0;   // o_E0: inv r of the lines, kept between the sweeps of an application
  long long C = 0, rows_nc = 0, rows_nc1 = 0, total_ni = 0;
  size_t tj = 8, tb = 8;   // bytes of face-Jacobian and basis storage entries
  size_t tf = 8;           // bytes of the sweep factor entries (G, C, P, Q)
  // workspace layout (offsets)
  size_t o_cases = 0, o_tiles = 0, o_chunks = 0, o_groups = 0, o_cpoff = 0, o_live = 0, o_ctl = 0;
  size_t o_vec[kNumVec] = {};
  size_t o_diag = 0, o_dt = 0, o_JIL = 0, o_JIR = 0, o_JJL = 0, o_JJR = 0, o_INV = 0, o_CF = 0, o_PQG = 0, o_V = 0;
  size_t o_H = 0, o_h1 = 0, o_h2 = 0, o_scale = 0, o_y = 0, o_wn0 = 0, o_circ = 0, o_circ_rk = 0;
  size_t o_tpart = 0, o_cpart = 0, o_cpart2 = 0, o_cpartn = 0, o_coef = 0, o_cp = 0, o_hrn = 0, o_hcl = 0,
         o_cnt = 0, o_idx = 0;
  size_t o_sat = 0;        // saturated FP16 factor entries since bind (a2d_factor_saturations)
  size_t o_jtiles = 0, o_ftiles = 0;
  Batch jbatch{};          // the batch with the JVP's tile list
  std::vector<Tile> ftiles;    // 16x4 tiles, none when they would be more than kFineTiles32
  Batch fbatch{};          // the batch with these
  int pstride = 0;
  size_t bytes = 0;
  char* ws = nullptr;
  Batch batch{};
  cudaGraphExec_t graph = nullptr;
  bool graph_failed = false;   // by the step before
  cudaStream_t graph_stream = nullptr;
  // a step's live count and failure flag on the host; not pinned: 8 bytes whose reader waits anyway, while
  // cudaMallocHost and cudaFreeHost took 0.9 to 2.5 and 0.4 ms of a plan's life
  int host_count[2] = {0, 0};
  int steps_taken = 0;
  int kernels_per_step = 0;
  a2d_plan* coarse = nullptr;   // FAS multigrid: the same cases on grids of every other node

  template <typename X> X* at(size_t off) const { return reinterpret_cast<X*>(ws + off); }
  double* vec(int s) const { return at<double>(o_vec[s]); }
  CaseCtl* ctl() const { return at<CaseCtl>(o_ctl); }
  uint32_t* live() const { return at<uint32_t>(o_live); }
};

namespace a2d {

// ---------------------------------------------------------------------------
// plan construction
// ---------------------------------------------------------------------------
// tiles of every case in the given shape, case after case
static std::vector<Tile> tile_list(const a2d_plan* P, int shape) {
  const int TI = tile_w(shape), TJ = tile_h(shape);
  std::vector<Tile> out;
  for (int k = 0; k < P->ncases; ++k) {
    const int ni = P->cases[k].g.ni, nc = P->cases[k].g.nc;
    for (int j0 = 0; j0 < nc; j0 += TJ)
      for (int i0 = 0; i0 < ni; i0 += TI)
        out.push_back(Tile{k, i0, j0, std::min(TI, ni - i0), std::min(TJ, nc - j0)});
  }
  return out;
}

static void build_tables(a2d_plan* P, const int* ni, const int* nc, const void* const* metrics,
                         const double* winf) {
  long long cell = 0, rnc = 0, rnc1 = 0, cpo = 0;
  for (int k = 0; k < P->ncases; ++k) {
    CaseDev c{};
    c.g = grid_view(metrics[k], ni[k], nc[k]);
    for (int q = 0; q < 4; ++q) c.winf[q] = winf[4 * k + q];
    c.cell_off = cell;
    c.rows_nc = rnc;
    c.rows_nc1 = rnc1;
    const int ngr = (ni[k] + kLanes - 1) / kLanes;
    c.tile0 = (int)P->tiles.size();
    for (int j0 = 0; j0 < nc[k]; j0 += kTJ)
      for (int i0 = 0; i0 < ni[k]; i0 += kTI)
        P->tiles.push_back(Tile{k, i0, j0, std::min(kTI, ni[k] - i0), std::min(kTJ, nc[k] - j0)});
    c.ntiles = (int)P->tiles.size() - c.tile0;
    const long long n4 = 4LL * ni[k] * nc[k];
    c.chunk0 = (int)P->chunks.size();
    for (long long b0 = 0; b0 < n4; b0 += kChunk)
      P->chunks.push_back(Chunk{k, (int)b0, (int)std::min<long long>(kChunk, n4 - b0)});
    c.nchunks = (int)P->chunks.size() - c.chunk0;
    P->max_chunks = std::max(P->max_chunks, c.nchunks);
    c.group0 = (int)P->groups.size();
    for (int g = 0; g < ngr; ++g)
      P->groups.push_back(Group{k, g, g * kLanes, std::min(kLanes, ni[k] - g * kLanes)});
    c.ngroups = ngr;
    P->cases.push_back(c);
    P->cp_off.push_back(cpo);
    cell += (long long)ni[k] * nc[k];
    rnc += (long long)ngr * nc[k];
    rnc1 += (long long)ngr * (nc[k] + 1);
    cpo += ni[k];
    P->max_ni = std::max(P->max_ni, ni[k]);
    P->max_nc = std::max(P->max_nc, nc[k]);
  }
  P->C = cell;
  P->rows_nc = rnc;
  P->rows_nc1 = rnc1;
  P->total_ni = cpo;
  for (int sh = 0; sh < kNumTileShapes; ++sh) P->max_jtiles = std::max(P->max_jtiles, (int)tile_list(P, sh).size());
  P->jtiles = tile_list(P, P->jvp_tile);
  P->ftiles = tile_list(P, kTile16x4);
  if ((int)P->ftiles.size() > kFineTiles32) P->ftiles.clear();
  std::map<std::pair<int, int>, int> irs_at;
  for (int k = 0; k < P->ncases; ++k) {
    P->cases[k].irs_off = -1;
    if (P->p.irs_eps <= 0) continue;
    const size_t smem = irs_smem_bytes(ni[k], nc[k], P->p.irs_eps, P->p.precision == A2D_MIXED);
    if (smem > kIrsMaxSmem) {
      P->irs_rest = true;
      continue;
    }
    const auto it = irs_at.emplace(std::make_pair(ni[k], nc[k]), (int)P->irs_entries);
    P->cases[k].irs_off = it.first->second;
    if (it.second) P->irs_entries += irs_table_entries(ni[k], nc[k]);
    P->irs_smem = std::max(P->irs_smem, smem);
  }
  std::map<std::pair<int, bool>, std::vector<int>> by_groups;
  for (int k = 0; k < P->ncases; ++k) {
    const int groups = P->cases[k].ngroups;
    const bool fits = P->p.precision == A2D_MIXED ? lines_take<float>(groups, nc[k]) : lines_take<double>(groups, nc[k]);
    by_groups[{groups, fits}].push_back(k);
  }
  for (const auto& g : by_groups) {
    a2d_plan::LineClass c{g.first.first, 0, (int)P->line_cases.size(), (int)g.second.size(), g.first.second, false};
    for (int k : g.second) c.rows = std::max(c.rows, nc[k]);
    P->line_cases.insert(P->line_cases.end(), g.second.begin(), g.second.end());
    P->line_classes.push_back(c);
  }
}

static void layout(a2d_plan* P) {
  Carve cv;
  const int B = P->ncases;
  const size_t C = (size_t)P->C;
  P->o_cases = cv.take(sizeof(CaseDev) * B);
  P->o_tiles = cv.take(sizeof(Tile) * P->tiles.size());
  P->o_chunks = cv.take(sizeof(Chunk) * P->chunks.size());
  P->o_groups = cv.take(sizeof(Group) * P->groups.size());
  P->o_cpoff = cv.take(sizeof(long long) * B);
  P->o_live = cv.take(sizeof(uint32_t) * B);
  P->o_ctl = cv.take(sizeof(CaseCtl) * B);
  for (int s = 0; s < kNumVec; ++s) P->o_vec[s] = cv.take(8 * 4 * C);
  P->o_diag = cv.take(8 * C);
  P->o_dt = cv.take(8 * C);
  const size_t lb = (size_t)16 * kLanes;
  P->o_JIL = cv.take(P->tj * lb * P->rows_nc);
  P->o_JIR = cv.take(P->tj * lb * P->rows_nc);
  P->o_JJL = cv.take(P->tj * lb * P->rows_nc1);
  P->o_JJR = cv.take(P->tj * lb * P->rows_nc1);
  P->o_INV = cv.take(P->tj * lb * P->rows_nc);
  P->o_CF = cv.take(P->tf * lb * P->rows_nc);
  P->o_PQG = cv.take(3 * P->tf * lb * P->rows_nc);
  P->o_E0 = cv.take(P->tj * lb / 4 * P->rows_nc);
  P->o_V = cv.take(P->tb * 4 * C * (size_t)(P->m + 1));
  P->o_H = cv.take(8 * (size_t)B * kMaxRestart * (kMaxRestart + 1));
  P->o_h1 = cv.take(8 * (size_t)B * kHStride);
  P->o_h2 = cv.take(8 * (size_t)B * kHStride);
  P->o_scale = cv.take(8 * (size_t)B * (P->m + 1));
  P->o_y = cv.take(8 * (size_t)B * kMaxRestart);
  P->o_wn0 = cv.take(8 * (size_t)B);
  P->o_circ = cv.take(8 * (size_t)B);
  P->o_circ_rk = cv.take(8 * (size_t)B);
  P->o_tpart = cv.take(8 * kTilePartStride * P->tiles.size());
  P->pstride = P->m + 2;
  P->o_cpart = cv.take(8 * (size_t)P->pstride * P->chunks.size());
  P->o_cpart2 = cv.take(8 * (size_t)P->pstride * P->chunks.size());   // pass 2's, while pass 1's are read
  P->o_cpartn = cv.take(8 * P->chunks.size());
  P->o_coef = cv.take(8 * 3 * (size_t)B);
  P->o_cp = cv.take(8 * (size_t)P->total_ni);
  P->o_hrn = cv.take(8 * (size_t)B * P->p.max_iter);
  P->o_hcl = cv.take(8 * (size_t)B * P->p.max_iter);
  P->o_cnt = cv.take(8);   // [0] live-case count, [1] failure flag of the kernels' bounded waits
  P->o_idx = cv.take(sizeof(int) * (size_t)B);   // case index lists of a2d_case_restart / _retire
  P->o_sat = cv.take(sizeof(unsigned long long));
  P->o_jtiles = cv.take(sizeof(Tile) * (size_t)P->max_jtiles);
  P->o_ftiles = cv.take(sizeof(Tile) * P->ftiles.size());
  P->o_irs = cv.take(8 * P->irs_entries);
  P->o_lcases = cv.take(sizeof(int) * (size_t)B);
  P->o_rgroups = cv.take(sizeof(Group) * P->groups.size());
  P->bytes = cv.off + 256;
}

// ---------------------------------------------------------------------------
// kernels of this file: init, counting, layout conversion, point flux
// ---------------------------------------------------------------------------
__global__ void k_init_state(Batch b, double* U) {
  const Tile t = b.tiles[blockIdx.x];
  const CaseDev cs = b.cases[t.cs];
  const GridDev& g = cs.g;
  const double rho = cs.winf[0], u = cs.winf[1], v = cs.winf[2], p = cs.winf[3];
  const double Uc[4] = {rho, rho * u, rho * v, p / kGm1 + 0.5 * rho * (u * u + v * v)};
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int j = t.j0 + c / t.ti, i = t.i0 + c % t.ti;
#pragma unroll
    for (int k = 0; k < 4; ++k) U[4 * cs.cell_off + vidx(g, k, j, i)] = Uc[k];
  }
}

__global__ void k_reset(int ncases, CaseCtl* ctl, uint32_t* live, double cfl0) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ncases) return;
  CaseCtl c{};
  c.cfl = cfl0;
  c.rn = NAN;
  c.lastrn = NAN;
  c.r0 = 1.0;
  c.omega = 1.0;
  ctl[k] = c;
  live[k] = kLiveNewton;
}

// restarts the listed cases (one block each) with the freestream now in their
// table entry: U := freestream and Newton state as k_reset; with keep, U stays
// (the previous point's solution) and so does r0, the residual reference of
// the sweep's first (cold) point, so that the tolerance keeps its absolute
// level and the SER CFL starts from the converged state's small residual
__global__ void k_restart_cases(Batch b, const int* idx, int keep, double* U, CaseCtl* ctl, uint32_t* live,
                                double cfl0) {
  const int k = idx[blockIdx.x];
  const CaseDev cs = b.cases[k];
  if (!keep) {
    const double rho = cs.winf[0], u = cs.winf[1], v = cs.winf[2], p = cs.winf[3];
    const double Uc[4] = {rho, rho * u, rho * v, p / kGm1 + 0.5 * rho * (u * u + v * v)};
    const long long n = (long long)cs.g.ni * cs.g.nc;
    double* Uk = U + 4 * cs.cell_off;
    for (long long c = threadIdx.x; c < n; c += blockDim.x) {
#pragma unroll
      for (int q = 0; q < 4; ++q) Uk[q * n + c] = Uc[q];
    }
  }
  if (threadIdx.x == 0) {
    const double r0 = ctl[k].r0;
    const bool carry = keep && ctl[k].nsteps > 0 && isfinite(r0) && r0 > 0.0;
    CaseCtl c{};
    c.cfl = cfl0;
    c.rn = NAN;
    c.lastrn = NAN;
    c.r0 = carry ? r0 : 1.0;
    c.keep_r0 = carry ? 1 : 0;
    c.omega = 1.0;
    ctl[k] = c;
    live[k] = kLiveNewton;
  }
}

__global__ void k_retire_cases(const int* idx, int n, uint32_t* live) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) live[idx[q]] = 0;
}

__global__ void k_count(int ncases, const CaseCtl* ctl, const uint32_t* live, int retire, int* out) {
  __shared__ int s;
  if (threadIdx.x == 0) s = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < ncases; k += blockDim.x) {
    const int busy = retire ? ((live[k] & kLiveNewton) ? 1 : 0) : (ctl[k].done ? 0 : 1);
    if (busy) atomicAdd(&s, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) *out = s;
}

// Cell vectors between the reference layout [4][ni][nc] and the internal one [4][nc][ni], of the
// cases of b's tiles from tile0 on; ref is case k's vector at 4 (cell_off(k) - off0), so off0 = 0
// for a whole batch and the case's own offset for one case.  A CTA turns one 32x8 tile over in
// shared memory: 64 contiguous bytes per load or store on the reference side, 256 on the
// internal.  Bound by memory: 64 cases of 256x64, 67 MB in and out, 14 us in and 12 out (one launch per
// case with one side strided was 64 times 2.4 us, and the host behind with the launches).
enum { kLayoutIn, kLayoutOut, kLayoutPrim };
template <int MODE>
__device__ __forceinline__ void layout_tile(const Batch& b, int tile0, long long off0, const double* __restrict__ src,
                                            double* __restrict__ dst) {
  __shared__ double sm[4][kTI][kTJ + 1];
  const Tile t = b.tiles[tile0 + blockIdx.x];
  const CaseDev& cs = b.cases[t.cs];
  const int ni = cs.g.ni, nc = cs.g.nc;
  const int ir = threadIdx.x / kTJ, jr = threadIdx.x % kTJ;   // the reference side's cell, j fastest
  const int ii = threadIdx.x % kTI, ji = threadIdx.x / kTI;   // the internal side's, i fastest
  const bool hr = ir < t.ti && jr < t.tj, hi = ii < t.ti && ji < t.tj;
  const size_t N = (size_t)ni * nc;
  const size_t qr = 4 * (size_t)(cs.cell_off - off0) + (size_t)(t.i0 + ir) * nc + t.j0 + jr;
  const size_t qi = 4 * (size_t)cs.cell_off + (size_t)(t.j0 + ji) * ni + t.i0 + ii;
  if constexpr (MODE == kLayoutIn) {
    if (hr) {
#pragma unroll
      for (int k = 0; k < 4; ++k) sm[k][ir][jr] = src[qr + k * N];
    }
    __syncthreads();
    if (hi) {
#pragma unroll
      for (int k = 0; k < 4; ++k) dst[qi + k * N] = sm[k][ii][ji];
    }
  } else {
    if (hi) {
      State4<double> u;
#pragma unroll
      for (int k = 0; k < 4; ++k) u.c[k] = src[qi + k * N];
      if constexpr (MODE == kLayoutPrim) u = cons_to_prim<double, double>(u);
#pragma unroll
      for (int k = 0; k < 4; ++k) sm[k][ii][ji] = u.c[k];
    }
    __syncthreads();
    if (hr) {
#pragma unroll
      for (int k = 0; k < 4; ++k) dst[qr + k * N] = sm[k][ir][jr];
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(256) k_layout(Batch b, int tile0, long long off0, const double* __restrict__ src,
                                                double* __restrict__ dst) {
  grid_wait();
  layout_tile<MODE>(b, tile0, off0, src, dst);
}

// a residual and the primitives of its state out together, one launch for both
__global__ void __launch_bounds__(256) k_layout_residual(Batch b, int tile0, long long off0,
                                                         const double* __restrict__ R, double* __restrict__ Rout,
                                                         const double* __restrict__ U, double* __restrict__ Wout) {
  grid_wait();
  if (blockIdx.y == 0) layout_tile<kLayoutOut>(b, tile0, off0, R, Rout);
  else layout_tile<kLayoutPrim>(b, tile0, off0, U, Wout);
}

__global__ void k_point_flux(int n, const double* WL, const double* WR, const double* S, double* F) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  State4<double> L, R;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    L.c[k] = WL[(size_t)k * n + q];
    R.c[k] = WR[(size_t)k * n + q];
  }
  const State4<double> f = hllc<double, double>(L, R, S[q], S[(size_t)n + q]);
#pragma unroll
  for (int k = 0; k < 4; ++k) F[(size_t)k * n + q] = f.c[k];
}

}  // namespace a2d

// ---------------------------------------------------------------------------
// orchestration
// ---------------------------------------------------------------------------
namespace a2d {

// NVTX range for profilers (no cost without one attached): the stages of a Newton
// step when it runs without a graph, and the C ABI's solver entry points
struct Range {
  explicit Range(const char* name) { nvtxRangePushA(name); }
  ~Range() { nvtxRangePop(); }
  Range(const Range&) = delete;
  Range& operator=(const Range&) = delete;
};

static SweepArgs sweep_args(const a2d_plan* P, uint32_t need) {
  SweepArgs a;
  a.INV = P->at<void>(P->o_INV);
  a.PQG = P->at<void>(P->o_PQG);
  a.dtmp = P->vec(kPD);
  a.CF = P->at<void>(P->o_CF);
  a.err = P->at<uint32_t>(P->o_cnt) + 1;
  a.need = need;
  return a;
}

static FactorArgs factor_args(const a2d_plan* P, uint32_t need) {
  FactorArgs fa;
  fa.U = P->vec(kU);
  fa.ctl = P->ctl();
  fa.JIL = P->at<void>(P->o_JIL);
  fa.JIR = P->at<void>(P->o_JIR);
  fa.JJL = P->at<void>(P->o_JJL);
  fa.JJR = P->at<void>(P->o_JJR);
  fa.INV = P->at<void>(P->o_INV);
  fa.CF = P->at<void>(P->o_CF);
  fa.PQG = P->at<void>(P->o_PQG);
  fa.diag = P->at<double>(P->o_diag);
  fa.cfl_base = P->p.cfl;
  fa.sat = P->at<unsigned long long>(P->o_sat);
  fa.err = P->at<uint32_t>(P->o_cnt) + 1;
  fa.need = need;
  return fa;
}

// whether an application's sweeps run as one launch for some cases (lines.cu)
static bool one_launch(const a2d_plan* P) {
  return P->rest_groups.size() < P->groups.size() &&
         P->sweep_variant == (P->p.precision == A2D_MIXED ? kSweepHalves : kSweepLanes);
}

// Which classes take the one-launch preconditioner.  Its launches follow each other, a class at a time, while the
// per-sweep kernels take every group of the batch at once, so one class alone is faster in one
// launch while its clusters run together, but not always in several waves of them, nor several small
// classes one after another.  The estimate, in us per row of a line for four sweeps on a B200: a wave
// of clusters `few` to `full` as it fills the device, a wave of per-sweep CTAs `sfew` to
// `sfull`.  The figures are fitted to 559 uniform mixed batches (2 to 16 groups, 48 to 300 rows, 8 to
// 128 cases: within 0.5 % of the better path on average, 1.95x faster than always one launch at 96
// cases of 384 x 143, and slower than that nowhere) and 128 FP64 ones.  Ragged, one launch a class
// against the per-sweep kernels (48 rows, a case each, mixed / FP64): two classes 58 and 66 us / 96 and 128, three
// 86 and 66 / 143 and 129, sixteen 530 and 69 / 763 and 138; two cases each of
// 96 x 24, 128 x 32, 192 x 48, 256 x 64 and 384 x 96 cells 179 and 129 / 267 and 267.
static void choose_lines(a2d_plan* P) {
  const bool mixed = P->p.precision == A2D_MIXED;
  struct Fit {
    double few, full, full1;   // full1: where only one CTA fits an SM
    int two_rows;              // rows up to which two do
    double sfew, sfull;
    int ctas;                  // per-sweep CTAs that run at once
  };
  const Fit f = mixed ? Fit{0.58, 0.85, 0.86, 142, 1.2, 2.9, 4 * 148} : Fit{1.0, 1.2, 1.2, 0, 2.45, 4.7, 3 * 148};
  const size_t n = P->line_classes.size();
  std::vector<double> cost(n, 0.0);
  std::vector<char> can(n, 0);
  for (size_t q = 0; q < n; ++q) {
    const a2d_plan::LineClass& c = P->line_classes[q];
    if (!c.fits) continue;
    const int at_once = mixed ? lines_clusters<float>(c.groups, c.rows) : lines_clusters<double>(c.groups, c.rows);
    // FP64: one CTA per SM, and a second wave loses to the per-sweep kernels (256 x 64: 8 cases
    // 111 against 193 us, 16 cases in two waves 196 against 180)
    can[q] = at_once > 0 && (mixed || c.count <= at_once);
    if (!can[q]) continue;
    const double full = c.rows <= f.two_rows ? f.full : f.full1;
    const int waves = (c.count - 1) / at_once;
    const double last = (double)(c.count - waves * at_once) / at_once;
    cost[q] = c.rows * (waves * full + f.few + (full - f.few) * last);
  }
  auto total = [&](const std::vector<char>& one) {
    double t = 0.0;
    int groups = 0, rows = 0;
    for (size_t q = 0; q < n; ++q) {
      const a2d_plan::LineClass& c = P->line_classes[q];
      if (one[q]) {
        t += cost[q];
      } else {
        groups += c.groups * c.count;
        rows = std::max(rows, c.rows);
      }
    }
    if (groups == 0) return t;
    const int waves = (groups - 1) / f.ctas;
    const double last = (double)(groups - waves * f.ctas) / f.ctas;
    return t + rows * (waves * f.sfull + f.sfew + (f.sfull - f.sfew) * last);
  };
  // from every class that fits, and from none: change the class that gains most while one does
  std::vector<char> best(n, 0);
  double best_t = total(best);
  for (int start = 0; start < 2; ++start) {
    std::vector<char> one(n, 0);
    if (start == 0) one = can;
    double t = total(one);
    for (bool more = true; more;) {
      more = false;
      size_t at = 0;
      for (size_t q = 0; q < n; ++q) {
        if (!can[q]) continue;
        one[q] ^= 1;
        const double u = total(one);
        one[q] ^= 1;
        if (u < t) {
          t = u;
          at = q;
          more = true;
        }
      }
      if (more) one[at] ^= 1;
    }
    if (t <= best_t) {
      best_t = t;
      best = one;
    }
  }
  P->rest_groups.clear();
  for (size_t q = 0; q < n; ++q) {
    a2d_plan::LineClass& c = P->line_classes[q];
    c.one = best[q] != 0;
    if (c.one) continue;
    for (int k = c.first; k < c.first + c.count; ++k) {
      const CaseDev& cs = P->cases[P->line_cases[k]];
      P->rest_groups.insert(P->rest_groups.end(), P->groups.begin() + cs.group0, P->groups.begin() + cs.group0 + cs.ngroups);
    }
  }
}

// x = M^-1 r: jacobi_sweeps line-Jacobi sweeps (aero2d/implicit.py:150-157);
// rin may be dst
template <typename TJ>
static void precond(a2d_plan* P, const Batch& B, const double* rin, double* dst, uint32_t need, cudaStream_t s) {
  SweepArgs a = sweep_args(P, need);
  const int sweeps = std::max(1, P->p.jacobi_sweeps);
  Batch rest = B;
  if (one_launch(P)) {
    a.r = rin;
    a.e0 = P->at<double>(P->o_E0);
    a.x = dst;
    for (const a2d_plan::LineClass& c : P->line_classes)
      if (c.one) launch_lines<TJ>(B, a, P->at<int>(P->o_lcases) + c.first, c.count, c.groups, c.rows, sweeps, s);
    if (P->rest_groups.empty()) return;
    rest.groups = P->at<Group>(P->o_rgroups);
    rest.ngroups = (int)P->rest_groups.size();
  }
  double* bufs[2] = {P->vec(kPA), P->vec(kPB)};
  a.r = rin;
  a.e0 = sweeps > 1 ? P->vec(kPE) : nullptr;
  a.x = sweeps > 1 ? bufs[0] : dst;
  launch_sweep<TJ, true>(rest, a, sweeps == 1, s, P->sweep_variant);
  for (int sw = 1; sw < sweeps; ++sw) {
    const bool last = sw == sweeps - 1;
    a.xprev = a.x;
    a.x = last ? dst : bufs[sw & 1];
    launch_sweep<TJ, false>(rest, a, last, s, P->sweep_variant);
  }
}

template <typename TJ>
static void precond_setup(a2d_plan* P, const Batch& B, uint32_t need, cudaStream_t s) {
  JacArgs ja;
  ja.U = P->vec(kU);
  ja.circ = P->at<double>(P->o_circ);
  ja.JIL = P->at<void>(P->o_JIL);
  ja.JIR = P->at<void>(P->o_JIR);
  ja.JJL = P->at<void>(P->o_JJL);
  ja.JJR = P->at<void>(P->o_JJR);
  ja.vortex = P->p.vortex_correction;
  ja.need = need;
  launch_face_jac<TJ>(B, ja, s);
  launch_factor<TJ, typename FactorStore<TJ>::type>(B, factor_args(P, need), s);
}

// one smoothing of R by the plan's coefficient (> 0): the stage update U = U0 - a (dt / vol) R~, or
// (U0 null) out = R~.  A case's own shape says which kernels take it, whatever it is beside;
// tmp: the smoothed R of those that the fused one does not
static void smoothed(a2d_plan* P, const Batch& B, double* R, const double* U0, double* out, double* tmp, double a,
                     cudaStream_t s) {
  const bool fp32 = P->p.precision == A2D_MIXED;
  if (P->irs_entries > 0) {
    IrsArgs p;
    p.R = R;
    p.U0 = U0;
    p.dt = P->at<double>(P->o_dt);
    p.out = out;
    p.tab = P->at<double>(P->o_irs);
    p.e = P->p.irs_eps;
    p.a = a;
    p.max_ni = P->max_ni;
    p.smem = P->irs_smem;
    launch_irs_fused(B, p, fp32, s);
  }
  if (!P->irs_rest) return;
  launch_irs(B, R, tmp, P->p.irs_eps, P->max_ni, P->max_nc, fp32, s);
  if (U0 != nullptr) launch_rk_stage(B, U0, tmp, P->at<double>(P->o_dt), out, a, true, fp32, s);
}

// the vector of case k, or of all cases (k < 0), one after another
template <int MODE>
static void layout(const a2d_plan* P, int k, const double* src, double* dst, cudaStream_t s) {
  const CaseDev& c = P->cases[k < 0 ? 0 : k];
  launch(k_layout<MODE>, k < 0 ? P->batch.ntiles : c.ntiles, 256, 0, s, P->batch, c.tile0, c.cell_off, src, dst);
}

static StencilArgs<double> residual_args(a2d_plan* P) {
  StencilArgs<double> a;
  a.U = P->vec(kU);
  a.lim_k = P->p.lim_k;
  a.order = P->p.order;
  a.vortex = P->p.vortex_correction;
  return a;
}

// The stencil on the tile list that suits the plan.  A batch whose 16x4 tiles all run at once
// takes these: a small batch is bound by the latency of one tile, whose 148 faces are one round
// of the CTA's 256 threads and the 552 of a 32x8 tile three, while the chip has SMs to spare.
// One 128x48 case: FP32 JVP 14.4 -> 8.4 us, FP64 JVP 25.7 -> 18.4, explicit FP64 residual of
// three 16.1 -> 10.9.  From the second wave on the wider halo costs more than the latency saved:
// 8 cases of 128x48 are 14.4 on either in FP32 and 30.8 on 32x8, 32.8 on 16x4 in FP64; 8 of
// 256x64 are 18.5 and 24.7.  The squared residual sums of a Newton step are per 32x8 tile, so
// its residual keeps these, and a JVP shape that was asked for stays.
template <typename T, bool LIN, typename VT>
static void tile_stencil(const a2d_plan* P, const uint32_t* live, const StencilArgs<VT>& a, cudaStream_t s) {
  constexpr bool knob = LIN && sizeof(T) == 4;
  int shape = knob ? P->jvp_tile : kTile32x8;
  Batch b = knob ? P->jbatch : P->batch;
  const size_t limit = sizeof(T) == 4 ? kFineTiles32 : kFineTiles64;
  if (!P->ftiles.empty() && P->ftiles.size() <= limit && a.tile_part == nullptr &&
      (!knob || P->jvp_tile == kTile32x16)) {
    shape = kTile16x4;
    b = P->fbatch;
  }
  b.live = live;
  launch_stencil<T, LIN, VT>(b, a, s, shape);
}

template <typename TV, typename TJ, typename TB>
static void newton_step_launches(a2d_plan* P, cudaStream_t s) {
  const Batch& B = P->batch;
  const uint32_t NW = kLiveNewton, KR = kLiveNewton | kLiveKrylov;
  double* U = P->vec(kU);
  double* b = P->vec(kB);
  double* x0 = P->vec(kX0);
  double* t = P->vec(kT);
  double* r = P->vec(kRr);
  double* z = P->vec(kZ);
  double* w = P->vec(kW);
  double* dU = P->vec(kDU);
  double* diag = P->at<double>(P->o_diag);
  double* tpart = P->at<double>(P->o_tpart);
  double* cpart = P->at<double>(P->o_cpart);
  double* cpartn = P->at<double>(P->o_cpartn);
  TB* V = P->at<TB>(P->o_V);
  const size_t vs = 4 * (size_t)P->C;
  CaseCtl* ctl = P->ctl();
  uint32_t* live = P->live();

  nvtxRangePushA("newton: residual and line preconditioner");
  launch_mark_stepped(B, live, ctl, s);
  // Newton right-hand side b = -R(U) in FP64, circulation from U, residual-norm partials
  StencilArgs<double> ra = residual_args(P);
  ra.out = b;
  ra.sign = -1.0;
  ra.circ_out = P->at<double>(P->o_circ);
  ra.tile_part = tpart;
  ra.need = NW;
  tile_stencil<double, false>(P, live, ra, s);
  // line preconditioner at U
  precond_setup<TJ>(P, B, NW, s);
  nvtxRangePop();
  nvtxRangePushA("newton: GMRES start");
  // x0 = M b; ptol from ||b||, ||M b||
  precond<TJ>(P, B, b, x0, NW, s);
  launch_norms2(B, b, x0, cpart, P->pstride, NW, s);
  launch_gm_setup(B, cpart, P->pstride, ctl, P->p.gmres_tol, s);
  // t = b - A x0, A v = diag v + J v
  StencilArgs<double> ta = residual_args(P);
  ta.V = x0;
  ta.diag = diag;
  ta.bvec = b;
  ta.out = t;
  ta.need = NW;
  tile_stencil<TV, true>(P, live, ta, s);
  // r = M t, v0 = r / ||r||
  precond<TJ>(P, B, t, r, NW, s);
  double* h1 = P->at<double>(P->o_h1);
  double* h2 = P->at<double>(P->o_h2);
  double* wn0 = P->at<double>(P->o_wn0);
  double* scale = P->at<double>(P->o_scale);
  GsArgs<TB> g0;
  g0.w = r;
  g0.Vout = V;
  g0.part_norm = cpartn;
  g0.need = NW;
  launch_gs_start<TB>(B, g0, s);
  GsCloseArgs c0;
  c0.part_norm = cpartn;
  c0.scale = scale;
  c0.ctl = ctl;
  c0.live = live;
  c0.k = -1;
  c0.need = NW;
  launch_gs_close(B, c0, s);
  nvtxRangePop();
  nvtxRangePushA("newton: Arnoldi");
  for (int k = 0; k < P->m; ++k) {
    StencilArgs<TB> za;
    za.U = U;
    za.V = V + (size_t)k * vs;
    za.vscale = scale + (size_t)k * P->ncases;
    za.diag = diag;
    za.out = z;
    za.lim_k = P->p.lim_k;
    za.order = P->p.order;
    za.vortex = P->p.vortex_correction;
    za.need = KR;
    tile_stencil<TV, true>(P, live, za, s);
    precond<TJ>(P, B, z, w, KR, s);
    // classical Gram-Schmidt run twice, three passes over the basis; passes 2 and 3 reduce
    // the partials of the pass before, so pass 2 writes its own to a second buffer
    GsArgs<TB> g;
    g.w = w;
    g.V = V;
    g.vstride = vs;
    g.nq = k + 1;
    g.pstride = P->pstride;
    g.scale = scale;
    g.need = KR;
    GsCloseArgs ck;
    ck.part_norm = cpartn;
    ck.wn0 = wn0;
    ck.h1 = h1;
    ck.h2 = h2;
    ck.H = P->at<double>(P->o_H);
    ck.scale = scale;
    ck.ctl = ctl;
    ck.live = live;
    ck.k = k;
    ck.need = KR;
    if constexpr (std::is_same<TB, Basis16>::value) {
      if (k < P->gs_vectors) {
        g.Vout = V + (size_t)(k + 1) * vs;
        launch_gs_case(B, g, ck, P->at<uint32_t>(P->o_cnt) + 1, P->gs_cluster, P->max_chunks, s);
        continue;
      }
    }
    GsArgs<TB> gd = g;
    gd.part = cpart;
    launch_gs_dots<TB>(B, gd, s);
    GsArgs<TB> gp = g;
    gp.fold_part = cpart;
    gp.fold_h = h1;
    gp.fold_wn0 = wn0;
    gp.part = P->at<double>(P->o_cpart2);
    launch_gs_project<TB>(B, gp, s);
    GsArgs<TB> gf = g;
    gf.fold_part = P->at<double>(P->o_cpart2);
    gf.fold_h = h2;
    gf.h1 = h1;
    gf.Vout = V + (size_t)(k + 1) * vs;
    gf.part_norm = cpartn;
    launch_gs_finish<TB>(B, gf, s);
    launch_gs_close(B, ck, s);
  }
  nvtxRangePop();
  nvtxRangePushA("newton: least squares and update");
  launch_lstsq(B, live, ctl, P->at<double>(P->o_H), P->at<double>(P->o_y), s);
  CombineArgs<TB> ca;
  ca.x0 = x0;
  ca.V = V;
  ca.vstride = vs;
  ca.y = P->at<double>(P->o_y);
  ca.scale = scale;
  ca.ctl = ctl;
  ca.out = dU;
  ca.need = NW;
  launch_combine<TB>(B, ca, s);
  // positivity step limit, finiteness, per-case controller, commit, forces
  launch_update_rel(B, U, dU, tpart, NW, s);
  launch_update_check(B, U, dU, tpart, ctl, P->p.max_update, NW, s);
  CtlParams cp;
  cp.cfl0 = P->p.cfl0;
  cp.cfl_max = P->p.cfl_max;
  cp.tol = P->p.tol;
  cp.retire = P->p.retire;
  launch_controller(B, tpart, ctl, live, P->at<double>(P->o_hrn), P->p.max_iter, cp, s);
  launch_commit(B, U, dU, ctl, s);
  launch_forces(B, U, P->at<double>(P->o_coef), P->at<double>(P->o_cp), P->at<long long>(P->o_cpoff), ctl,
                P->at<double>(P->o_hcl), P->p.max_iter, s);
  nvtxRangePop();
}

static void newton_dispatch(a2d_plan* P, cudaStream_t s) {
  if (P->p.precision == A2D_MIXED) newton_step_launches<float, float, Basis16>(P, s);
  else newton_step_launches<double, double, double>(P, s);
}

// what the failure word of a plan's kernels stands for
static int wait_failure() {
  return fail(A2D_ERR_CUDA,
              "a bounded wait inside a kernel ran out of time (line sweeps, line factors or a one-launch Arnoldi step)");
}

// the graph of a Newton step, captured on a stream of its own; a failure leaves no error behind
static int build_graph(a2d_plan* P) {
  auto failed = [](const char* what, cudaError_t e) {
    (void)cudaGetLastError();
    return fail(A2D_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  };
  cudaStream_t cap;
  if (cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking)) return failed("graph capture", e);
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    newton_dispatch(P, cap);
    e = cudaStreamEndCapture(cap, &g);
  }
  cudaStreamDestroy(cap);
  if (e != cudaSuccess) return failed("graph capture", e);
  size_t nn = 0;
  if (cudaGraphGetNodes(g, nullptr, &nn) == cudaSuccess && nn > 0) {
    std::vector<cudaGraphNode_t> nodes(nn);
    if (cudaGraphGetNodes(g, nodes.data(), &nn) == cudaSuccess) {
      int nk = 0;
      for (size_t q = 0; q < nn; ++q) {
        cudaGraphNodeType ty;
        if (cudaGraphNodeGetType(nodes[q], &ty) == cudaSuccess && ty == cudaGraphNodeTypeKernel) ++nk;
      }
      P->kernels_per_step = nk;
    }
  }
  cudaGraphExec_t exec = nullptr;
  e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return failed("graph instantiate", e);
  P->graph = exec;
  return A2D_OK;
}

static int newton_step(a2d_plan* P, cudaStream_t s) {
  if (!P->p.use_graph) {
    newton_dispatch(P, s);
    A2D_CK(cudaGetLastError());
    return A2D_OK;
  }
  if (P->graph == nullptr) {
    // a plan's first step goes out kernel by kernel, and the graph of the later ones is captured
    // and instantiated while it runs.  If that fails the step is made all the same; the next
    // one then builds the graph before anything of it runs, so that no error follows a step
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    A2D_CK(cudaStreamIsCapturing(s, &status));
    if (status == cudaStreamCaptureStatusNone && !P->graph_failed) {
      newton_dispatch(P, s);
      A2D_CK(cudaGetLastError());
      P->graph_failed = build_graph(P) != A2D_OK;
      return A2D_OK;
    }
    if (int e = build_graph(P)) return e;
    P->graph_failed = false;
  }
  A2D_CK(cudaGraphLaunch(P->graph, s));
  return A2D_OK;
}

}  // namespace a2d

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
#define A2D_BOUND(P)                                                     \
  do {                                                                   \
    if ((P) == nullptr) return fail(A2D_ERR_ARG, "null plan");           \
    if ((P)->ws == nullptr) return fail(A2D_ERR_STATE, "plan not bound"); \
  } while (0)

extern "C" {

int a2d_version(void) { return 100; }

const char* a2d_last_error(void) { return g_last_error.c_str(); }

void a2d_default_params(a2d_params* p) {
  if (p == nullptr) return;
  p->gmres_restart = 50;
  p->jacobi_sweeps = 4;
  p->gmres_tol = 0.01;
  p->cfl0 = 10.0;
  p->cfl_max = 300.0;
  p->max_update = 0.2;
  p->tol = 1e-8;
  p->cfl = 2.5;
  p->irs_eps = 0.6;
  p->lim_k = 0.02;
  p->order = 2;
  p->vortex_correction = 1;
  p->precision = A2D_FP64;
  p->retire = 1;
  p->max_iter = 200;
  p->use_graph = 1;
}

int a2d_metrics_bytes(int ni, int nj, size_t* bytes) {
  if (bytes == nullptr || ni < 4 || nj < 3) return fail(A2D_ERR_ARG, "metrics: need ni >= 4, nj >= 3");
  *bytes = metrics_total_bytes(ni, nj - 1);
  return A2D_OK;
}

int a2d_metrics_build(int ni, int nj, const double* x, const double* y, void* metrics, void* stream) {
  return a2d_metrics_build_each(1, ni, nj, x, y, &metrics, stream);
}

int a2d_metrics_build_each(int n, int ni, int nj, const double* x, const double* y, void* const* metrics, void* stream) {
  if (x == nullptr || y == nullptr || metrics == nullptr || ni < 4 || nj < 3 || n < 1)
    return fail(A2D_ERR_ARG, "metrics: bad arguments");
  for (int k = 0; k < n; ++k)
    if (metrics[k] == nullptr || reinterpret_cast<uintptr_t>(metrics[k]) % 8 != 0)
      return fail(A2D_ERR_ARG, "metrics: bad arguments");
  launch_metrics(n, ni, nj - 1, x, y, metrics, metrics_float_offset(ni, nj - 1), static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_metrics_build_batch(int n, int ni, int nj, const double* x, const double* y, void* metrics, size_t stride,
                            void* stream) {
  if (x == nullptr || y == nullptr || metrics == nullptr || ni < 4 || nj < 3 || n < 1 || n > 65535 || stride % 8 != 0 ||
      (n > 1 && stride < metrics_total_bytes(ni, nj - 1)))
    return fail(A2D_ERR_ARG, "metrics: bad arguments");
  std::vector<void*> each(n);
  for (int k = 0; k < n; ++k) each[k] = static_cast<char*>(metrics) + stride * k;
  return a2d_metrics_build_each(n, ni, nj, x, y, each.data(), stream);
}

int a2d_plan_create(int ncases, const int* ni, const int* nc, const void* const* metrics, const double* winf,
                    const a2d_params* params, a2d_plan** out) {
  if (out == nullptr || ncases <= 0 || ni == nullptr || nc == nullptr || metrics == nullptr || winf == nullptr)
    return fail(A2D_ERR_ARG, "plan_create: bad arguments");
  a2d_params p;
  a2d_default_params(&p);
  if (params != nullptr) p = *params;
  if (p.gmres_restart < 1 || p.gmres_restart > kMaxRestart)
    return fail(A2D_ERR_ARG, "gmres_restart must be in [1, 64]");
  if (p.jacobi_sweeps < 1) return fail(A2D_ERR_ARG, "jacobi_sweeps must be >= 1");
  if (p.order != 1 && p.order != 2) return fail(A2D_ERR_ARG, "order must be 1 or 2");
  if (p.precision != A2D_FP64 && p.precision != A2D_MIXED) return fail(A2D_ERR_ARG, "unknown precision");
  if (p.max_iter < 1) return fail(A2D_ERR_ARG, "max_iter must be >= 1");
  for (int k = 0; k < ncases; ++k) {
    if (ni[k] < 4 || nc[k] < 2 || metrics[k] == nullptr)
      return fail(A2D_ERR_ARG, "case " + std::to_string(k) + ": need ni >= 4, nc >= 2 and metrics");
  }
  a2d_plan* P = new a2d_plan();
  P->p = p;
  if (p.precision != A2D_MIXED) P->sweep_variant = kSweepLanes;   // rows runs mixed plans only
  P->ncases = ncases;
  P->m = p.gmres_restart;
  P->tj = p.precision == A2D_MIXED ? 4 : 8;
  P->tf = p.precision == A2D_MIXED ? 2 : 8;
  P->tb = p.precision == A2D_MIXED ? sizeof(Basis16) : 8;
  build_tables(P, ni, nc, metrics, winf);
  layout(P);
  *out = P;
  return A2D_OK;
}

int a2d_plan_workspace_bytes(const a2d_plan* P, size_t* bytes) {
  if (P == nullptr || bytes == nullptr) return fail(A2D_ERR_ARG, "null argument");
  *bytes = P->bytes;
  return A2D_OK;
}

int a2d_plan_ncases(const a2d_plan* P) { return P ? P->ncases : 0; }

int a2d_plan_set_tuning(a2d_plan* P, int jvp_tile, int sweep_variant, void* stream) {
  if (P == nullptr) return fail(A2D_ERR_ARG, "null plan");
  if (jvp_tile < 0 || jvp_tile >= kNumTileShapes) return fail(A2D_ERR_ARG, "set_tuning: unknown JVP tile shape");
  if (sweep_variant < 0 || sweep_variant >= kNumSweepVariants)
    return fail(A2D_ERR_ARG, "set_tuning: unknown sweep variant");
  if ((sweep_variant == kSweepRows || sweep_variant == kSweepHalves) && P->p.precision != A2D_MIXED)
    return fail(A2D_ERR_ARG, "set_tuning: the rows and halves sweeps run mixed-precision plans only");
  if (jvp_tile != P->jvp_tile) {
    P->jvp_tile = jvp_tile;
    P->jtiles = tile_list(P, jvp_tile);
    if (P->ws != nullptr) {
      cudaStream_t s = static_cast<cudaStream_t>(stream);
      A2D_CK(cudaMemcpyAsync(P->ws + P->o_jtiles, P->jtiles.data(), sizeof(Tile) * P->jtiles.size(),
                             cudaMemcpyHostToDevice, s));
      A2D_CK(cudaStreamSynchronize(s));
      P->jbatch.ntiles = (int)P->jtiles.size();
    }
  }
  P->sweep_variant = sweep_variant;
  P->graph_failed = false;
  if (P->graph != nullptr) {   // the captured step holds the old launch configuration
    cudaGraphExecDestroy(P->graph);
    P->graph = nullptr;
  }
  return A2D_OK;
}

int a2d_plan_get_tuning(const a2d_plan* P, int* jvp_tile, int* sweep_variant) {
  if (P == nullptr) return fail(A2D_ERR_ARG, "null plan");
  if (jvp_tile != nullptr) *jvp_tile = P->jvp_tile;
  if (sweep_variant != nullptr) *sweep_variant = P->sweep_variant;
  return A2D_OK;
}

int a2d_plan_paths(const a2d_plan* P, unsigned* paths) {
  if (paths == nullptr) return fail(A2D_ERR_ARG, "null output");
  A2D_BOUND(P);
  const bool mixed = P->p.precision == A2D_MIXED;
  unsigned v = 0;
  if (!P->ftiles.empty() && P->ftiles.size() <= (size_t)(mixed ? kFineTiles32 : kFineTiles64)) v |= A2D_PATH_FINE_TILES;
  if (P->rest_groups.size() < P->groups.size()) v |= A2D_PATH_LINES;
  if (!P->rest_groups.empty()) v |= A2D_PATH_SWEEPS;
  if (P->gs_vectors > 0) v |= A2D_PATH_ARNOLDI;
  if (P->irs_entries > 0) v |= A2D_PATH_SMOOTH;
  if (P->irs_rest) v |= A2D_PATH_SMOOTH_ROWS;
  *paths = v;
  return A2D_OK;
}

int a2d_plan_bind(a2d_plan* P, void* workspace, size_t bytes, void* stream) {
  if (P == nullptr || workspace == nullptr) return fail(A2D_ERR_ARG, "bind: null argument");
  if (bytes < P->bytes) return fail(A2D_ERR_ARG, "bind: workspace too small");
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return fail(A2D_ERR_ARG, "bind: workspace not 256-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  P->graph_failed = false;
  if (P->graph != nullptr) {
    cudaGraphExecDestroy(P->graph);
    P->graph = nullptr;
  }
  P->ws = static_cast<char*>(workspace);
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_cases, P->cases.data(), sizeof(CaseDev) * P->ncases,
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_tiles, P->tiles.data(), sizeof(Tile) * P->tiles.size(),
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_chunks, P->chunks.data(), sizeof(Chunk) * P->chunks.size(),
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_groups, P->groups.data(), sizeof(Group) * P->groups.size(),
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_cpoff, P->cp_off.data(), sizeof(long long) * P->ncases,
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemsetAsync(P->ws + P->o_vec[0], 0, P->o_diag - P->o_vec[0], s));
  Batch& B = P->batch;
  B.cases = P->at<CaseDev>(P->o_cases);
  B.tiles = P->at<Tile>(P->o_tiles);
  B.chunks = P->at<Chunk>(P->o_chunks);
  B.groups = P->at<Group>(P->o_groups);
  B.live = P->live();
  B.ncases = P->ncases;
  B.ntiles = (int)P->tiles.size();
  B.nchunks = (int)P->chunks.size();
  B.ngroups = (int)P->groups.size();
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_jtiles, P->jtiles.data(), sizeof(Tile) * P->jtiles.size(),
                         cudaMemcpyHostToDevice, s));
  P->jbatch = B;
  P->jbatch.tiles = P->at<Tile>(P->o_jtiles);
  P->jbatch.ntiles = (int)P->jtiles.size();
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_ftiles, P->ftiles.data(), sizeof(Tile) * P->ftiles.size(),
                         cudaMemcpyHostToDevice, s));
  P->fbatch = B;
  P->fbatch.tiles = P->at<Tile>(P->o_ftiles);
  P->fbatch.ntiles = (int)P->ftiles.size();
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_lcases, P->line_cases.data(), sizeof(int) * P->line_cases.size(),
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemsetAsync(P->ws + P->o_cnt, 0, 8, s));
  A2D_CK(cudaMemsetAsync(P->ws + P->o_sat, 0, sizeof(unsigned long long), s));
  A2D_CK(sweep_init());
  choose_lines(P);
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_rgroups, P->rest_groups.data(), sizeof(Group) * P->rest_groups.size(),
                         cudaMemcpyHostToDevice, s));
  A2D_CK(gs_init());
  // Arnoldi steps in one launch while every case's cluster runs at once (a second wave would cost
  // more than the launches saved); of the cluster sizes the one whose shared memory takes
  // the most vectors, and of these the largest
  P->gs_cluster = P->gs_vectors = 0;
  if (P->p.precision == A2D_MIXED) {
    for (int c = 16; c >= 4 && P->gs_vectors < P->m; --c) {
      const int n = gs_case_vectors(P->ncases, c, P->max_chunks, P->m);
      if (n > P->gs_vectors) {
        P->gs_cluster = c;
        P->gs_vectors = n;
      }
    }
  }
  A2D_CK(irs_init());
  // here and not at the first smoothing, which may be made under capture, where nothing runs
  if (P->irs_entries > 0)
    launch_irs_table(B, P->at<double>(P->o_irs), P->p.irs_eps, P->p.precision == A2D_MIXED, s);
  A2D_CK(factor_init());
  stencil_init_fp64();
  stencil_init_fp32();
  k_reset<<<(P->ncases + 63) / 64, 64, 0, s>>>(P->ncases, P->ctl(), P->live(), P->p.cfl0);
  A2D_CK(cudaMemsetAsync(P->ws + P->o_circ_rk, 0, 8 * (size_t)P->ncases, s));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_plan_destroy(a2d_plan* P) {
  if (P == nullptr) return A2D_OK;
  if (P->graph != nullptr) cudaGraphExecDestroy(P->graph);
  delete P;
  return A2D_OK;
}

static int check_case(const a2d_plan* P, int slot, int k) {
  if (slot < 0 || slot > A2D_VEC_DU) return fail(A2D_ERR_ARG, "unknown vector slot");
  if (k < 0 || k >= P->ncases) return fail(A2D_ERR_ARG, "case index out of range");
  return A2D_OK;
}

int a2d_vec_set(a2d_plan* P, int slot, int k, const double* src, void* stream) {
  A2D_BOUND(P);
  if (int e = check_case(P, slot, k)) return e;
  if (src == nullptr) return fail(A2D_ERR_ARG, "null source");
  layout<kLayoutIn>(P, k, src, P->vec(slot), static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_vec_get(const a2d_plan* P, int slot, int k, double* dst, void* stream) {
  A2D_BOUND(P);
  if (int e = check_case(P, slot, k)) return e;
  if (dst == nullptr) return fail(A2D_ERR_ARG, "null destination");
  layout<kLayoutOut>(P, k, P->vec(slot), dst, static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_vec_get_prim(const a2d_plan* P, int slot, int k, double* dst, void* stream) {
  A2D_BOUND(P);
  if (int e = check_case(P, slot, k)) return e;
  if (dst == nullptr) return fail(A2D_ERR_ARG, "null destination");
  layout<kLayoutPrim>(P, k, P->vec(slot), dst, static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_batch_set(a2d_plan* P, int slot, const double* src, void* stream) {
  A2D_BOUND(P);
  if (int e = check_case(P, slot, 0)) return e;
  if (src == nullptr) return fail(A2D_ERR_ARG, "null source");
  layout<kLayoutIn>(P, -1, src, P->vec(slot), static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_batch_get(const a2d_plan* P, int slot, double* dst, void* stream) {
  A2D_BOUND(P);
  if (int e = check_case(P, slot, 0)) return e;
  if (dst == nullptr) return fail(A2D_ERR_ARG, "null destination");
  layout<kLayoutOut>(P, -1, P->vec(slot), dst, static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_local_dt(const a2d_plan* P, int k, const double* W, double* dt, void* stream) {
  A2D_BOUND(P);
  if (k < 0 || k >= P->ncases) return fail(A2D_ERR_ARG, "local_dt: case index out of range");
  if (W == nullptr || dt == nullptr) return fail(A2D_ERR_ARG, "local_dt: null pointer");
  launch_local_dt_prim(P->cases[k].g, W, dt, P->p.cfl, static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_init_freestream(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_init_state<<<P->batch.ntiles, 256, 0, s>>>(P->batch, P->vec(kU));
  k_reset<<<(P->ncases + 63) / 64, 64, 0, s>>>(P->ncases, P->ctl(), P->live(), P->p.cfl0);
  A2D_CK(cudaGetLastError());
  P->steps_taken = 0;
  return A2D_OK;
}

int a2d_reset(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  k_reset<<<(P->ncases + 63) / 64, 64, 0, static_cast<cudaStream_t>(stream)>>>(P->ncases, P->ctl(), P->live(),
                                                                                P->p.cfl0);
  A2D_CK(cudaGetLastError());
  P->steps_taken = 0;
  return A2D_OK;
}

int a2d_case_restart(a2d_plan* P, int n, const int* cases, const double* winf, int keep_state, void* stream) {
  A2D_BOUND(P);
  if (n < 0 || n > P->ncases || (n > 0 && (cases == nullptr || winf == nullptr)))
    return fail(A2D_ERR_ARG, "case_restart: bad arguments");
  if (n == 0) return A2D_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int q = 0; q < n; ++q) {
    const int k = cases[q];
    if (k < 0 || k >= P->ncases) return fail(A2D_ERR_ARG, "case_restart: case index out of range");
    for (int c = 0; c < 4; ++c) P->cases[k].winf[c] = winf[4 * q + c];
  }
  // the per-case table and the index list; pageable sources are staged before the call returns
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_cases, P->cases.data(), sizeof(CaseDev) * P->ncases,
                         cudaMemcpyHostToDevice, s));
  A2D_CK(cudaMemcpyAsync(P->at<int>(P->o_idx), cases, sizeof(int) * n, cudaMemcpyHostToDevice, s));
  k_restart_cases<<<n, 256, 0, s>>>(P->batch, P->at<int>(P->o_idx), keep_state, P->vec(kU), P->ctl(), P->live(),
                                    P->p.cfl0);
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_case_forces(a2d_plan* P, double* coef, double* cp, void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Batch B = P->batch;
  B.live = nullptr;
  launch_forces(B, P->vec(kU), P->at<double>(P->o_coef), P->at<double>(P->o_cp), P->at<long long>(P->o_cpoff),
                nullptr, nullptr, 0, s);
  if (coef != nullptr)
    A2D_CK(cudaMemcpyAsync(coef, P->at<double>(P->o_coef), 8 * 3 * (size_t)P->ncases, cudaMemcpyDeviceToHost, s));
  if (cp != nullptr)
    A2D_CK(cudaMemcpyAsync(cp, P->at<double>(P->o_cp), 8 * (size_t)P->total_ni, cudaMemcpyDeviceToHost, s));
  A2D_CK(cudaStreamSynchronize(s));
  return A2D_OK;
}

int a2d_case_set_grid(a2d_plan* P, int n, const int* cases, const void* const* metrics, void* stream) {
  A2D_BOUND(P);
  if (n < 0 || n > P->ncases || (n > 0 && (cases == nullptr || metrics == nullptr)))
    return fail(A2D_ERR_ARG, "case_set_grid: bad arguments");
  if (n == 0) return A2D_OK;
  for (int q = 0; q < n; ++q) {
    const int k = cases[q];
    if (k < 0 || k >= P->ncases) return fail(A2D_ERR_ARG, "case_set_grid: case index out of range");
    if (metrics[q] == nullptr) return fail(A2D_ERR_ARG, "case_set_grid: null metrics");
  }
  for (int q = 0; q < n; ++q) {
    CaseDev& c = P->cases[cases[q]];
    c.g = grid_view(metrics[q], c.g.ni, c.g.nc);
  }
  A2D_CK(cudaMemcpyAsync(P->ws + P->o_cases, P->cases.data(), sizeof(CaseDev) * P->ncases, cudaMemcpyHostToDevice,
                         static_cast<cudaStream_t>(stream)));
  return A2D_OK;
}

int a2d_case_retire(a2d_plan* P, int n, const int* cases, void* stream) {
  A2D_BOUND(P);
  if (n < 0 || n > P->ncases || (n > 0 && cases == nullptr)) return fail(A2D_ERR_ARG, "case_retire: bad arguments");
  if (n == 0) return A2D_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int q = 0; q < n; ++q)
    if (cases[q] < 0 || cases[q] >= P->ncases) return fail(A2D_ERR_ARG, "case_retire: case index out of range");
  A2D_CK(cudaMemcpyAsync(P->at<int>(P->o_idx), cases, sizeof(int) * n, cudaMemcpyHostToDevice, s));
  k_retire_cases<<<(n + 63) / 64, 64, 0, s>>>(P->at<int>(P->o_idx), n, P->live());
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_residual(a2d_plan* P, const double* circ, void* stream) {
  A2D_BOUND(P);
  StencilArgs<double> a = residual_args(P);
  a.circ_in = circ;
  a.out = P->vec(kR);
  a.sign = 1.0;
  a.circ_out = P->at<double>(P->o_circ);
  tile_stencil<double, false>(P, nullptr, a, static_cast<cudaStream_t>(stream));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_residual_of(a2d_plan* P, int k, const double* U, const double* circ, double* R, double* W, void* stream) {
  A2D_BOUND(P);
  if (U == nullptr || R == nullptr || W == nullptr) return fail(A2D_ERR_ARG, "residual_of: null pointer");
  if (int e = a2d_vec_set(P, A2D_VEC_U, k, U, stream)) return e;
  if (int e = a2d_residual(P, circ, stream)) return e;
  const CaseDev& c = P->cases[k];
  launch(k_layout_residual, dim3(c.ntiles, 2), 256, 0, static_cast<cudaStream_t>(stream), P->batch, c.tile0, c.cell_off,
         P->vec(kR), R, P->vec(kU), W);
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_jvp(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  StencilArgs<double> a = residual_args(P);
  a.V = P->vec(kVin);
  a.out = P->vec(kJV);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (P->p.precision == A2D_MIXED) tile_stencil<float, true>(P, nullptr, a, s);
  else tile_stencil<double, true>(P, nullptr, a, s);
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_forces(a2d_plan* P, double* coef, double* cp, void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Batch B = P->batch;
  B.live = nullptr;
  launch_forces(B, P->vec(kU), P->at<double>(P->o_coef), P->at<double>(P->o_cp), P->at<long long>(P->o_cpoff),
                nullptr, nullptr, 0, s);
  if (coef != nullptr)
    A2D_CK(cudaMemcpyAsync(coef, P->at<double>(P->o_coef), 8 * 3 * (size_t)P->ncases, cudaMemcpyDeviceToDevice, s));
  if (cp != nullptr)
    A2D_CK(cudaMemcpyAsync(cp, P->at<double>(P->o_cp), 8 * (size_t)P->total_ni, cudaMemcpyDeviceToDevice, s));
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_set_cfl(a2d_plan* P, const double* cfl, void* stream) {
  A2D_BOUND(P);
  if (cfl == nullptr) return fail(A2D_ERR_ARG, "null cfl");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int k = 0; k < P->ncases; ++k)
    A2D_CK(cudaMemcpyAsync(&P->ctl()[k].cfl, &cfl[k], sizeof(double), cudaMemcpyHostToDevice, s));
  A2D_CK(cudaStreamSynchronize(s));
  return A2D_OK;
}

int a2d_precond_setup(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // circulation of U for the far-field block (as the Newton step forms it)
  StencilArgs<double> a = residual_args(P);
  a.out = P->vec(kB);
  a.sign = -1.0;
  a.circ_out = P->at<double>(P->o_circ);
  a.tile_part = P->at<double>(P->o_tpart);
  Batch B = P->batch;
  B.live = nullptr;
  launch_stencil<double, false, double>(B, a, s);
  if (P->p.precision == A2D_MIXED) precond_setup<float>(P, B, 0, s);
  else precond_setup<double>(P, B, 0, s);
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_precond_apply(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Batch B = P->batch;
  B.live = nullptr;
  if (P->p.precision == A2D_MIXED) precond<float>(P, B, P->vec(kVin), P->vec(kJV), 0, s);
  else precond<double>(P, B, P->vec(kVin), P->vec(kJV), 0, s);
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_newton_step(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  Range range("a2d_newton_step");
  const int e = newton_step(P, static_cast<cudaStream_t>(stream));
  if (e == A2D_OK) P->steps_taken += 1;
  return e;
}

int a2d_newton_run(a2d_plan* P, int max_steps, int* steps, void* stream) {
  A2D_BOUND(P);
  Range range("a2d_newton_run");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int done = 0;
  int* dcount = P->at<int>(P->o_cnt);
  for (int it = 0; it < max_steps; ++it) {
    if (P->steps_taken >= P->p.max_iter) break;
    if (int e = newton_step(P, s)) return e;
    P->steps_taken += 1;
    ++done;
    k_count<<<1, 256, 0, s>>>(P->ncases, P->ctl(), P->live(), P->p.retire, dcount);
    A2D_CK(cudaMemcpyAsync(P->host_count, dcount, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    A2D_CK(cudaStreamSynchronize(s));
    if (P->host_count[1] != 0) return wait_failure();
    if (*P->host_count == 0) break;
  }
  if (steps != nullptr) *steps = done;
  return A2D_OK;
}

int a2d_factor_saturations(a2d_plan* P, unsigned long long* count, int reset, void* stream) {
  A2D_BOUND(P);
  if (count == nullptr) return fail(A2D_ERR_ARG, "null output");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  A2D_CK(cudaMemcpyAsync(count, P->ws + P->o_sat, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  if (reset) A2D_CK(cudaMemsetAsync(P->ws + P->o_sat, 0, sizeof(unsigned long long), s));
  A2D_CK(cudaStreamSynchronize(s));
  return A2D_OK;
}

int a2d_live_count(a2d_plan* P, int* n, void* stream) {
  A2D_BOUND(P);
  if (n == nullptr) return fail(A2D_ERR_ARG, "null output");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int* dcount = P->at<int>(P->o_cnt);
  k_count<<<1, 256, 0, s>>>(P->ncases, P->ctl(), P->live(), P->p.retire, dcount);
  A2D_CK(cudaMemcpyAsync(P->host_count, dcount, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
  A2D_CK(cudaStreamSynchronize(s));
  if (P->host_count[1] != 0) return wait_failure();
  *n = *P->host_count;
  return A2D_OK;
}

int a2d_plan_stats(const a2d_plan* P, int* kernels_per_step, int* steps_taken, size_t* table_bytes) {
  if (P == nullptr) return fail(A2D_ERR_ARG, "null plan");
  if (kernels_per_step) *kernels_per_step = P->kernels_per_step;
  if (steps_taken) *steps_taken = P->steps_taken;
  if (table_bytes)
    *table_bytes = sizeof(CaseDev) * P->ncases + sizeof(Tile) * P->tiles.size() + sizeof(Chunk) * P->chunks.size() +
                   sizeof(Group) * P->groups.size() + sizeof(long long) * P->ncases;
  return A2D_OK;
}

int a2d_time_kernel(a2d_plan* P, int which, int reps, float* ms, void* stream) {
  A2D_BOUND(P);
  if (ms == nullptr || reps < 1) return fail(A2D_ERR_ARG, "time_kernel: bad arguments");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Batch B = P->batch;
  B.live = nullptr;
  const bool mixed = P->p.precision == A2D_MIXED;
  const size_t vs = 4 * (size_t)P->C;
  const int half = std::max(1, P->m / 2);
  // where the sweeps of an application are one launch, that launch is timed and its
  // time shared between them
  const bool whole = one_launch(P) && (which == A2D_K_SWEEP || which == A2D_K_SWEEP_FIRST);
  auto launch_once = [&]() {
    switch (which) {
      case A2D_K_JVP: {
        if (mixed) {
          StencilArgs<Basis16> a;
          a.U = P->vec(kU);
          a.V = P->at<Basis16>(P->o_V);
          a.diag = P->at<double>(P->o_diag);
          a.out = P->vec(kZ);
          a.lim_k = P->p.lim_k;
          a.order = P->p.order;
          a.vortex = P->p.vortex_correction;
          tile_stencil<float, true>(P, nullptr, a, s);
        } else {
          StencilArgs<double> a = residual_args(P);
          a.V = P->at<double>(P->o_V);
          a.diag = P->at<double>(P->o_diag);
          a.out = P->vec(kZ);
          tile_stencil<double, true>(P, nullptr, a, s);
        }
        break;
      }
      case A2D_K_SWEEP: {
        if (whole) {
          if (mixed) precond<float>(P, B, P->vec(kZ), P->vec(kT), 0, s);
          else precond<double>(P, B, P->vec(kZ), P->vec(kT), 0, s);
          break;
        }
        SweepArgs a = sweep_args(P, 0);
        a.e0 = P->vec(kPE);
        a.xprev = P->vec(kPB);
        a.x = P->vec(kPA);
        if (mixed) launch_sweep<float, false>(B, a, false, s, P->sweep_variant);
        else launch_sweep<double, false>(B, a, false, s, P->sweep_variant);
        break;
      }
      case A2D_K_SWEEP_FIRST: {
        if (whole) {
          if (mixed) precond<float>(P, B, P->vec(kZ), P->vec(kT), 0, s);
          else precond<double>(P, B, P->vec(kZ), P->vec(kT), 0, s);
          break;
        }
        SweepArgs a = sweep_args(P, 0);
        a.r = P->vec(kZ);
        a.e0 = P->vec(kPE);
        a.x = P->vec(kPA);
        if (mixed) launch_sweep<float, true>(B, a, false, s, P->sweep_variant);
        else launch_sweep<double, true>(B, a, false, s, P->sweep_variant);
        break;
      }
      case A2D_K_DOTS:
      case A2D_K_UPDATE:
      case A2D_K_PROJECT: {
        // Gram-Schmidt passes with restart/2 basis vectors; the output vector is a
        // scratch slot past the ones read
        auto run = [&](auto* Vb) {
          using TB = std::remove_pointer_t<decltype(Vb)>;
          GsArgs<TB> g;
          g.w = P->vec(kW);
          g.V = Vb;
          g.vstride = vs;
          g.nq = half;
          g.part = P->at<double>(which == A2D_K_PROJECT ? P->o_cpart2 : P->o_cpart);
          g.pstride = P->pstride;
          g.fold_part = P->at<double>(which == A2D_K_PROJECT ? P->o_cpart : P->o_cpart2);
          g.fold_h = P->at<double>(P->o_h2);
          g.h1 = P->at<double>(P->o_h1);
          g.scale = P->at<double>(P->o_scale);
          g.Vout = Vb + (size_t)P->m * vs;
          g.part_norm = P->at<double>(P->o_cpartn);
          if (which == A2D_K_DOTS) launch_gs_dots<TB>(B, g, s);
          else if (which == A2D_K_PROJECT) launch_gs_project<TB>(B, g, s);
          else launch_gs_finish<TB>(B, g, s);
        };
        if (mixed) run(P->at<Basis16>(P->o_V));
        else run(P->at<double>(P->o_V));
        break;
      }
      case A2D_K_RESIDUAL: {
        StencilArgs<double> a = residual_args(P);
        a.out = P->vec(kPA);
        a.sign = -1.0;
        a.circ_out = P->at<double>(P->o_circ);
        a.tile_part = P->at<double>(P->o_tpart);
        launch_stencil<double, false, double>(B, a, s);
        break;
      }
      case A2D_K_FACEJAC:
      case A2D_K_FACTOR: {
        JacArgs ja;
        ja.U = P->vec(kU);
        ja.circ = P->at<double>(P->o_circ);
        ja.JIL = P->at<void>(P->o_JIL);
        ja.JIR = P->at<void>(P->o_JIR);
        ja.JJL = P->at<void>(P->o_JJL);
        ja.JJR = P->at<void>(P->o_JJR);
        ja.vortex = P->p.vortex_correction;
        if (which == A2D_K_FACEJAC) {
          if (mixed) launch_face_jac<float>(B, ja, s);
          else launch_face_jac<double>(B, ja, s);
        } else {
          const FactorArgs fa = factor_args(P, 0);
          if (mixed) launch_factor<float, __half>(B, fa, s);
          else launch_factor<double, double>(B, fa, s);
        }
        break;
      }
      default:
        break;
    }
  };
  if (which < 0 || which > A2D_K_PROJECT) return fail(A2D_ERR_ARG, "time_kernel: unknown kernel");
  cudaEvent_t e0, e1;
  A2D_CK(cudaEventCreate(&e0));
  A2D_CK(cudaEventCreate(&e1));
  launch_once();   // warm-up launch
  A2D_CK(cudaEventRecord(e0, s));
  for (int q = 0; q < reps; ++q) launch_once();
  A2D_CK(cudaEventRecord(e1, s));
  A2D_CK(cudaEventSynchronize(e1));
  float t = 0.f;
  A2D_CK(cudaEventElapsedTime(&t, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  A2D_CK(cudaGetLastError());
  *ms = t / reps / (whole ? std::max(1, P->p.jacobi_sweeps) : 1);
  return A2D_OK;
}

int a2d_case_status(const a2d_plan* P, int* nsteps, int* done, int* frozen, double* lastrn, double* r0,
                    void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  std::vector<CaseCtl> h(P->ncases);
  A2D_CK(cudaMemcpyAsync(h.data(), P->ctl(), sizeof(CaseCtl) * P->ncases, cudaMemcpyDeviceToHost, s));
  A2D_CK(cudaStreamSynchronize(s));
  for (int k = 0; k < P->ncases; ++k) {
    if (nsteps) nsteps[k] = h[k].nsteps;
    if (done) done[k] = h[k].done;
    if (frozen) frozen[k] = h[k].frozen;
    if (lastrn) lastrn[k] = h[k].lastrn;
    if (r0) r0[k] = h[k].r0;
  }
  return A2D_OK;
}

int a2d_case_scalars(const a2d_plan* P, double* out, void* stream) {
  A2D_BOUND(P);
  if (out == nullptr) return fail(A2D_ERR_ARG, "null output");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  std::vector<CaseCtl> h(P->ncases);
  std::vector<double> circ(P->ncases);
  A2D_CK(cudaMemcpyAsync(h.data(), P->ctl(), sizeof(CaseCtl) * P->ncases, cudaMemcpyDeviceToHost, s));
  A2D_CK(cudaMemcpyAsync(circ.data(), P->at<double>(P->o_circ), 8 * (size_t)P->ncases, cudaMemcpyDeviceToHost, s));
  A2D_CK(cudaStreamSynchronize(s));
  for (int k = 0; k < P->ncases; ++k) {
    double* o = out + 8 * (size_t)k;
    o[0] = h[k].rn;
    o[1] = h[k].omega;
    o[2] = h[k].cfl;
    o[3] = h[k].r0;
    o[4] = circ[k];
    o[5] = h[k].beta;
    o[6] = (double)h[k].k_used;
    o[7] = (double)h[k].commit;
  }
  return A2D_OK;
}

int a2d_history(const a2d_plan* P, int steps, double* rn, double* cl, void* stream) {
  A2D_BOUND(P);
  if (steps < 0 || steps > P->p.max_iter) return fail(A2D_ERR_ARG, "history: steps out of range");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t n = (size_t)steps * P->ncases * 8;
  if (rn != nullptr && n) A2D_CK(cudaMemcpyAsync(rn, P->at<double>(P->o_hrn), n, cudaMemcpyDeviceToHost, s));
  if (cl != nullptr && n) A2D_CK(cudaMemcpyAsync(cl, P->at<double>(P->o_hcl), n, cudaMemcpyDeviceToHost, s));
  A2D_CK(cudaStreamSynchronize(s));
  return A2D_OK;
}

int a2d_set_circulation(a2d_plan* P, const double* circ, void* stream) {
  A2D_BOUND(P);
  if (circ == nullptr) return fail(A2D_ERR_ARG, "null circulation");
  A2D_CK(cudaMemcpyAsync(P->at<double>(P->o_circ_rk), circ, 8 * (size_t)P->ncases, cudaMemcpyHostToDevice,
                         static_cast<cudaStream_t>(stream)));
  return A2D_OK;
}

int a2d_smooth(a2d_plan* P, void* stream) {
  A2D_BOUND(P);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Batch B = P->batch;
  B.live = nullptr;
  if (P->p.irs_eps > 0) {
    smoothed(P, B, P->vec(kR), nullptr, P->vec(kPA), P->vec(kPA), 0.0, s);
    A2D_CK(cudaMemcpyAsync(P->vec(kR), P->vec(kPA), 8 * 4 * (size_t)P->C, cudaMemcpyDeviceToDevice, s));
  }
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_plan_set_coarse(a2d_plan* P, a2d_plan* coarse) {
  if (P == nullptr) return fail(A2D_ERR_ARG, "null plan");
  if (coarse != nullptr) {
    if (coarse == P || coarse->ncases != P->ncases) return fail(A2D_ERR_ARG, "set_coarse: not the same cases");
    for (int k = 0; k < P->ncases; ++k) {
      const GridDev& f = P->cases[k].g;
      const GridDev& c = coarse->cases[k].g;
      if (f.ni % 2 || f.nc % 2 || c.ni * 2 != f.ni || c.nc * 2 != f.nc)
        return fail(A2D_ERR_ARG, "set_coarse: the coarse grids must have ni/2 x nc/2 cells (even ni, nc)");
    }
    for (const a2d_plan* q = coarse; q != nullptr; q = q->coarse)
      if (q == P) return fail(A2D_ERR_ARG, "set_coarse: the levels would form a cycle");
  }
  P->coarse = coarse;
  return A2D_OK;
}

}  // extern "C"

namespace a2d {

// one 4-stage RK iteration of plan P (aero2d/euler.py:334-346): residual at the
// circulation circ (per case), plus the FAS forcing when given, smoothed, stage update
static cudaError_t rk_iter(a2d_plan* P, const double* circ, const double* forcing, cudaStream_t s) {
  Batch B = P->batch;
  B.live = nullptr;
  double* U = P->vec(kU);
  double* U0 = P->vec(kU0);
  double* R = P->vec(kR);
  double* dt = P->at<double>(P->o_dt);
  const double alphas[4] = {0.25, 1.0 / 3.0, 0.5, 1.0};
  // dtype=float32: residual, local time steps, smoothing and stage update in FP32
  // (the reference casts its whole explicit iteration to the solver dtype,
  // aero2d/euler.py:222-234); the state keeps FP32-rounded values in FP64 storage
  const bool fp32 = P->p.precision == A2D_MIXED;
  launch_local_dt(B, U, U0, dt, P->p.cfl, fp32, s);
  for (int st = 0; st < 4; ++st) {
    StencilArgs<double> a = residual_args(P);
    a.circ_in = circ;
    a.out = R;
    a.sign = 1.0;
    if (fp32) tile_stencil<float, false>(P, nullptr, a, s);
    else tile_stencil<double, false>(P, nullptr, a, s);
    if (forcing != nullptr) launch_add_forcing(B, R, forcing, s);
    if (P->p.irs_eps > 0) smoothed(P, B, R, U0, U, P->vec(kPA), alphas[st], s);
    else launch_rk_stage(B, U0, R, dt, U, alphas[st], false, fp32, s);
  }
  return cudaGetLastError();
}

// one FAS V-cycle from plan P down (aero2d/euler.py:368-381); at the top level
// the pseudo-time residual of the first iteration goes to the tile partials
static cudaError_t fas_cycle(a2d_plan* P, const double* circ, const double* forcing, bool top, cudaStream_t s) {
  Batch B = P->batch;
  B.live = nullptr;
  if (cudaError_t e = rk_iter(P, circ, forcing, s)) return e;
  if (top) launch_rk_res(B, P->vec(kU0), P->vec(kU), P->at<double>(P->o_dt), P->at<double>(P->o_tpart), s);
  a2d_plan* Cp = P->coarse;
  if (Cp == nullptr) return cudaGetLastError();
  Batch CB = Cp->batch;
  CB.live = nullptr;
  // fine residual (plus this level's forcing) at the smoothed state
  StencilArgs<double> a = residual_args(P);
  a.circ_in = circ;
  a.out = P->vec(kR);
  a.sign = 1.0;
  if (P->p.precision == A2D_MIXED) tile_stencil<float, false>(P, nullptr, a, s);
  else tile_stencil<double, false>(P, nullptr, a, s);
  if (forcing != nullptr) launch_add_forcing(B, P->vec(kR), forcing, s);
  // coarse start state Uc0 (kept in the coarse plan's JV slot) and forcing (its V slot)
  double* Uc = Cp->vec(kU);
  double* Uc0 = Cp->vec(kJV);
  double* Pc = Cp->vec(kVin);
  launch_fas_restrict(B, CB, P->vec(kU), Uc, Uc0, s);
  StencilArgs<double> ca = residual_args(Cp);
  ca.circ_in = circ;
  ca.out = Pc;
  ca.sign = 1.0;
  if (Cp->p.precision == A2D_MIXED) tile_stencil<float, false>(Cp, nullptr, ca, s);
  else tile_stencil<double, false>(Cp, nullptr, ca, s);
  launch_fas_forcing(B, CB, P->vec(kR), Pc, s);
  if (cudaError_t e = fas_cycle(Cp, circ, Pc, false, s)) return e;
  launch_fas_prolong(B, CB, P->vec(kU), Uc, Uc0, s);
  return rk_iter(P, circ, forcing, s);
}

}  // namespace a2d

extern "C" {

int a2d_rk_iterate(a2d_plan* P, int n, double* res, void* stream) {
  A2D_BOUND(P);
  Range range("a2d_rk_iterate");
  if (n < 0) return fail(A2D_ERR_ARG, "negative iteration count");
  for (const a2d_plan* q = P->coarse; q != nullptr; q = q->coarse)
    if (q->ws == nullptr) return fail(A2D_ERR_STATE, "rk_iterate: a coarse level is not bound");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Batch B = P->batch;
  B.live = nullptr;
  double* circ = P->at<double>(P->o_circ_rk);
  double* tpart = P->at<double>(P->o_tpart);
  for (int it = 0; it < n; ++it) {
    A2D_CK(fas_cycle(P, circ, nullptr, true, s));
    launch_forces(B, P->vec(kU), P->at<double>(P->o_coef), P->at<double>(P->o_cp), P->at<long long>(P->o_cpoff), nullptr,
                  nullptr, 0, s);
    launch_rk_finish(B, tpart, P->at<double>(P->o_coef), (it == n - 1) ? res : nullptr, circ, s);
  }
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

int a2d_hllc_flux(int n, const double* WL, const double* WR, const double* S, double* F, void* stream) {
  if (n < 0 || (n > 0 && (WL == nullptr || WR == nullptr || S == nullptr || F == nullptr)))
    return fail(A2D_ERR_ARG, "hllc_flux: bad arguments");
  if (n == 0) return A2D_OK;
  k_point_flux<<<(n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(n, WL, WR, S, F);
  A2D_CK(cudaGetLastError());
  return A2D_OK;
}

}  // extern "C"
