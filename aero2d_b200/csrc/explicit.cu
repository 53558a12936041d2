// Explicit 4-stage Runge-Kutta pseudo-time stepping with local time steps and
// implicit residual smoothing, the fallback solver of aero2d/euler.py:289-346.
//
// Smoothing along i (periodic, constant coefficients -e, 1+2e, -e) is the
// exact solution of the circulant system, which the reference obtains by FFT
// (euler.py:302-303).  Here it is applied through the system's periodic Green's
// function g_m = G0 (l^m + l^(n-m)) / (1 - l^n), l the root in (0,1) of
// e l^2 - (1+2e) l + e = 0 and G0 = 1 / (e (1/l - l)); terms with l^|m| below
// 1e-18 of the diagonal are dropped, so results equal the FFT's to rounding.
// Smoothing along j is a Thomas solve of (-e, 1+2e, -e) with end diagonals 1+e.
#include <algorithm>
#include <cmath>

#include "batch.cuh"
#include "explicit.cuh"
#include "launch.cuh"
#include "physics.cuh"
#include "quotient.cuh"

namespace a2d {

// local time step of cell (j, i) from its primitives W = (rho, u, v, p):
// dt = cfl vol / (lambda_i + lambda_j), face vectors averaged to the cell
// centre, in the operation order of euler.py:289-296; T is the compute type
// (FP32 reads the grid's FP32 metric copies)
template <typename T>
__device__ __forceinline__ T local_dt_cell(const GridDev& g, const State4<T>& W, int j, int i, T cfl) {
  const Metric<T> m{g};
  const int ip = (i + 1 == g.ni) ? 0 : i + 1;
  const T cc = sqrt(T(kGamma) * W.c[3] / W.c[0]);
  const T s0 = T(0.5) * (m.si(0, j, i) + m.si(0, j, ip));
  const T s1 = T(0.5) * (m.si(1, j, i) + m.si(1, j, ip));
  const T t0 = T(0.5) * (m.sj(0, j + 1, i) + m.sj(0, j, i));
  const T t1 = T(0.5) * (m.sj(1, j + 1, i) + m.sj(1, j, i));
  const T li = fabs(W.c[1] * s0 + W.c[2] * s1) + cc * sqrt(s0 * s0 + s1 * s1);
  const T lj = fabs(W.c[1] * t0 + W.c[2] * t1) + cc * sqrt(t0 * t0 + t1 * t1);
  return cfl * m.vol(j, i) / (li + lj);
}

// local time steps of every case from its conserved state, which is kept as the
// iteration's start state U0 (the RK iteration)
template <typename T>
__global__ void __launch_bounds__(256) k_local_dt(Batch b, const double* __restrict__ U, double* __restrict__ U0,
                                                  double* __restrict__ dt, double cfl) {
  grid_wait();
  const Tile t = b.tiles[blockIdx.x];
  const CaseDev cs = b.cases[t.cs];
  const GridDev& g = cs.g;
  const double* Uc = U + 4 * cs.cell_off;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int j = t.j0 + c / t.ti, i = t.i0 + c % t.ti;
    State4<T> u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double v = Uc[vidx(g, k, j, i)];
      U0[4 * cs.cell_off + vidx(g, k, j, i)] = v;
      u.c[k] = T(v);
    }
    dt[cs.cell_off + (size_t)j * g.ni + i] = (double)local_dt_cell<T>(g, cons_to_prim<T, T>(u), j, i, T(cfl));
  }
}

// local time steps of one case from primitives given in the reference layout
// W[4][ni][nc], written as dt[ni][nc] (EulerSolver.local_dt, euler.py:289-296)
__global__ void __launch_bounds__(256) k_local_dt_prim(GridDev g, const double* __restrict__ W,
                                                       double* __restrict__ dt, double cfl) {
  const size_t N = (size_t)g.ni * g.nc;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < N; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / g.nc), j = (int)(q % g.nc);
    State4<double> w;
#pragma unroll
    for (int k = 0; k < 4; ++k) w.c[k] = W[k * N + q];
    dt[q] = local_dt_cell<double>(g, w, j, i, cfl);
  }
}

// periodic smoothing along i: one block per (case, component, row j); T is the
// compute type (values stay in FP64 arrays, rounded to T when T is FP32)
template <typename T>
__global__ void __launch_bounds__(256) k_irs_i(Batch b, const double* __restrict__ R, double* __restrict__ out,
                                               double e_, int reach) {
  grid_wait();
  const int row = blockIdx.x;   // rows enumerated as (case, k, j) via the row table below
  const int cs_id = blockIdx.y;
  const CaseDev cs = b.cases[cs_id];
  if (cs.irs_off >= 0) return;   // k_irs takes it
  const GridDev& g = cs.g;
  const int ni = g.ni, nc = g.nc;
  if (row >= 4 * nc) return;
  const int k = row / nc, j = row % nc;
  extern __shared__ __align__(8) unsigned char irs_sm[];
  T* r = reinterpret_cast<T*>(irs_sm);   // ni
  T* gm = r + ni;                         // up to ni/2 + 1
  const double* src = R + 4 * cs.cell_off + vidx(g, k, j, 0);
  for (int i = threadIdx.x; i < ni; i += blockDim.x) r[i] = T(src[i]);
  // the Green's function in FP64, then rounded to T (its terms below 1e-18 of
  // the diagonal dropped: the FFT's solution to rounding)
  const double e = e_;
  const double lam = ((1.0 + 2.0 * e) - sqrt(1.0 + 4.0 * e)) / (2.0 * e);
  const double G0 = 1.0 / (e * (1.0 / lam - lam));
  const int M = min(reach, ni / 2);
  const double ln = pow(lam, (double)ni);
  for (int m = threadIdx.x; m <= M; m += blockDim.x)
    gm[m] = T(G0 * (pow(lam, (double)m) + pow(lam, (double)(ni - m))) / (1.0 - ln));
  __syncthreads();
  double* dst = out + 4 * cs.cell_off + vidx(g, k, j, 0);
  const bool full = (2 * M + 1 >= ni);
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    T s = gm[0] * r[i];
    if (full) {
      for (int d = 1; d < ni; ++d) {
        const int m = d <= ni / 2 ? d : ni - d;
        int q = i - d;
        if (q < 0) q += ni;
        s += gm[m] * r[q];
      }
    } else {
      for (int m = 1; m <= M; ++m) {
        int qm = i - m, qp = i + m;
        if (qm < 0) qm += ni;
        if (qp >= ni) qp -= ni;
        s += gm[m] * (r[qm] + r[qp]);
      }
    }
    dst[i] = (double)s;
  }
}

// smoothing along j: Thomas solve per (case, component, line i); thread per line.
// The elimination coefficients depend on j only and are formed once per block.
template <typename T>
__global__ void __launch_bounds__(128) k_irs_j(Batch b, double* __restrict__ R, double e_) {
  grid_wait();
  const int cs_id = blockIdx.y;
  const CaseDev cs = b.cases[cs_id];
  if (cs.irs_off >= 0) return;
  const GridDev& g = cs.g;
  const int ni = g.ni, nc = g.nc;
  extern __shared__ __align__(8) unsigned char irs_sm[];
  T* cpj = reinterpret_cast<T*>(irs_sm);   // nc
  const T e = T(e_);
  if (threadIdx.x == 0) {
    T cp = T(0);
    for (int j = 0; j < nc; ++j) {
      const T dj = (j == 0 || j == nc - 1) ? T(1) + e : T(1) + T(2) * e;
      const T lj = (j == 0) ? T(0) : -e;
      const T uj = (j == nc - 1) ? T(0) : -e;
      cp = uj / (dj - lj * cp);
      cpj[j] = cp;
    }
  }
  __syncthreads();
  const int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= 4 * ni) return;
  const int k = line / ni, i = line % ni;
  double* x = R + 4 * cs.cell_off;
  T dprev = T(0);
  for (int j = 0; j < nc; ++j) {
    const T dj = (j == 0 || j == nc - 1) ? T(1) + e : T(1) + T(2) * e;
    const T lj = (j == 0) ? T(0) : -e;
    const T den = dj - lj * (j == 0 ? T(0) : cpj[j - 1]);
    const T v = (T(x[vidx(g, k, j, i)]) - lj * dprev) / den;
    x[vidx(g, k, j, i)] = (double)v;
    dprev = v;
  }
  T xn = T(0);
  for (int j = nc - 1; j >= 0; --j) {
    const T v = T(x[vidx(g, k, j, i)]) - cpj[j] * xn;
    x[vidx(g, k, j, i)] = (double)v;
    xn = v;
  }
}

// ---------------------------------------------------------------------------
// smoothing and stage update in one kernel
// ---------------------------------------------------------------------------
// A CTA takes 32 columns of one component of one case: the rows of R with a halo of M columns
// (the Green's function's reach, 35 at e = 0.6) into shared memory, the smoothing along i from
// there (four outputs of a row per thread, each value read once per four terms as a 16-byte
// vector), the Thomas solves along j (a thread per column, rows in shared memory) and the
// stage update U = U0 - a (dt / vol) R of euler.py:344 -- or, without STAGE, the smoothed R.
//
// What bounded the three kernels this replaces: the Green's function's pow calls in every
// block, two shared-memory reads per term, and along j a global load and a division in
// every step of the recurrence.  The tables (irs_table) are now made once per plan, and
// the division by the step's constant pivot is one multiplication by its reciprocal and a
// correction (quotient.cuh), the quotient to the bit.
// Measured (B200, per stage): FP32, 32 cases of 256 x 64, 120 -> 31 us; FP64, 3 cases of
// 128 x 48, 31 -> 13 us.  Left: the Thomas recurrence's length, one warp of a CTA.
constexpr int kIrsCols = 32;

// entries of a shape's table: M, g_0 .. g_{ni/2}, then per row the pivot, its reciprocal and c'
__host__ __device__ inline int irs_gm_entries(int ni) { return ni / 2 + 2; }

// reach of the Green's function on a long ring: terms below 1e-18 of the diagonal are dropped.  Formed
// on the host alone: it sizes the shared memory, and a device logarithm that rounds the other way
// at an integer would lay out more than that
static int irs_reach(double e) {
  const double lam = ((1.0 + 2.0 * e) - std::sqrt(1.0 + 4.0 * e)) / (2.0 * e);
  const double M = std::ceil(std::log(1e-18) / std::log(lam));
  return M > 0.0 ? (int)std::min(M, 1e9) : 0;   // 0 too where lam has cancelled away
}
size_t irs_table_entries(int ni, int nc) { return (size_t)irs_gm_entries(ni) + 3 * (size_t)nc; }

// tables of every case's shape (cases of one shape share a table and write the same values)
template <typename T>
__global__ void __launch_bounds__(64) k_irs_table(Batch b, double* __restrict__ tab, double e_, int reach) {
  const CaseDev cs = b.cases[blockIdx.x];
  if (cs.irs_off < 0) return;
  const int ni = cs.g.ni, nc = cs.g.nc;
  double* t = tab + cs.irs_off;
  const double e = e_;
  const double lam = ((1.0 + 2.0 * e) - sqrt(1.0 + 4.0 * e)) / (2.0 * e);
  const double G0 = 1.0 / (e * (1.0 / lam - lam));
  const int M = min(reach, ni / 2);
  const double ln = pow(lam, (double)ni);
  for (int m = threadIdx.x; m <= M; m += blockDim.x)
    t[1 + m] = (double)T(G0 * (pow(lam, (double)m) + pow(lam, (double)(ni - m))) / (1.0 - ln));
  if (threadIdx.x == 0) {
    t[0] = M;
    double* piv = t + irs_gm_entries(ni);
    const T ee = T(e_);
    T cp = T(0);
    for (int j = 0; j < nc; ++j) {
      const T dj = (j == 0 || j == nc - 1) ? T(1) + ee : T(1) + T(2) * ee;
      const T lj = (j == 0) ? T(0) : -ee;
      const T uj = (j == nc - 1) ? T(0) : -ee;
      const T den = dj - lj * cp;
      cp = uj / den;
      piv[j] = (double)den;
      piv[nc + j] = (double)(T(1) / den);
      piv[2 * nc + j] = (double)cp;
    }
  }
}

__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&v)[4]) {
  const double2 t = reinterpret_cast<const double2*>(p)[0], u = reinterpret_cast<const double2*>(p)[1];
  v[0] = t.x; v[1] = t.y; v[2] = u.x; v[3] = u.y;
}

struct IrsShape {
  int halo, width;      // columns of a row in shared memory: halo + 32 + halo, or the whole ring
  bool full;
};
// full: the reach covers the ring, every column is summed
__host__ __device__ inline IrsShape irs_shape(int M, int ni) {
  IrsShape s;
  s.full = 2 * M + 1 >= ni;
  s.halo = s.full ? 0 : (M + 3) & ~3;
  s.width = s.full ? (ni + 3) & ~3 : kIrsCols + 2 * s.halo;
  return s;
}
// shared memory of a CTA for shapes up to these: the rows, the smoothed columns, the tables
template <typename T>
static size_t irs_smem(int width, int nc, int reach) {
  return sizeof(T) * ((size_t)nc * (width + kIrsCols + 1) + 3 * (size_t)nc + ((reach + 8) & ~3));
}

template <typename T, bool STAGE>
__global__ void __launch_bounds__(256) k_irs(Batch b, const double* __restrict__ R, const double* __restrict__ U0,
                                             const double* __restrict__ dt, double* __restrict__ out,
                                             const double* __restrict__ tab, double e_, double a) {
  grid_wait();
  const CaseDev cs = b.cases[blockIdx.z];
  const GridDev& g = cs.g;
  const int ni = g.ni, nc = g.nc, c0 = blockIdx.x * kIrsCols, comp = blockIdx.y;
  if (c0 >= ni || cs.irs_off < 0) return;
  const double* t = tab + cs.irs_off;
  const int M = (int)t[0];
  const IrsShape sh = irs_shape(M, ni);
  extern __shared__ __align__(16) unsigned char irs_sm[];
  T* raw = reinterpret_cast<T*>(irs_sm);             // [nc][width]
  T* gm = raw + (size_t)nc * sh.width;               // g_0 .., and room to read past M in vectors
  T* piv = gm + ((M + 8) & ~3);                      // pivots, reciprocals, c' [nc] each
  T* sm = piv + 3 * nc;                              // smoothed columns [nc][33]
  const size_t base = 4 * (size_t)cs.cell_off + vidx(g, comp, 0, 0);
  // rows to warps, columns to lanes; four rows' values on the way at a time
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kWarps = 8, kRowsAtOnce = 4;
  for (int x = lane; x < sh.width; x += 32) {
    int i = sh.full ? x : c0 - sh.halo + x;
    i += i < 0 ? ni : 0;
    i -= i >= ni ? ni : 0;     // the last CTA's columns past the ring wrap
    i = min(i, ni - 1);        // and what lies past its halo is not used
    const double* src = R + base + i;
    for (int j0 = warp; j0 < nc; j0 += kWarps * kRowsAtOnce) {
      double v[kRowsAtOnce];
#pragma unroll
      for (int u = 0; u < kRowsAtOnce; ++u) {
        const int j = j0 + u * kWarps;
        v[u] = j < nc ? src[(size_t)j * ni] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kRowsAtOnce; ++u) {
        const int j = j0 + u * kWarps;
        if (j < nc) raw[j * sh.width + x] = T(v[u]);
      }
    }
  }
  for (int m = threadIdx.x; m < ((M + 8) & ~3); m += blockDim.x) gm[m] = m <= M ? T(t[1 + m]) : T(0);
  for (int q = threadIdx.x; q < 3 * nc; q += blockDim.x) piv[q] = T(t[irs_gm_entries(ni) + q]);
  __syncthreads();
  if (sh.full) {
    for (int q = threadIdx.x; q < nc * kIrsCols; q += blockDim.x) {
      const int j = q / kIrsCols, c = q % kIrsCols, i = c0 + c;
      if (i >= ni) continue;
      const T* r = raw + (size_t)j * sh.width;
      T s = gm[0] * r[i];
      for (int d = 1; d < ni; ++d) {
        const int m = d <= ni / 2 ? d : ni - d;
        int p = i - d;
        if (p < 0) p += ni;
        s += gm[m] * r[p];
      }
      sm[j * (kIrsCols + 1) + c] = s;
    }
  } else {
    for (int q = threadIdx.x; q < nc * (kIrsCols / 4); q += blockDim.x) {
      const int j = q / (kIrsCols / 4), c = q % (kIrsCols / 4) * 4;
      const T* r = raw + (size_t)j * sh.width + sh.halo + c;
      // terms m = 4 h + 1 .. 4 h + 4 of the four outputs c .. c + 3: the columns from 4 h + 4
      // before to 4 h + 7 after are two vectors on either side, one of them new
      T s[4], L[4], P[4], Ln[4], Pn[4];
      ld4(r, L);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        P[v] = L[v];
        s[v] = gm[0] * L[v];
      }
      for (int h = 0; 4 * h < M; ++h) {
        ld4(r - 4 * (h + 1), Ln);
        ld4(r + 4 * (h + 1), Pn);
#pragma unroll
        for (int k = 1; k <= 4; ++k) {
          if (4 * h + k <= M) {
            const T w = gm[4 * h + k];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const T lo = v - k >= 0 ? L[(v - k) & 3] : Ln[(4 + v - k) & 3];
              const T hi = v + k < 4 ? P[(v + k) & 3] : Pn[(v + k) & 3];
              s[v] += w * (lo + hi);
            }
          }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          L[v] = Ln[v];
          P[v] = Pn[v];
        }
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) sm[j * (kIrsCols + 1) + c + v] = s[v];
    }
  }
  __syncthreads();
  // Thomas solves by one warp; the others fetch what the stage update needs meanwhile, into the
  // raw rows, which are done with (two values a cell: rings of fewer columns fetch it after)
  const bool ahead = STAGE && sh.width >= 2 * kIrsCols;
  const int n = min(kIrsCols, ni - c0);
  const Metric<T> m{g};
  T* fs = raw;
  T* us = raw + nc * kIrsCols;
  auto factor = [&](int j, int i) { return T(a) * (T(dt[cs.cell_off + (size_t)j * ni + i]) / m.vol(j, i)); };
  if (warp == 0) {
    T* col = sm + lane;
    constexpr int st = kIrsCols + 1;
    const T e = T(e_);
    T prev = T(0), x = col[0];
    for (int j = 0; j < nc; ++j) {
      const T xn = j + 1 < nc ? col[(j + 1) * st] : T(0);
      const T v = quotient(j == 0 ? x : fma(e, prev, x), piv[j], piv[nc + j]);
      col[j * st] = v;
      prev = v;
      x = xn;
    }
    T xn = T(0), y = col[(nc - 1) * st];
    for (int j = nc - 1; j >= 0; --j) {
      const T yn = j > 0 ? col[(j - 1) * st] : T(0);
      const T v = y - piv[2 * nc + j] * xn;
      col[j * st] = v;
      xn = v;
      y = yn;
    }
  } else if (ahead && lane < n) {
#pragma unroll 4
    for (int j = warp - 1; j < nc; j += kWarps - 1) {
      fs[j * kIrsCols + lane] = factor(j, c0 + lane);
      us[j * kIrsCols + lane] = T(U0[base + (size_t)j * ni + c0 + lane]);
    }
  }
  __syncthreads();
  if (lane >= n) return;
#pragma unroll 4
  for (int j = warp; j < nc; j += kWarps) {
    const T v = sm[j * (kIrsCols + 1) + lane];
    const size_t o = base + (size_t)j * ni + c0 + lane;
    if constexpr (STAGE) {
      const T f = ahead ? fs[j * kIrsCols + lane] : factor(j, c0 + lane);
      const T u = ahead ? us[j * kIrsCols + lane] : T(U0[o]);
      out[o] = (double)(u - f * v);
    } else {
      out[o] = (double)v;
    }
  }
}

// U = U0 - a (dt / vol) R   (euler.py:344), in the compute type T (with FP32
// the state is rounded to FP32 at every stage, as the reference's float32 run keeps it);
// rest: of the cases that k_irs does not take
template <typename T>
__global__ void __launch_bounds__(256) k_rk_stage(Batch b, const double* __restrict__ U0,
                                                  const double* __restrict__ R, const double* __restrict__ dt,
                                                  double* __restrict__ U, double a, bool rest) {
  grid_wait();
  const Tile t = b.tiles[blockIdx.x];
  const CaseDev cs = b.cases[t.cs];
  if (rest && cs.irs_off >= 0) return;
  const GridDev& g = cs.g;
  const Metric<T> m{g};
  const size_t base = 4 * cs.cell_off;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int j = t.j0 + c / t.ti, i = t.i0 + c % t.ti;
    const size_t cell = (size_t)j * g.ni + i;
    const T f = T(a) * (T(dt[cs.cell_off + cell]) / m.vol(j, i));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const size_t q = base + vidx(g, k, j, i);
      U[q] = (double)(T(U0[q]) - f * T(R[q]));
    }
  }
}

// per-tile sum of ((U_rho - U0_rho) / dt)^2
__global__ void __launch_bounds__(256) k_rk_res(Batch b, const double* __restrict__ U0,
                                                const double* __restrict__ U, const double* __restrict__ dt,
                                                double* __restrict__ tpart) {
  grid_wait();
  const Tile t = b.tiles[blockIdx.x];
  const CaseDev cs = b.cases[t.cs];
  const GridDev& g = cs.g;
  const size_t base = 4 * cs.cell_off;
  double s = 0.0;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int j = t.j0 + c / t.ti, i = t.i0 + c % t.ti;
    const size_t q = base + vidx(g, 0, j, i);
    const double r = (U[q] - U0[q]) / dt[cs.cell_off + (size_t)j * g.ni + i];
    s += r * r;
  }
  __shared__ double sc[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) sc[w] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) tot += sc[q];
    tpart[(size_t)blockIdx.x * kTilePartStride + 3] = tot;
  }
}

// res = sqrt(mean(...)) per case; circ = 1/2 Cl M from the forces   (euler.py:345, :401-403); a
// block per case, the tiles' sums fetched together and added in order
__global__ void __launch_bounds__(128) k_rk_finish(Batch b, const double* tpart, const double* coef, double* res,
                                                   double* circ) {
  grid_wait();
  __shared__ double part[128];
  const int cs = blockIdx.x;
  const CaseDev c = b.cases[cs];
  double s = 0.0;
  if (res != nullptr) {
    for (int q0 = 0; q0 < c.ntiles; q0 += 128) {
      if (q0 + (int)threadIdx.x < c.ntiles)
        part[threadIdx.x] = tpart[(size_t)(c.tile0 + q0 + threadIdx.x) * kTilePartStride + 3];
      __syncthreads();
      if (threadIdx.x == 0)
        for (int q = 0; q < min(128, c.ntiles - q0); ++q) s += part[q];
      __syncthreads();
    }
  }
  if (threadIdx.x != 0) return;
  const double N = (double)c.g.ni * (double)c.g.nc;
  if (res != nullptr) res[cs] = sqrt(s / N);
  const double mach = sqrt(c.winf[1] * c.winf[1] + c.winf[2] * c.winf[2]);
  circ[cs] = 0.5 * coef[3 * cs] * mach;
}

// ---------------------------------------------------------------------------
// FAS multigrid transfers (aero2d/euler.py:349-381) between a fine batch and
// the coarse batch of the same cases on grids of every other node (ni/2 x nc/2
// cells).  Every sum and product is rounded separately, in the reference's
// order, as the NumPy/JAX expressions evaluate them.
// ---------------------------------------------------------------------------
// R += P over the cells of every case (the forcing term of a coarse level)
__global__ void __launch_bounds__(256) k_add_forcing(Batch b, double* __restrict__ R, const double* __restrict__ P) {
  grid_wait();
  const Tile t = b.tiles[blockIdx.x];
  const CaseDev cs = b.cases[t.cs];
  const size_t base = 4 * cs.cell_off;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int j = t.j0 + c / t.ti, i = t.i0 + c % t.ti;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const size_t q = base + vidx(cs.g, k, j, i);
      R[q] = __dadd_rn(R[q], P[q]);
    }
  }
}

// sum4(a) = a(2i, 2j) + a(2i+1, 2j) + a(2i, 2j+1) + a(2i+1, 2j+1), left to right
__device__ __forceinline__ double sum4(double a00, double a10, double a01, double a11) {
  return __dadd_rn(__dadd_rn(__dadd_rn(a00, a10), a01), a11);
}

// one thread per coarse cell (tiles of the coarse batch): Uc = Uc0 = sum4(U vol) / sum4(vol);
// with R != nullptr also Pc = sum4(R (+ P)) - Rc, where Rc is read from Pc (the coarse
// residual at Uc0) and P (nullable) is the fine level's own forcing
__global__ void __launch_bounds__(256) k_fas_restrict(Batch fb, Batch cb, const double* __restrict__ Uf,
                                                     double* __restrict__ Uc, double* __restrict__ Uc0) {
  grid_wait();
  const Tile t = cb.tiles[blockIdx.x];
  const CaseDev cc = cb.cases[t.cs];
  const CaseDev cf = fb.cases[t.cs];
  const GridDev& gf = cf.g;
  const size_t bf = 4 * cf.cell_off, bc = 4 * cc.cell_off;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int jc = t.j0 + c / t.ti, ic = t.i0 + c % t.ti;
    const int i0 = 2 * ic, j0 = 2 * jc;
    const double v00 = gf.vol[(size_t)j0 * gf.ni + i0], v10 = gf.vol[(size_t)j0 * gf.ni + i0 + 1];
    const double v01 = gf.vol[(size_t)(j0 + 1) * gf.ni + i0], v11 = gf.vol[(size_t)(j0 + 1) * gf.ni + i0 + 1];
    const double vs = sum4(v00, v10, v01, v11);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double* u = Uf + bf;
      const double a = sum4(__dmul_rn(u[vidx(gf, k, j0, i0)], v00), __dmul_rn(u[vidx(gf, k, j0, i0 + 1)], v10),
                            __dmul_rn(u[vidx(gf, k, j0 + 1, i0)], v01),
                            __dmul_rn(u[vidx(gf, k, j0 + 1, i0 + 1)], v11));
      const size_t q = bc + vidx(cc.g, k, jc, ic);
      const double r = __ddiv_rn(a, vs);
      Uc[q] = r;
      Uc0[q] = r;
    }
  }
}

// Pc := sum4(Rf) - Pc (Pc holds the coarse residual at Uc0 on entry); Rf already includes
// the fine level's forcing
__global__ void __launch_bounds__(256) k_fas_forcing(Batch fb, Batch cb, const double* __restrict__ Rf,
                                                    double* __restrict__ Pc) {
  grid_wait();
  const Tile t = cb.tiles[blockIdx.x];
  const CaseDev cc = cb.cases[t.cs];
  const CaseDev cf = fb.cases[t.cs];
  const GridDev& gf = cf.g;
  const double* r = Rf + 4 * cf.cell_off;
  const size_t bc = 4 * cc.cell_off;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int jc = t.j0 + c / t.ti, ic = t.i0 + c % t.ti;
    const int i0 = 2 * ic, j0 = 2 * jc;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double a = sum4(r[vidx(gf, k, j0, i0)], r[vidx(gf, k, j0, i0 + 1)], r[vidx(gf, k, j0 + 1, i0)],
                            r[vidx(gf, k, j0 + 1, i0 + 1)]);
      const size_t q = bc + vidx(cc.g, k, jc, ic);
      Pc[q] = __dsub_rn(a, Pc[q]);
    }
  }
}

// Uf += prolong(Uc - Uc0): in i 3/4 d(ic) + 1/4 d(ic -+ 1) (periodic), then in j
// 3/4 a(jc) + 1/4 a(jc -+ 1) held at the ends (aero2d/euler.py:354-366); one thread
// per fine cell
__global__ void __launch_bounds__(256) k_fas_prolong(Batch fb, Batch cb, double* __restrict__ Uf,
                                                    const double* __restrict__ Uc,
                                                    const double* __restrict__ Uc0) {
  grid_wait();
  const Tile t = fb.tiles[blockIdx.x];
  const CaseDev cf = fb.cases[t.cs];
  const CaseDev cc = cb.cases[t.cs];
  const GridDev& gc = cc.g;
  const size_t bf = 4 * cf.cell_off, bc = 4 * cc.cell_off;
  for (int c = threadIdx.x; c < t.ti * t.tj; c += blockDim.x) {
    const int j = t.j0 + c / t.ti, i = t.i0 + c % t.ti;
    const int ic = i >> 1, jc = j >> 1;
    const int icn = (i & 1) ? (ic + 1 == gc.ni ? 0 : ic + 1) : (ic == 0 ? gc.ni - 1 : ic - 1);
    const int jcn = (j & 1) ? (jc + 1 == gc.nc ? jc : jc + 1) : (jc == 0 ? 0 : jc - 1);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      auto d = [&](int jj, int ii) {
        const size_t q = bc + vidx(gc, k, jj, ii);
        return __dsub_rn(Uc[q], Uc0[q]);
      };
      const double a0 = __dadd_rn(__dmul_rn(0.75, d(jc, ic)), __dmul_rn(0.25, d(jc, icn)));
      const double a1 = __dadd_rn(__dmul_rn(0.75, d(jcn, ic)), __dmul_rn(0.25, d(jcn, icn)));
      const double v = __dadd_rn(__dmul_rn(0.75, a0), __dmul_rn(0.25, a1));
      const size_t q = bf + vidx(cf.g, k, j, i);
      Uf[q] = __dadd_rn(Uf[q], v);
    }
  }
}

void launch_local_dt(const Batch& b, const double* U, double* U0, double* dt, double cfl, bool fp32, cudaStream_t s) {
  if (b.ntiles == 0) return;
  if (fp32) launch(k_local_dt<float>, b.ntiles, 256, 0, s, b, U, U0, dt, cfl);
  else launch(k_local_dt<double>, b.ntiles, 256, 0, s, b, U, U0, dt, cfl);
}
void launch_local_dt_prim(const GridDev& g, const double* W, double* dt, double cfl, cudaStream_t s) {
  const size_t N = (size_t)g.ni * g.nc;
  const int blocks = (int)std::min<size_t>((N + 255) / 256, 148 * 8);
  if (N) k_local_dt_prim<<<blocks, 256, 0, s>>>(g, W, dt, cfl);
}
void launch_irs(const Batch& b, double* R, double* tmp, double e, int max_ni, int max_nc, bool fp32,
                cudaStream_t s) {
  if (e <= 0.0 || b.ncases == 0) return;
  dim3 gi(4 * max_nc, b.ncases);
  const size_t sm = (size_t)(max_ni + max_ni / 2 + 2) * sizeof(double);
  dim3 gj((4 * max_ni + 127) / 128, b.ncases);
  if (fp32) {
    launch(k_irs_i<float>, gi, 256, sm, s, b, R, tmp, e, irs_reach(e));
    launch(k_irs_j<float>, gj, 128, (size_t)max_nc * sizeof(double), s, b, tmp, e);
  } else {
    launch(k_irs_i<double>, gi, 256, sm, s, b, R, tmp, e, irs_reach(e));
    launch(k_irs_j<double>, gj, 128, (size_t)max_nc * sizeof(double), s, b, tmp, e);
  }
}
void launch_irs_table(const Batch& b, double* tab, double e, bool fp32, cudaStream_t s) {
  if (b.ncases == 0) return;
  if (fp32) k_irs_table<float><<<b.ncases, 64, 0, s>>>(b, tab, e, irs_reach(e));
  else k_irs_table<double><<<b.ncases, 64, 0, s>>>(b, tab, e, irs_reach(e));
}
template <typename T, bool STAGE>
static void irs_launch(const Batch& b, const IrsArgs& p, size_t smem, cudaStream_t s) {
  launch(k_irs<T, STAGE>, dim3((p.max_ni + kIrsCols - 1) / kIrsCols, 4, b.ncases), 256, smem, s, b, p.R, p.U0, p.dt, p.out,
                                                                                            p.tab, p.e, p.a);
}
void launch_irs_fused(const Batch& b, const IrsArgs& p, bool fp32, cudaStream_t s) {
  if (b.ncases == 0) return;
  const size_t smem = p.smem;
  if (p.U0 != nullptr) {
    if (fp32) irs_launch<float, true>(b, p, smem, s);
    else irs_launch<double, true>(b, p, smem, s);
  } else {
    if (fp32) irs_launch<float, false>(b, p, smem, s);
    else irs_launch<double, false>(b, p, smem, s);
  }
}
size_t irs_smem_bytes(int ni, int nc, double e, bool fp32) {
  const int M = std::min(irs_reach(e), ni / 2);
  const IrsShape sh = irs_shape(M, ni);
  return fp32 ? irs_smem<float>(sh.width, nc, M) : irs_smem<double>(sh.width, nc, M);
}
cudaError_t irs_init() {
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* f) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kIrsMaxSmem);
  };
  set(reinterpret_cast<const void*>(&k_irs<float, true>));
  set(reinterpret_cast<const void*>(&k_irs<float, false>));
  set(reinterpret_cast<const void*>(&k_irs<double, true>));
  set(reinterpret_cast<const void*>(&k_irs<double, false>));
  return e;
}
void launch_rk_stage(const Batch& b, const double* U0, const double* R, const double* dt, double* U, double a,
                     bool rest, bool fp32, cudaStream_t s) {
  if (b.ntiles == 0) return;
  if (fp32) launch(k_rk_stage<float>, b.ntiles, 256, 0, s, b, U0, R, dt, U, a, rest);
  else launch(k_rk_stage<double>, b.ntiles, 256, 0, s, b, U0, R, dt, U, a, rest);
}
void launch_rk_res(const Batch& b, const double* U0, const double* U, const double* dt, double* tpart,
                   cudaStream_t s) {
  if (b.ntiles) launch(k_rk_res, b.ntiles, 256, 0, s, b, U0, U, dt, tpart);
}
void launch_rk_finish(const Batch& b, const double* tpart, const double* coef, double* res, double* circ,
                      cudaStream_t s) {
  if (b.ncases) launch(k_rk_finish, b.ncases, 128, 0, s, b, tpart, coef, res, circ);
}

void launch_add_forcing(const Batch& b, double* R, const double* P, cudaStream_t s) {
  if (b.ntiles) launch(k_add_forcing, b.ntiles, 256, 0, s, b, R, P);
}
void launch_fas_restrict(const Batch& fine, const Batch& coarse, const double* Uf, double* Uc, double* Uc0,
                         cudaStream_t s) {
  if (coarse.ntiles) launch(k_fas_restrict, coarse.ntiles, 256, 0, s, fine, coarse, Uf, Uc, Uc0);
}
void launch_fas_forcing(const Batch& fine, const Batch& coarse, const double* Rf, double* Pc, cudaStream_t s) {
  if (coarse.ntiles) launch(k_fas_forcing, coarse.ntiles, 256, 0, s, fine, coarse, Rf, Pc);
}
void launch_fas_prolong(const Batch& fine, const Batch& coarse, double* Uf, const double* Uc, const double* Uc0,
                        cudaStream_t s) {
  if (fine.ntiles) launch(k_fas_prolong, fine.ntiles, 256, 0, s, fine, coarse, Uf, Uc, Uc0);
}

}  // namespace a2d
