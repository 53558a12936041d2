// Block-tridiagonal line preconditioner of the Newton-Krylov solver.
//
//  k_face_jac   4x4 Jacobian blocks dF/dU_left, dF/dU_right of the first-order
//               HLLC flux on every i- and j-face, plus the wall and far-field
//               closures (aero2d/implicit.py:32-64), by forward-mode dual
//               numbers; one thread per cell, 32 lines x 8 rows per CTA.
//  k_factor     assembles D = sum of face blocks + vol/dtau I and runs the
//               block-Thomas forward elimination along each wall-normal line
//               in FP64: den_j = D_j - A_j c_{j-1}, inv_j = den_j^-1,
//               c_j = inv_j C_j (aero2d/implicit.py:81-128), and stores inv_j,
//               c_j, G_j = -inv_j A_j and the premultiplied i-couplings
//               P_j = inv_j JIL(i), Q_j = inv_j JIR(i+1) of the sweeps.  A
//               lane per line, a CTA per line group.
// The sweeps themselves are in lines.cu and sweep*.cu.
//
// The blocks are stored lane-blocked ([group][row][entry][lane]): the blocks
// of one line group at one row j are one contiguous run, which the sweep
// kernel streams with bulk copies.
#include <cuda_fp16.h>

#include "batch.cuh"
#include "kernels.cuh"
#include "launch.cuh"
#include "physics.cuh"
#include "tma.cuh"

namespace a2d {

template <typename T>
__device__ __forceinline__ State4<T> load_state(const double* U, const GridDev& g, int j, int i) {
  State4<T> r;
#pragma unroll
  for (int k = 0; k < 4; ++k) r.c[k] = T(U[vidx(g, k, j, i)]);
  return r;
}

// Jacobian d f / d u (f: conserved state -> flux, 4x4 [out][in]) by one dual pass
template <typename T, class F>
__device__ __forceinline__ void jac4(const State4<T>& u, F f, T J[16]) {
  using D = Dual<T, 4>;
  State4<D> ud;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ud.c[k].v = u.c[k];
#pragma unroll
    for (int q = 0; q < 4; ++q) ud.c[k].d[q] = (q == k) ? T(1) : T(0);
  }
  const State4<D> r = f(ud);
#pragma unroll
  for (int o = 0; o < 4; ++o)
#pragma unroll
    for (int q = 0; q < 4; ++q) J[o * 4 + q] = r.c[o].d[q];
}

template <typename T>
__device__ __forceinline__ State4<Dual<T, 4>> const_dual(const State4<T>& u) {
  State4<Dual<T, 4>> r;
#pragma unroll
  for (int k = 0; k < 4; ++k) r.c[k] = make_const<T, 4>(u.c[k]);
  return r;
}

// dF/dUL, dF/dUR of the first-order flux hllc(prim(UL), prim(UR), S)
template <typename T>
__device__ __forceinline__ void face_jac(const State4<T>& UL, const State4<T>& UR, T sx, T sy, T AL[16],
                                         T AR[16]) {
  using D = Dual<T, 4>;
  const State4<D> WRc = cons_to_prim<D, T>(const_dual(UR));
  jac4<T>(UL, [&](const State4<D>& u) { return hllc<D, T>(cons_to_prim<D, T>(u), WRc, sx, sy); }, AL);
  const State4<D> WLc = cons_to_prim<D, T>(const_dual(UL));
  jac4<T>(UR, [&](const State4<D>& u) { return hllc<D, T>(WLc, cons_to_prim<D, T>(u), sx, sy); }, AR);
}

template <typename TS, typename T>
__device__ __forceinline__ void store_block(TS* base, long long row0, int rows, int g, int j, int lane,
                                            const T A[16]) {
#pragma unroll
  for (int e = 0; e < 16; ++e) base[lbidx(row0, rows, g, j, e, lane)] = TS(A[e]);
}

// Bound by the dual flux's instructions and their latency.  FP32 left alone takes 174 registers, one
// CTA per SM; held to 128 (28 bytes of spills) it runs two: 64 cases of 256x64 350 -> 238 us.  Three
// are slower (263), and FP64 fills its 255.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) k_face_jac(Batch b, JacArgs a) {
  grid_wait();
  const Tile t = b.tiles[blockIdx.x];
  if (!case_live(b, t.cs, a.need)) return;
  const CaseDev cs = b.cases[t.cs];
  const GridDev& g = cs.g;
  Metric<T> m{g};
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  if (lane >= t.ti || row >= t.tj) return;
  const int ni = g.ni, nc = g.nc;
  const int i = t.i0 + lane, j = t.j0 + row, grp = t.i0 / kLanes;
  const double* U = a.U + 4 * cs.cell_off;
  T* JIL = static_cast<T*>(a.JIL);
  T* JIR = static_cast<T*>(a.JIR);
  T* JJL = static_cast<T*>(a.JJL);
  T* JJR = static_cast<T*>(a.JJR);
  const State4<T> Uc = load_state<T>(U, g, j, i);
  T AL[16], AR[16];
  {  // i-face between cells i-1 and i
    const int im = i == 0 ? ni - 1 : i - 1;
    face_jac<T>(load_state<T>(U, g, j, im), Uc, m.si(0, j, i), m.si(1, j, i), AL, AR);
    store_block(JIL, cs.rows_nc, nc, grp, j, lane, AL);
    store_block(JIR, cs.rows_nc, nc, grp, j, lane, AR);
  }
  if (j == 0) {  // wall face: mirrored ghost on its low side
    const T sx = m.sj(0, 0, i), sy = m.sj(1, 0, i);
    using D = Dual<T, 4>;
    jac4<T>(Uc,
            [&](const State4<D>& u) {
              const State4<D> w = cons_to_prim<D, T>(u);
              return hllc<D, T>(wall_mirror<D, T>(w, sx, sy), w, sx, sy);
            },
            AR);
#pragma unroll
    for (int e = 0; e < 16; ++e) AL[e] = T(0);
    store_block(JJL, cs.rows_nc1, nc + 1, grp, 0, lane, AL);
    store_block(JJR, cs.rows_nc1, nc + 1, grp, 0, lane, AR);
  } else {  // interior j-face between cells j-1 and j
    face_jac<T>(load_state<T>(U, g, j - 1, i), Uc, m.sj(0, j, i), m.sj(1, j, i), AL, AR);
    store_block(JJL, cs.rows_nc1, nc + 1, grp, j, lane, AL);
    store_block(JJR, cs.rows_nc1, nc + 1, grp, j, lane, AR);
  }
  if (j == nc - 1) {  // far-field face, circulation held fixed (implicit.py:54-59)
    const T sx = m.sj(0, nc, i), sy = m.sj(1, nc, i);
    const T rinf = T(cs.winf[0]), uinf = T(cs.winf[1]), vinf = T(cs.winf[2]), pinf = T(cs.winf[3]);
    const T circ = a.vortex ? T(a.circ[t.cs]) : T(0);
    const T xf = m.xf(i), yf = m.yf(i);
    using D = Dual<T, 4>;
    const D cd = make_const<T, 4>(circ);
    jac4<T>(Uc,
            [&](const State4<D>& u) {
              const State4<D> w = cons_to_prim<D, T>(u);
              const State4<D> wb = farfield_ghost<D, T>(w, sx, sy, rinf, uinf, vinf, pinf, xf, yf, cd);
              return hllc<D, T>(w, wb, sx, sy);
            },
            AL);
#pragma unroll
    for (int e = 0; e < 16; ++e) AR[e] = T(0);
    store_block(JJL, cs.rows_nc1, nc + 1, grp, nc, lane, AL);
    store_block(JJR, cs.rows_nc1, nc + 1, grp, nc, lane, AR);
  }
}

// ---------------------------------------------------------------------------
// 4x4 FP64 inverse by Gauss-Jordan elimination with partial pivoting
// ---------------------------------------------------------------------------
__device__ __forceinline__ void inv4(const double A[16], double X[16]) {
  double a[4][8];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      a[r][c] = A[r * 4 + c];
      a[r][c + 4] = (r == c) ? 1.0 : 0.0;
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    int p = c;
    double best = fabs(a[c][c]);
#pragma unroll
    for (int r = c + 1; r < 4; ++r) {
      const double v = fabs(a[r][c]);
      if (v > best) {
        best = v;
        p = r;
      }
    }
#pragma unroll
    for (int r = c + 1; r < 4; ++r) {
      if (p == r) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const double tmp = a[c][k];
          a[c][k] = a[r][k];
          a[r][k] = tmp;
        }
      }
    }
    const double ip = 1.0 / a[c][c];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[c][k] *= ip;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r != c) {
        const double f = a[r][c];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[r][k] -= f * a[c][k];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) X[r * 4 + c] = a[r][c + 4];
}

template <typename TJ>
__device__ __forceinline__ void load_block(const TJ* base, long long row0, int rows, int g, int j, int lane,
                                           double A[16]) {
#pragma unroll
  for (int e = 0; e < 16; ++e) A[e] = (double)base[lbidx(row0, rows, g, j, e, lane)];
}

// the four entries of a block row, contiguous per lane (fbidx), with one or two vector stores
__device__ __forceinline__ void store4(double* out, const double v[4]) {
  reinterpret_cast<double2*>(out)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(out)[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void store4(float* out, const double v[4]) {
  *reinterpret_cast<float4*>(out) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
}
__device__ __forceinline__ void store4(__half* out, const double v[4]) {
  __half2 h[2] = {__halves2half2(from_f64<__half>(v[0]), from_f64<__half>(v[1])),
                  __halves2half2(from_f64<__half>(v[2]), from_f64<__half>(v[3]))};
  *reinterpret_cast<uint2*>(out) = *reinterpret_cast<uint2*>(h);
}

// block m of the interleaved P, Q, G rows = sgn A B (4x4, FP64), stored in TF (fbidx3)
template <typename TF>
__device__ __forceinline__ void mul4_store(const double A[16], const double B[16], double sgn, TF* out, long long row0,
                                           int rows, int g, int j, int m, int lane, unsigned& nsat) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    double v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double s = A[r * 4 + 0] * B[0 * 4 + c];
#pragma unroll
      for (int k = 1; k < 4; ++k) s += A[r * 4 + k] * B[k * 4 + c];
      v[c] = sgn * s;
      nsat += out_of_range<TF>(v[c]);
    }
    store4(&out[fbidx3(row0, rows, g, j, m, r, 0, lane)], v);
  }
}

// C = sgn A B (4x4)
__device__ __forceinline__ void mul4(const double A[16], const double B[16], double C[16], double sgn) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double s = A[r * 4 + 0] * B[0 * 4 + c];
#pragma unroll
      for (int q = 1; q < 4; ++q) s += A[r * 4 + q] * B[q * 4 + c];
      C[r * 4 + c] = sgn * s;
    }
}
// D += sgn A B
__device__ __forceinline__ void mul4_add(const double A[16], const double B[16], double D[16], double sgn) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double s = A[r * 4 + 0] * B[0 * 4 + c];
#pragma unroll
      for (int q = 1; q < 4; ++q) s += A[r * 4 + q] * B[q * 4 + c];
      D[r * 4 + c] = D[r * 4 + c] + sgn * s;
    }
}

// A row of a line group between its helper and its chain warp, a lane per line
struct FactorRow {
  double D[16][kLanes];     // the diagonal block, then its elimination's inverse
  double L[16][kLanes];     // JJL(j)
  double R[16][kLanes];     // JJR(j+1)
};
template <int H>
struct FactorSmem {
  FactorRow row[2][H];
  double cfar[16][kLanes];    // c'_{k+1} of each line
  double seen[2][kLanes];
  uint64_t assembled[2][H], inverted[2][H], far;
};
constexpr int kFactorWide = 148;   // line groups up to which each gets an SM
constexpr int factor_threads(int H) { return 32 * 2 * (1 + H); }

__device__ __forceinline__ void get_block(const double (*base)[kLanes], int lane, double A[16]) {
#pragma unroll
  for (int e = 0; e < 16; ++e) A[e] = base[e][lane];
}

// a warp hands over what it wrote to shared memory
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// One CTA per 32-line group.  The line system is L_j x_{j-1} + D_j x_j + U_j x_{j+1} = r_j with
// L_j = -JJL(j), U_j = JJR(j+1) (aero2d/implicit.py:81-128), eliminated from both ends:
//   wall side, rows 0 .. k-1:  den_j = D_j - L_j c_{j-1}, c_j = den_j^-1 U_j, G_j = -den_j^-1 L_j;
//     later d_j = inv_j r_j + G_j d_{j-1}, x_j = d_j - c_j x_{j+1}
//   far side, rows nc-1 .. k+1:  den'_j = D_j - U_j c'_{j+1}, c'_j = den'_j^-1 L_j,
//     G'_j = -den'_j^-1 U_j; later d'_j = inv'_j r_j + G'_j d'_{j+1}, x_j = d'_j - c'_j x_{j-1}
//   twist row k:  den_k = D_k - L_k c_{k-1} - U_k c'_{k+1}; x_k = inv_k r_k + G_k d_{k-1} + H_k d'_{k+1},
//     G_k = -inv_k L_k, H_k = -inv_k U_k (kept in the C slot, row k having no back substitution)
// Only den, its inverse and c depend on the row before.  So each half has one chain warp that
// does nothing else, and H helper warps that take the rows in turn: a helper assembles its
// row for the chain, waits for the inverse, forms and stores the row's factors from it, and goes
// on to its next row.
// Bound by the chain, some 2500 cycles a row of dependent FP64 operations, for small batches and
// by the helpers' memory and conversions for large ones.  One warp per half doing all of a row in
// turn took 4 to 7 us a row, most of it waiting for its loads: one mixed 128x48 case 107 -> 40 us,
// one FP64 192x48 case 165 -> 45, 64 mixed 256x64 cases 236 -> 202 and FP64 452 -> 281.
template <typename TJ, typename TF, int H>
__global__ void __launch_bounds__(factor_threads(H), 512 / factor_threads(H)) k_factor(Batch b, FactorArgs a) {
  grid_wait();
  extern __shared__ double factor_smem[];
  FactorSmem<H>& sm = *reinterpret_cast<FactorSmem<H>*>(factor_smem);
  const Group grp = b.groups[blockIdx.x];
  if (!case_live(b, grp.cs, a.need)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = warp & 1;               // 0: from the wall, 1: from the far field
  const int helper = (warp >> 1) - 1;      // -1: the chain
  const bool own = lane < grp.n;           // lanes past the group's last line only meet the barriers
  const CaseDev cs = b.cases[grp.cs];
  const GridDev& g = cs.g;
  const int ni = g.ni, nc = g.nc;
  const int k = nc / 2;
  // rows of the half in the order of its elimination; the wall's last one is the twist row
  const int rows = half == 0 ? k + 1 : nc - 1 - k;
  if (threadIdx.x < 4 * H + 1) mbar_init(&sm.assembled[0][0] + threadIdx.x, 1);
  __syncthreads();
  bool ok = true;

  if (helper < 0) {
    double c[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) c[e] = 0.0;
    uint32_t phase = 0;
    for (int q = 0, h = 0; q < rows; ++q) {
      FactorRow& row = sm.row[half][h];
      const bool twist = half == 0 && q == k;
      ok = mbar_wait_warp(&sm.assembled[half][h], phase);
      if (ok && twist) ok = mbar_wait_warp(&sm.far, 0);
      if (!ok) break;
      if (own) {
        double D[16], B[16], inv[16];
        get_block(row.D, lane, D);
        get_block(half == 0 ? row.L : row.R, lane, B);
        if (half == 0) mul4_add(B, c, D, 1.0);
        else mul4_add(B, c, D, -1.0);
        if (twist) {
          get_block(row.R, lane, B);
          get_block(sm.cfar, lane, c);
          mul4_add(B, c, D, -1.0);
        }
        inv4(D, inv);
#pragma unroll
        for (int e = 0; e < 16; ++e) row.D[e][lane] = inv[e];
        get_block(half == 0 ? row.R : row.L, lane, B);
        if (half == 0) mul4(inv, B, c, 1.0);
        else mul4(inv, B, c, -1.0);
        // the arrival does not wait for loads under way, a store of what all of B went into does:
        // the helper may then overwrite it
        sm.seen[half][lane] = (c[0] + c[1]) + (c[2] + c[3]);
      }
      warp_arrive(&sm.inverted[half][h], lane);
      if (++h == H) {
        h = 0;
        phase ^= 1;
      }
    }
    if (half == 1 && ok) {
#pragma unroll
      for (int e = 0; e < 16; ++e) sm.cfar[e][lane] = c[e];
      warp_arrive(&sm.far, lane);
    }
    if (!ok && lane == 0 && a.err != nullptr) atomicExch(a.err, 1u);
    return;
  }

  const int i = grp.i0 + (own ? lane : grp.n - 1);
  const int ip = (i + 1 == ni) ? 0 : i + 1;
  const int gp = ip / kLanes, lp = ip % kLanes;
  const TJ* JIL = static_cast<const TJ*>(a.JIL);
  const TJ* JIR = static_cast<const TJ*>(a.JIR);
  const TJ* JJL = static_cast<const TJ*>(a.JJL);
  const TJ* JJR = static_cast<const TJ*>(a.JJR);
  TJ* INV = static_cast<TJ*>(a.INV);
  TF* CF = static_cast<TF*>(a.CF);
  TF* PQG = static_cast<TF*>(a.PQG);
  const double* U = a.U + 4 * cs.cell_off;
  const double cfl = a.ctl[grp.cs].cfl;
  unsigned nsat = 0;      // factor entries this line stores saturated (FP16 storage)
  FactorRow& row = sm.row[half][helper];
  uint32_t phase = 0;
  for (int q = helper; q < rows; q += H, phase ^= 1) {
    const int j = half == 0 ? q : nc - 1 - q;
    if (own) {
      // D_j: the diagonal block of row j (face blocks + vol/dtau I); writes diag
      double D[16], T1[16];
      load_block(JIL, cs.rows_nc, nc, gp, j, lp, D);
      load_block(JIR, cs.rows_nc, nc, grp.g, j, lane, T1);
#pragma unroll
      for (int e = 0; e < 16; ++e) D[e] = D[e] - T1[e];
      if (j < nc - 1) {
        load_block(JJL, cs.rows_nc1, nc + 1, grp.g, j + 1, lane, T1);
#pragma unroll
        for (int e = 0; e < 16; ++e) D[e] = D[e] + T1[e];
      }
      load_block(JJR, cs.rows_nc1, nc + 1, grp.g, j, lane, T1);
#pragma unroll
      for (int e = 0; e < 16; ++e) D[e] = D[e] - T1[e];
      if (j == nc - 1) {
        load_block(JJL, cs.rows_nc1, nc + 1, grp.g, nc, lane, T1);
#pragma unroll
        for (int e = 0; e < 16; ++e) D[e] = D[e] + T1[e];
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        row.L[e][lane] = (double)JJL[lbidx(cs.rows_nc1, nc + 1, grp.g, j, e, lane)];
        row.R[e][lane] = (double)JJR[lbidx(cs.rows_nc1, nc + 1, grp.g, j + 1, e, lane)];
      }
      // local pseudo-time step (aero2d/euler.py:289-296, aero2d/implicit.py:173-177)
      const State4<double> W = cons_to_prim<double, double>(load_state<double>(U, g, j, i));
      const double c = sqrt(kGamma * W.c[3] / W.c[0]);
      const size_t N = (size_t)ni * nc;
      const double* Si = g.Si;
      const double* Sj = g.Sj;
      const double s0 = 0.5 * (Si[(size_t)j * ni + i] + Si[(size_t)j * ni + ip]);
      const double s1 = 0.5 * (Si[N + (size_t)j * ni + i] + Si[N + (size_t)j * ni + ip]);
      const size_t NJ = (size_t)(nc + 1) * ni;
      const double t0 = 0.5 * (Sj[(size_t)(j + 1) * ni + i] + Sj[(size_t)j * ni + i]);
      const double t1 = 0.5 * (Sj[NJ + (size_t)(j + 1) * ni + i] + Sj[NJ + (size_t)j * ni + i]);
      const double li = fabs(W.c[1] * s0 + W.c[2] * s1) + c * sqrt(s0 * s0 + s1 * s1);
      const double lj = fabs(W.c[1] * t0 + W.c[2] * t1) + c * sqrt(t0 * t0 + t1 * t1);
      const double vol = g.vol[(size_t)j * ni + i];
      const double dt = a.cfl_base * vol / (li + lj);
      const double dtl = dt / a.cfl_base * cfl;
      const double dinv = 1.0 / dtl;
      const double dg = vol * dinv;
      a.diag[cs.cell_off + (size_t)j * ni + i] = dg;
      D[0] += dg;
      D[5] += dg;
      D[10] += dg;
      D[15] += dg;
#pragma unroll
      for (int e = 0; e < 16; ++e) row.D[e][lane] = D[e];
    }
    warp_arrive(&sm.assembled[half][helper], lane);
    ok = mbar_wait_warp(&sm.inverted[half][helper], phase);
    if (!ok) break;
    if (own) {
      // row j's sweep factors: inv, C (the back-substitution coupling), G (the
      // forward-recurrence coupling) and the i-couplings P = inv JIL(i), Q = inv JIR(i+1)
      double inv[16], B[16];
      get_block(row.D, lane, inv);
      get_block(half == 0 ? row.R : row.L, lane, B);
      const double sgn = half == 0 && q < k ? 1.0 : -1.0;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        double v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          double s = inv[r * 4 + 0] * B[0 * 4 + c];
#pragma unroll
          for (int m = 1; m < 4; ++m) s += inv[r * 4 + m] * B[m * 4 + c];
          v[c] = sgn * s;
          nsat += out_of_range<TF>(v[c]);
        }
        const size_t x = fbidx(cs.rows_nc, nc, grp.g, j, r, 0, lane);
        store4(&CF[x], v);
        store4(&INV[x], &inv[r * 4]);
      }
      get_block(half == 0 ? row.L : row.R, lane, B);
      mul4_store(inv, B, half == 0 ? 1.0 : -1.0, PQG, cs.rows_nc, nc, grp.g, j, 2, lane, nsat);
      load_block(JIL, cs.rows_nc, nc, grp.g, j, lane, B);
      mul4_store(inv, B, 1.0, PQG, cs.rows_nc, nc, grp.g, j, 0, lane, nsat);
      load_block(JIR, cs.rows_nc, nc, gp, j, lp, B);
      mul4_store(inv, B, 1.0, PQG, cs.rows_nc, nc, grp.g, j, 1, lane, nsat);
    }
  }
  if (nsat != 0 && a.sat != nullptr) atomicAdd(a.sat, (unsigned long long)nsat);
  if (!ok && lane == 0 && a.err != nullptr) atomicExch(a.err, 1u);
}

template <typename TJ, typename TF, int H>
cudaError_t factor_smem_limit() {
  return cudaFuncSetAttribute(k_factor<TJ, TF, H>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(FactorSmem<H>));
}
cudaError_t factor_init() {
  cudaError_t e = factor_smem_limit<double, double, 7>();
  if (e == cudaSuccess) e = factor_smem_limit<double, double, 3>();
  if (e == cudaSuccess) e = factor_smem_limit<float, __half, 7>();
  if (e == cudaSuccess) e = factor_smem_limit<float, __half, 3>();
  return e;
}

template <typename T>
void launch_face_jac(const Batch& b, const JacArgs& a, cudaStream_t s) {
  if (b.ntiles == 0) return;
  launch(k_face_jac<T>, b.ntiles, 256, 0, s, b, a);
}
template <typename TJ, typename TF>
void launch_factor(const Batch& b, const FactorArgs& a, cudaStream_t s) {
  if (b.ngroups == 0) return;
  auto go = [&](auto f, int threads, size_t smem) { launch(f, b.ngroups, threads, smem, s, b, a); };
  // Seven helpers per half take an SM to themselves; three leave room for a second CTA.  One
  // wave of groups is faster with seven (one 128x48 case 40 us against 50, 16 of 256x64 in FP64
  // 74 and 101), more with three (64 of 256x64 in mixed precision 202 against 292, FP64 281 and 294).
  if (b.ngroups <= kFactorWide) go(k_factor<TJ, TF, 7>, factor_threads(7), sizeof(FactorSmem<7>));
  else go(k_factor<TJ, TF, 3>, factor_threads(3), sizeof(FactorSmem<3>));
}

template void launch_face_jac<double>(const Batch&, const JacArgs&, cudaStream_t);
template void launch_face_jac<float>(const Batch&, const JacArgs&, cudaStream_t);
template void launch_factor<double, double>(const Batch&, const FactorArgs&, cudaStream_t);
template void launch_factor<float, __half>(const Batch&, const FactorArgs&, cudaStream_t);

}  // namespace a2d
