// O-grid generation on the device (a2d_grid_spacing, a2d_grid_build in
// include/aero2d_b200.h): the hyperbolic marching of aero2d/grid.py:50-81 for
// many airfoils at once, one CTA per grid, one thread per circumferential node.
//
// The layers are sequential in j and every smoothing pass couples each node to
// its two neighbours along the layer, so a CTA keeps the current layer and the
// smoothed field in shared memory (ping-pong buffers: one barrier per pass) and
// writes each finished layer once.  Every operation is the reference's, in its
// order and with IEEE rounding at each step (no contraction into FMAs), so
// layers 0 .. nj-2 are bitwise the host generator's; the spacings come from the
// host (a2d_grid_spacing) for the same reason.  The outer layer is snapped to a
// circle with CUDA's atan2/cos/sin, whose last bits may differ from the host
// library's; its mean radius is summed in NumPy's pairwise order, so only
// those functions' rounding separates it from the host grid.
#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "aero2d_b200.h"

namespace a2d {

int fail(int code, const std::string& msg);

namespace {

constexpr int kMaxRing = 1024;

// a + eps * (a[i-1] + a[i+1] - 2 a), the reference's expression order (aero2d/grid.py:44-47)
__device__ __forceinline__ double smooth1(double am, double a, double ap, double eps) {
  const double t = __dsub_rn(__dadd_rn(am, ap), __dmul_rn(2.0, a));
  return __dadd_rn(a, __dmul_rn(eps, t));
}

// A warp smooths a window of the ring in registers, two points a lane: kHalo passes need no more
// than shuffles when the window reaches kHalo points past those it owns on either side.
constexpr int kHalo = 10;
constexpr int kWindow = 64;
constexpr int kOwned = kWindow - 2 * kHalo;
constexpr int kMaxWarps = (kMaxRing + kOwned - 1) / kOwned;

struct Ring {
  double* buf;        // [2][2][ni]: what the warps exchange, two copies in turn
  int ni, copy;
  int at[2];          // the lane's ring points
  bool own[2];

  // the owned points of every warp into the ring's next copy, this warp's window out of it; one
  // barrier: a copy is written again only after the next exchange's
  __device__ __forceinline__ void exchange(double (&vx)[2], double (&vy)[2]) {
    double* c = buf + copy * 2 * ni;
    copy ^= 1;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (own[q]) {
        c[at[q]] = vx[q];
        c[ni + at[q]] = vy[q];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      vx[q] = c[at[q]];
      vy[q] = c[ni + at[q]];
    }
  }

  // `passes` smoothing passes of a 2-vector field whose window is valid; then its owned points are
  __device__ __forceinline__ void smooth(double (&vx)[2], double (&vy)[2], double eps, int passes) {
    while (true) {
      const int n = passes < kHalo ? passes : kHalo;
      for (int p = 0; p < n; ++p) {
        const double lx = __shfl_up_sync(0xffffffffu, vx[1], 1), ly = __shfl_up_sync(0xffffffffu, vy[1], 1);
        const double rx = __shfl_down_sync(0xffffffffu, vx[0], 1), ry = __shfl_down_sync(0xffffffffu, vy[0], 1);
        const double x0 = smooth1(lx, vx[0], vx[1], eps), y0 = smooth1(ly, vy[0], vy[1], eps);
        vx[1] = smooth1(vx[0], vx[1], rx, eps);
        vy[1] = smooth1(vy[0], vy[1], ry, eps);
        vx[0] = x0;
        vy[0] = y0;
      }
      passes -= n;
      if (passes == 0) return;
      exchange(vx, vy);
    }
  }
};

// NumPy's pairwise summation of a contiguous float64 array (blocks of 8
// partial sums up to 128 entries, halves at multiples of 8 above): the order of
// np.mean in aero2d/grid.py:75, so the mean radius is the host's to the bit
__device__ double pairwise_sum(const double* a, int n) {
  // explicit stack instead of recursion: (offset, length, state) frames
  struct Frame {
    int lo, n, stage;
    double left;
  };
  Frame st[16];
  int top = 0;
  st[0] = {0, n, 0, 0.0};
  double ret = 0.0;
  while (true) {
    Frame& f = st[top];
    if (f.n <= 128 && f.stage == 0) {
      double res;
      if (f.n < 8) {
        res = -0.0;
        for (int q = 0; q < f.n; ++q) res = __dadd_rn(res, a[f.lo + q]);
      } else {
        double r[8];
        for (int k = 0; k < 8; ++k) r[k] = a[f.lo + k];
        int q = 8;
        for (; q < f.n - (f.n % 8); q += 8)
          for (int k = 0; k < 8; ++k) r[k] = __dadd_rn(r[k], a[f.lo + q + k]);
        res = __dadd_rn(__dadd_rn(__dadd_rn(r[0], r[1]), __dadd_rn(r[2], r[3])),
                        __dadd_rn(__dadd_rn(r[4], r[5]), __dadd_rn(r[6], r[7])));
        for (; q < f.n; ++q) res = __dadd_rn(res, a[f.lo + q]);
      }
      ret = res;
      if (top == 0) return ret;
      --top;
      continue;
    }
    int n2 = f.n / 2;
    n2 -= n2 % 8;
    if (f.stage == 0) {           // left half first
      f.stage = 1;
      st[++top] = {f.lo, n2, 0, 0.0};
    } else if (f.stage == 1) {    // left done: keep it, then the right half
      f.left = ret;
      f.stage = 2;
      st[++top] = {f.lo + n2, f.n - n2, 0, 0.0};
    } else {                      // both done
      ret = __dadd_rn(f.left, ret);
      if (top == 0) return ret;
      --top;
    }
  }
}

// one grid per CTA; ring [n][ni][2], spacing [n][nj-1], x/y [n][ni][nj], min_area [n].
// A chain of some 26 smoothing passes a layer, each four dependent FP64 operations and a shuffle,
// is what bounds it: 16 grids of 256x65 points take 214 us.  A point per thread with a barrier per
// pass took 246, the cell areas read back at the end included; in windows (Ring) a layer
// has three barriers, and the areas are taken from the layers in shared memory.
__global__ void __launch_bounds__(32 * kMaxWarps) k_ogrid(int ni, int nj, const double* __restrict__ ring,
                                                          const double* __restrict__ spacing, int normal_smoothing,
                                                          double* __restrict__ x, double* __restrict__ y,
                                                          double* __restrict__ min_area) {
  extern __shared__ double sm[];
  double* layer[2] = {sm, sm + 2 * ni};   // [2][ni]: the last layer and the one being formed
  Ring r;
  r.buf = sm + 4 * ni;
  r.ni = ni;
  r.copy = 0;
  const int g = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int im[2], ip[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int w = 2 * lane + q - kHalo;   // from the warp's first owned point
    const int i = ((warp * kOwned + w) % ni + ni) % ni;
    r.at[q] = i;
    r.own[q] = w >= 0 && w < kOwned && warp * kOwned + w < ni;
    im[q] = i == 0 ? ni - 1 : i - 1;
    ip[q] = i == ni - 1 ? 0 : i + 1;
  }
  const double* rg = ring + 2 * (size_t)ni * g;
  const double* sp = spacing + (size_t)(nj - 1) * g;
  double* xg = x + (size_t)ni * nj * g;
  double* yg = y + (size_t)ni * nj * g;
  // the points of layer j that this warp owns
  auto put = [&](int j, const double (&cx)[2], const double (&cy)[2]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!r.own[q]) continue;
      const int i = r.at[q];
      layer[1][i] = cx[q];
      layer[1][ni + i] = cy[q];
      xg[(size_t)i * nj + j] = cx[q];
      yg[(size_t)i * nj + j] = cy[q];
    }
  };

  double cx[2], cy[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    cx[q] = rg[2 * r.at[q]];
    cy[q] = rg[2 * r.at[q] + 1];
  }
  put(0, cx, cy);
  __syncthreads();
  double amin = INFINITY;
  for (int j = 1; j < nj; ++j) {
    double* t = layer[0];
    layer[0] = layer[1];
    layer[1] = t;
    const double* cur = layer[0];
    // unit tangent from the neighbours, normal = (t_y, -t_x) (aero2d/grid.py:58-60)
    double nx[2], ny[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double tx = __dsub_rn(cur[ip[q]], cur[im[q]]);
      const double ty = __dsub_rn(cur[ni + ip[q]], cur[ni + im[q]]);
      const double len = __dsqrt_rn(__dadd_rn(__dmul_rn(tx, tx), __dmul_rn(ty, ty)));
      nx[q] = __ddiv_rn(ty, len);
      ny[q] = -__ddiv_rn(tx, len);
    }
    r.smooth(nx, ny, 0.25, j > 1 ? normal_smoothing : 2);
    // step out by this layer's spacing, then smooth along the layer (:62-64)
    const double frac = __ddiv_rn((double)j, (double)(nj - 1));
    const double s = sp[j - 1];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double len = __dsqrt_rn(__dadd_rn(__dmul_rn(nx[q], nx[q]), __dmul_rn(ny[q], ny[q])));
      cx[q] = __dadd_rn(cur[r.at[q]], __dmul_rn(s, __ddiv_rn(nx[q], len)));
      cy[q] = __dadd_rn(cur[ni + r.at[q]], __dmul_rn(s, __ddiv_rn(ny[q], len)));
    }
    const double eps = __dadd_rn(0.1, __dmul_rn(0.3, frac));
    const int passes = 2 + (int)__dmul_rn(8.0, frac);
    r.exchange(cx, cy);
    r.smooth(cx, cy, eps, passes);
    if (j == nj - 1) {
      // outer layer on a circle of the mean radius about (0.5, 0) (:65-69)
      double* rad = r.buf + r.copy * 2 * ni;
      double rx[2], ry[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        rx[q] = __dsub_rn(cx[q], 0.5);
        ry[q] = __dsub_rn(cy[q], 0.0);
        if (r.own[q]) rad[r.at[q]] = __dsqrt_rn(__dadd_rn(__dmul_rn(rx[q], rx[q]), __dmul_rn(ry[q], ry[q])));
      }
      __syncthreads();
      __shared__ double rmean;
      if (threadIdx.x == 0) rmean = __ddiv_rn(pairwise_sum(rad, ni), (double)ni);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double ang = atan2(ry[q], rx[q]);
        cx[q] = __dadd_rn(0.5, __dmul_rn(rmean, cos(ang)));
        cy[q] = __dadd_rn(0.0, __dmul_rn(rmean, sin(ang)));
      }
    }
    put(j, cx, cy);
    __syncthreads();
    // smallest cell area from the two diagonals (aero2d/grid.py:24-31, :78-80)
    const double* now = layer[1];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!r.own[q]) continue;
      const int i = r.at[q], n = ip[q];
      const double d1x = now[n] - cur[i], d1y = now[ni + n] - cur[ni + i];
      const double d2x = now[i] - cur[n], d2y = now[ni + i] - cur[ni + n];
      amin = fmin(amin, -0.5 * (d1x * d2y - d1y * d2x));
    }
  }
  for (int o = 16; o > 0; o >>= 1) amin = fmin(amin, __shfl_xor_sync(0xffffffffu, amin, o));
  __shared__ double wmin[kMaxWarps];
  if (lane == 0) wmin[warp] = amin;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = INFINITY;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmin(m, wmin[w]);
    min_area[g] = m;
  }
}

}  // namespace
}  // namespace a2d

using namespace a2d;

extern "C" {

int a2d_grid_spacing(int nj, double ds0, double radius, double* spacing) {
  if (nj < 2 || !(ds0 > 0.0) || !(radius > ds0) || spacing == nullptr)
    return fail(A2D_ERR_ARG, "grid_spacing: bad arguments");
  // growth ratio by 200 bisection steps on [1 + 1e-9, 2] (aero2d/grid.py:34-41)
  const int n = nj - 1;
  double lo = 1.0 + 1e-9, hi = 2.0;
  for (int it = 0; it < 200; ++it) {
    const double r = 0.5 * (lo + hi);
    const double total = ds0 * (std::pow(r, (double)n) - 1.0) / (r - 1.0);
    if (total < radius) lo = r;
    else hi = r;
  }
  const double r = 0.5 * (lo + hi);
  for (int k = 0; k < n; ++k) spacing[k] = ds0 * std::pow(r, (double)k);
  return A2D_OK;
}

int a2d_grid_build(int n, int ni, int nj, const double* ring, const double* spacing, int normal_smoothing,
                   double* x, double* y, double* min_area, void* stream) {
  if (n < 0 || ni < 3 || ni > kMaxRing || nj < 2 || normal_smoothing < 0 || normal_smoothing > 1000)
    return fail(A2D_ERR_ARG, "grid_build: bad sizes (3 <= ni <= 1024, nj >= 2)");
  if (n == 0) return A2D_OK;
  if (ring == nullptr || spacing == nullptr || x == nullptr || y == nullptr || min_area == nullptr)
    return fail(A2D_ERR_ARG, "grid_build: null pointer");
  const int threads = 32 * ((ni + kOwned - 1) / kOwned);
  const size_t smem = sizeof(double) * 8 * (size_t)ni;
  cudaFuncSetAttribute(k_ogrid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(double) * 8 * kMaxRing));
  k_ogrid<<<n, threads, smem, static_cast<cudaStream_t>(stream)>>>(ni, nj, ring, spacing, normal_smoothing, x,
                                                                   y, min_area);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(A2D_ERR_CUDA, std::string("grid_build: ") + cudaGetErrorString(e));
  return A2D_OK;
}

}  // extern "C"
