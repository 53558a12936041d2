// Arnoldi orthogonalisation of the GMRES cycle: classical Gram-Schmidt run
// twice (the scheme of aero2d/krylov.py:45-50), in three passes over the
// Krylov basis per Arnoldi step.
//
//   pass 1  k_gs_dots     raw projections V_raw[q] . w and w . w, per chunk
//   pass 2  k_gs_project  h1_q = s_q (V_raw[q] . w) reduced over the case's chunks, then
//                         w' = w - sum_q V_raw[q] s_q h1_q and V_raw[q] . w' from one
//                         read of the basis
//   pass 3  k_gs_sub      h2_q the same way, w'' = w - sum_q V_raw[q] s_q (h1_q + h2_q),
//                         written as the next raw basis vector, with its squared norm
//   close   k_gs_close    per case: h_{k+1,k} = ||w''||, the breakdown test against
//                         eps ||w|| (jax.scipy.sparse.linalg.gmres semantics), the
//                         Hessenberg column and s_{k+1} = 1 / ||w''||
//
// Basis vectors are stored unnormalised with their scale s_q, so no normalisation
// pass is needed; w' is never stored, since pass 3 subtracts h1 + h2 from the
// original w (equal to the two successive subtractions in exact arithmetic).
//
// The order of every sum.  A chunk of 4096 entries is 8 rows of 32 lanes with 16 entries
// each.  A lane's products are added one after the other (chain index i = 0 .. 15), the 32
// lanes of a row by a fixed tree, a chunk's 8 rows in order, a case's chunks in
// warp_chunk_sum's order.  None of it depends on how rows and vectors are dealt to warps
// and CTAs, nor on the other cases of a batch.  A subtraction's sum runs over the vectors in
// order, 32 at a time (the slices it was once cut into).  Products are fused into the sums
// and differences are not, spelled out, so that no unrolling changes a bit: h2 is made of w's
// rounding, and a marginal case's path follows it.
//
// Small mixed-precision cases run a whole step, passes and close, in one launch: k_gs_case.
//
// What bounds the passes: the basis from HBM (each pass reads it once from there), with few
// chunks the latency of one CTA.  A warp owns a row (in split launches a quarter of one)
// and runs it through alone: the row's entries of w stay in registers from the subtraction to
// the projections, the vectors go by through a ring of asynchronous copies of 1 KB each that every
// lane reads back itself, so nothing waits on a barrier, and pass 2's second reading of
// the row comes from L2.  (Partial sums of all vectors in a thread's registers, as
// the passes had before, held an SM to 16 warps.)  Where a batch has too few chunks for the
// GPU, the rows of a chunk are the CTAs of a cluster, whose first CTA adds their sums.
// Measured (B200, BF16, average over an Arnoldi process of 30 vectors, 64 cases of 256 x 64,
// passes 1 / 2 / 3): 46 / 64 / 40 -> 33 / 51 / 36 us, of 24 / 24 / 26 us at the HBM peak; one
// case of 128 x 48, 27 vectors: 19 / 25 / 17 -> 6 / 12 / 12 us; FP64, 16 cases of 256 x 64, 27
// vectors: 53 / 96 / 66 -> 39 / 75 / 45 us.  A ring of 8 KB or 2 KB, and four CTAs per SM, were slower.
#include <cfloat>
#include <cuda_bf16.h>
#include <type_traits>

#include "batch.cuh"
#include "cluster.cuh"
#include "gs.cuh"
#include "launch.cuh"

namespace a2d {

constexpr int kRows = kGsRows;           // rows of a chunk
// warps of a CTA: a row of the chunk each, or (split) four on the chunk's row blockIdx.y
constexpr int warps_of(bool split) { return split ? 4 : kRows; }
constexpr int kBatchQ = 8;               // vectors projected on at a time
constexpr int kChain = 16;               // entries of a lane in a row
static_assert(kRows * 32 * kChain == kChunk, "a chunk is 8 rows of 32 lanes with 16 entries");
constexpr int kSlice = 32;               // vectors of one subtraction sum

// fixed-order sum of a per-chunk partial over a case's chunks (every lane gets it)
__device__ __forceinline__ double warp_chunk_sum(const double* p, size_t stride, int nchunks) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int c = lane; c < nchunks; c += 32) s += p[(size_t)c * stride];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// this pass's coefficients s_q h_q of every vector into shared memory: one warp per
// coefficient reduces the case's partials of the pass before; the case's first CTA stores
// the result
template <bool SPLIT, typename TB>
__device__ __forceinline__ void coefficients(const GsArgs<TB>& a, const CaseDev& cs, int cs_id, int ncases, bool first,
                                             double* coef, bool both) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nred = a.nq + (a.fold_wn0 != nullptr ? 1 : 0);
  const double* part = a.fold_part + (size_t)cs.chunk0 * a.pstride;
#pragma unroll 4
  for (int q = warp; q < nred; q += warps_of(SPLIT)) {
    const double sum = warp_chunk_sum(part + q, a.pstride, cs.nchunks);
    if (lane == 0) {
      if (q < a.nq) {
        const double sc = a.scale[(size_t)q * ncases + cs_id];
        // rounded as H's column is (k_gs_close adds the stored h1 and h2)
        const double h = __dmul_rn(sum, sc);
        if (first) a.fold_h[(size_t)cs_id * kHStride + q] = h;
        const double hh = both ? __dadd_rn(a.h1[(size_t)cs_id * kHStride + q], h) : h;
        coef[q] = hh * sc;
      } else if (first) {
        a.fold_wn0[cs_id] = sqrt(sum);
      }
    }
  }
  __syncthreads();
}

// ---- a lane's entries of a row, four at a time (quad m: chain indices 4 m .. 4 m + 3) ----
// BF16: four consecutive entries, m a quarter of the chunk apart; FP64: entries a
// sixteenth of the chunk apart, so that a warp's loads are runs of 256 bytes either way
template <typename TB> struct Quad;
template <> struct Quad<__nv_bfloat16> {
  uint2 raw;
  static __device__ __forceinline__ int at(int r, int m, int lane) { return m * (kChunk / 4) + (32 * r + lane) * 4; }
  __device__ __forceinline__ void load(const __nv_bfloat16* p, int r, int m, int lane, int len) {
    const int e = at(r, m, lane);
    raw = e < len ? __ldg(reinterpret_cast<const uint2*>(p + e)) : make_uint2(0u, 0u);
  }
  __device__ __forceinline__ void read(const uint64_t* s, int m) { raw = *reinterpret_cast<const uint2*>(s + m * 32); }
  __device__ __forceinline__ double operator[](int t) const {
    const uint32_t w = t < 2 ? raw.x : raw.y;
    return (double)__uint_as_float(t & 1 ? w & 0xffff0000u : w << 16);
  }
};
template <> struct Quad<double> {
  double v[4];
  static __device__ __forceinline__ int at(int r, int i, int lane) { return i * (kChunk / 16) + 32 * r + lane; }
  __device__ __forceinline__ void load(const double* p, int r, int m, int lane, int len) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int e = at(r, 4 * m + t, lane);
      v[t] = e < len ? __ldg(p + e) : 0.0;
    }
  }
  __device__ __forceinline__ void read(const uint64_t* s, int m) {
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = reinterpret_cast<const double*>(s)[(4 * m + t) * 32];
  }
  __device__ __forceinline__ double operator[](int t) const { return v[t]; }
};
// the same entries of an FP64 vector; and calling f(t, entry offset) for those in the chunk
template <typename TB>
__device__ __forceinline__ void load_w(const double* w, int r, int m, int lane, int len, double (&v)[4]) {
  if constexpr (std::is_same<TB, double>::value) {
    Quad<double> q;
    q.load(w, r, m, lane, len);
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = q[t];
  } else {
    const int e = Quad<TB>::at(r, m, lane);
    const double2 z = make_double2(0.0, 0.0);
    const double2 a = e < len ? __ldg(reinterpret_cast<const double2*>(w + e)) : z;
    const double2 b = e < len ? __ldg(reinterpret_cast<const double2*>(w + e + 2)) : z;
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}
__device__ __forceinline__ void store_quad(__nv_bfloat16* p, int r, int m, int lane, int len, const double (&v)[4]) {
  const int e = Quad<__nv_bfloat16>::at(r, m, lane);
  if (e >= len) return;
  __nv_bfloat162 lo = __floats2bfloat162_rn((float)v[0], (float)v[1]);
  __nv_bfloat162 hi = __floats2bfloat162_rn((float)v[2], (float)v[3]);
  *reinterpret_cast<uint2*>(p + e) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
__device__ __forceinline__ void store_quad(double* p, int r, int m, int lane, int len, const double (&v)[4]) {
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int e = Quad<double>::at(r, 4 * m + t, lane);
    if (e < len) p[e] = v[t];
  }
}

// The sums over the 32 lanes of N values, by the tree l + (l + 16), .. + 8, 4, 2, 1: while more
// than one value is left a lane keeps half of them and hands the other half over, so N
// values take about N + 4 exchanges instead of 5 N.  The result's value index is lane_value<N>().
template <int N>
__device__ __forceinline__ double warp_tree(double (&v)[N], int o = 16) {
  const bool up = threadIdx.x & o;
  if constexpr (N == 1) {
    double s = v[0];
    for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  } else {
    constexpr int H = (N + 1) / 2;
    double k[H];
#pragma unroll
    for (int q = 0; q < H; ++q) {
      const double hi = q + H < N ? v[q + H] : 0.0;
      const double give = up ? v[q] : hi, keep = up ? hi : v[q];
      k[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
    return warp_tree<H>(k, o >> 1);
  }
}
// which of the N values this lane's sum is (-1: none), and whether it is the lane that stores it
template <int N>
__device__ __forceinline__ int lane_value(bool& owner, int o = 16) {
  if constexpr (N == 1) {
    owner = (threadIdx.x & (2 * o - 1)) == 0;
    return 0;
  } else {
    constexpr int H = (N + 1) / 2;
    const int inner = lane_value<H>(owner, o >> 1);
    const int q = inner + (threadIdx.x & o ? H : 0);
    return inner < 0 || q >= N ? -1 : q;
  }
}

// ---- a row of the basis, vector after vector, through a warp's ring in shared memory ----
// Every lane copies (cp.async, 8 bytes) and reads back its own entries only, so the ring needs no
// barrier, and the bytes in flight do not depend on registers: 24 warps of an SM keep
// kRingDepth KB each (BF16) on the way.
template <typename TB> struct RingDepth { static constexpr int value = 4; };
template <> struct RingDepth<double> { static constexpr int value = 2; };
template <typename TB>
struct Ring {
  static constexpr int D = RingDepth<TB>::value;
  static constexpr int kWords = 32 * kChain * sizeof(TB) / 8;   // 8-byte words of a row
  static constexpr int kLaneWords = kWords / 32;
  static constexpr uint32_t kBytes = D * kWords * 8;            // per warp
  const TB* V;          // the chunk's first entry of vector 0
  size_t vstride;
  const uint64_t* mem;  // this lane's words: [slot][word][lane]
  int nq, r, lane, len;
  __device__ __forceinline__ void issue(int q, int slot) {
    if (q < nq) {
      const TB* src = V + (size_t)q * vstride;
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(mem + slot * kWords));
#pragma unroll
      for (int k = 0; k < kLaneWords; ++k) {
        const int e = Quad<TB>::at(r, k, lane);
        const uint32_t n = e < len ? 8u : 0u;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + k * 256), "l"(src + (e < len ? e : 0)),
                     "r"(n)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void start() {
#pragma unroll
    for (int q = 0; q < D; ++q) issue(q, q);
  }
  // quads of vector q (in slot), which is then refilled with vector q + D
  __device__ __forceinline__ void take(int q, int slot, Quad<TB> (&v)[4]) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
    const uint64_t* s = mem + slot * kWords;
#pragma unroll
    for (int m = 0; m < 4; ++m) v[m].read(s, m);
    issue(q + D, slot);
  }
};

// ---- a chunk's sums from its rows', added in order ----
// split: the rows are CTAs of one cluster (rank = row), whose sums the first one reads from
// their shared memory
__device__ __forceinline__ double peer_value(const double* p, int rank) {
  uint32_t addr;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(addr)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
// out[q] = the chunk's sum q < n; rowsum: the CTA's rows (split: its one row)
template <bool SPLIT>
__device__ __forceinline__ void store_chunk(double* out, const double (*rowsum)[kMaxRestart + 1], int n) {
  if constexpr (SPLIT) {
    cluster_sync();
    if (blockIdx.y == 0 && threadIdx.x < n) {
      double v[kRows], s = 0.0;
#pragma unroll
      for (int r = 0; r < kRows; ++r) v[r] = peer_value(&rowsum[0][threadIdx.x], r);
#pragma unroll
      for (int r = 0; r < kRows; ++r) s += v[r];
      out[threadIdx.x] = s;
    }
    cluster_sync();   // the rows' shared memory stays until it is read
  } else {
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += 32 * warps_of(SPLIT)) {
      double s = 0.0;
#pragma unroll
      for (int r = 0; r < kRows; ++r) s += rowsum[r][q];
      out[q] = s;
    }
  }
}

// the projections of a row, whose entries of w are wv, on the vectors q0, q0 + step, ..;
// vec(v, q, m) gives quad m of vector q.  The sums go to rowsum[q].
template <typename TB, class F>
__device__ __forceinline__ void project_row(int nq, int q0, int step, F vec, const double (&wv)[kChain],
                                            double* rowsum) {
#pragma unroll 1
  for (int qb = q0; qb < nq; qb += kBatchQ * step) {
    double acc[kBatchQ];
#pragma unroll
    for (int j = 0; j < kBatchQ; ++j) acc[j] = 0.0;
#pragma unroll
    for (int j = 0; j < kBatchQ; ++j) {
      const int q = qb + step * j;
      if (q < nq) {
        Quad<TB> v[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) vec(v[m], q, m);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[j] = fma(v[m][t], wv[4 * m + t], acc[j]);
      }
    }
    bool owner;
    const int j = lane_value<kBatchQ>(owner);
    const double s = warp_tree<kBatchQ>(acc);
    const int q = qb + step * j;
    if (owner && q < nq) rowsum[q] = s;
  }
}

// x = w - sum_q V_q coef_q for one quad of entries, 32 vectors to a sum; vec(v, q) gives the
// quad of vector q
template <typename TB, class F>
__device__ __forceinline__ void subtract(int nq, F vec, const double* coef, double (&x)[4]) {
  constexpr int kAhead = std::is_same<TB, double>::value ? 4 : 8;   // quads loaded at a time
  for (int q0 = 0; q0 < nq; q0 += kSlice) {
    const int q1 = min(nq, q0 + kSlice);
    double sub[4] = {0.0, 0.0, 0.0, 0.0};
    auto take = [&](int q, int n, auto whole) {
      Quad<TB> v[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j)
        if (decltype(whole)::value || j < n) vec(v[j], q + j);
#pragma unroll
      for (int j = 0; j < kAhead; ++j)
        if (decltype(whole)::value || j < n) {
#pragma unroll
          for (int t = 0; t < 4; ++t) sub[t] = fma(v[j][t], coef[q + j], sub[t]);
        }
    };
    int q = q0;
#pragma unroll 1
    for (; q + kAhead <= q1; q += kAhead) take(q, kAhead, std::true_type());
    if (q < q1) take(q, q1 - q, std::false_type());
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = __dsub_rn(x[t], sub[t]);
  }
}

template <typename TB>
__device__ __forceinline__ Ring<TB> ring_of(unsigned char* sm, const TB* V, const GsArgs<TB>& a, int r, int len) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  return Ring<TB>{V, a.vstride, reinterpret_cast<const uint64_t*>(sm + warp * Ring<TB>::kBytes) + lane, a.nq, r, lane, len};
}

// the same two for a warp with the row to itself, every vector through its ring
template <typename TB>
__device__ __forceinline__ void project_ring(Ring<TB>& ring, const double (&wv)[kChain], double* rowsum) {
  constexpr int D = Ring<TB>::D;
  static_assert(kBatchQ % D == 0, "slots are known at compile time");
  ring.start();
#pragma unroll 1
  for (int qb = 0; qb < ring.nq; qb += kBatchQ) {
    double acc[kBatchQ];
#pragma unroll
    for (int j = 0; j < kBatchQ; ++j) {
      acc[j] = 0.0;
      if (qb + j < ring.nq) {
        Quad<TB> v[4];
        ring.take(qb + j, j % D, v);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[j] = fma(v[m][t], wv[4 * m + t], acc[j]);
      }
    }
    bool owner;
    const int j = lane_value<kBatchQ>(owner);
    const double s = warp_tree<kBatchQ>(acc);
    if (owner && qb + j < ring.nq) rowsum[qb + j] = s;
  }
}
template <typename TB>
__device__ __forceinline__ void subtract_ring(Ring<TB>& ring, const double* coef, double (&x)[4][4]) {
  constexpr int D = Ring<TB>::D;
  static_assert(kSlice % D == 0, "slots are known at compile time");
  for (int q0 = 0; q0 < ring.nq; q0 += kSlice) {
    const int q1 = min(ring.nq, q0 + kSlice);
    double sub[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int t = 0; t < 4; ++t) sub[m][t] = 0.0;
#pragma unroll 1
    for (int qb = q0; qb < q1; qb += D) {
#pragma unroll
      for (int j = 0; j < D; ++j) {
        if (qb + j < q1) {
          Quad<TB> v[4];
          ring.take(qb + j, j, v);
          const double c = coef[qb + j];
#pragma unroll
          for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int t = 0; t < 4; ++t) sub[m][t] = fma(v[m][t], c, sub[m][t]);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int t = 0; t < 4; ++t) x[m][t] = __dsub_rn(x[m][t], sub[m][t]);
  }
}

// pass 1 -----------------------------------------------------------------------
template <typename TB, bool SPLIT>
__global__ void __launch_bounds__(32 * warps_of(SPLIT), SPLIT ? 4 : (sizeof(TB) == 8 ? 2 : 3)) k_gs_dots(Batch b, GsArgs<TB> a) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char gs_sm[];
  __shared__ double rowsum[SPLIT ? 1 : kRows][kMaxRestart + 1];
  const Chunk ch = b.chunks[blockIdx.x];
  if (!case_live(b, ch.cs, a.need)) return;
  const size_t base = 4 * b.cases[ch.cs].cell_off + ch.begin;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, len = ch.len;
  const int r = SPLIT ? blockIdx.y : warp;
  const TB* V = a.V + base;
  double* rs = rowsum[SPLIT ? 0 : r];
  double wv[kChain];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    double t[4];
    load_w<TB>(a.w + base, r, m, lane, len, t);
#pragma unroll
    for (int u = 0; u < 4; ++u) wv[4 * m + u] = t[u];
  }
  if constexpr (SPLIT) {
    project_row<TB>(
        a.nq, warp, warps_of(true),
        [&](Quad<TB>& v, int q, int m) { v.load(V + (size_t)q * a.vstride, r, m, lane, len); }, wv, rs);
  } else {
    Ring<TB> ring = ring_of<TB>(gs_sm, V, a, r, len);
    project_ring(ring, wv, rs);
  }
  if (!SPLIT || warp == 0) {   // w . w
    double n[1] = {0.0};
#pragma unroll
    for (int i = 0; i < kChain; ++i) n[0] = fma(wv[i], wv[i], n[0]);
    const double s = warp_tree<1>(n);
    if (lane == 0) rs[a.nq] = s;
  }
  store_chunk<SPLIT>(a.part + (size_t)blockIdx.x * a.pstride, rowsum, a.nq + 1);
}

// pass 2 -----------------------------------------------------------------------
// A warp with a row of its own keeps the row's w' in registers and reads the basis again for
// the projections, from L2.  With the row split over four warps, each subtracts a quarter of the
// entries and projects on a quarter of the vectors, w' through shared memory; a BF16 row of
// the vectors (1 KB each) is copied there too and read from there both times.
template <typename TB>
__host__ __device__ inline size_t gs_tile_bytes(int nq) {
  return std::is_same<TB, double>::value ? 0 : (size_t)nq * 32 * kChain * sizeof(TB);
}

template <typename TB, bool SPLIT>
__global__ void __launch_bounds__(32 * warps_of(SPLIT), SPLIT ? 4 : (sizeof(TB) == 8 ? 2 : 3)) k_gs_project(Batch b, GsArgs<TB> a) {
  grid_wait();
  constexpr bool kTile = SPLIT && !std::is_same<TB, double>::value;
  extern __shared__ __align__(16) unsigned char gs_sm[];
  __shared__ double rowsum[SPLIT ? 1 : kRows][kMaxRestart + 1];
  __shared__ double wp[SPLIT ? kChain * 32 : 1];   // w' of the row, [chain index][lane]
  __shared__ double coef[kMaxRestart];
  const Chunk ch = b.chunks[blockIdx.x];
  if (!case_live(b, ch.cs, a.need)) return;
  const CaseDev cs = b.cases[ch.cs];
  const size_t base = 4 * cs.cell_off + ch.begin;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, len = ch.len, nq = a.nq;
  const int r = SPLIT ? blockIdx.y : warp;
  const TB* V = a.V + base;
  double* rs = rowsum[SPLIT ? 0 : r];
  auto global = [&](Quad<TB>& v, int q, int m) { v.load(V + (size_t)q * a.vstride, r, m, lane, len); };
  uint2* tile = reinterpret_cast<uint2*>(gs_sm);   // [vector][quad m][lane]
  if constexpr (kTile) {   // this thread's quad (m = warp) of every vector
    const int e = Quad<TB>::at(r, warp, lane);
    const uint32_t bytes = e < len ? 8u : 0u;
    const TB* src = V + (e < len ? e : 0);
    uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(tile + warp * 32 + lane));
#pragma unroll 4
    for (int q = 0; q < nq; ++q) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
      dst += 128 * sizeof(uint2);
      src += a.vstride;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  Ring<TB> ring = ring_of<TB>(gs_sm, V, a, r, len);
  if constexpr (!SPLIT) ring.start();
  coefficients<SPLIT>(a, cs, ch.cs, b.ncases, ch.begin == 0 && (!SPLIT || r == 0), coef, false);
  double wv[kChain];
  if constexpr (SPLIT) {
    double x[4];
    load_w<TB>(a.w + base, r, warp, lane, len, x);
    if constexpr (kTile) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      subtract<TB>(nq, [&](Quad<TB>& v, int q) { v.raw = tile[(size_t)q * 128 + warp * 32 + lane]; }, coef, x);
    } else {
      subtract<TB>(nq, [&](Quad<TB>& v, int q) { global(v, q, warp); }, coef, x);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) wp[(4 * warp + t) * 32 + lane] = x[t];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kChain; ++i) wv[i] = wp[i * 32 + lane];
  } else {
    double x[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m) load_w<TB>(a.w + base, r, m, lane, len, x[m]);
    subtract_ring(ring, coef, x);
#pragma unroll
    for (int i = 0; i < kChain; ++i) wv[i] = x[i / 4][i % 4];
    project_ring(ring, wv, rs);
  }
  if constexpr (kTile) {
    project_row<TB>(
        nq, warp, warps_of(true),
        [&](Quad<TB>& v, int q, int m) { v.raw = tile[(size_t)q * 128 + m * 32 + lane]; }, wv, rs);
  } else if constexpr (SPLIT) {
    project_row<TB>(nq, warp, warps_of(true), global, wv, rs);
  }
  store_chunk<SPLIT>(a.part + (size_t)blockIdx.x * a.pstride, rowsum, nq);
}

// pass 3 -----------------------------------------------------------------------
template <typename TB, bool SPLIT>
__global__ void __launch_bounds__(32 * warps_of(SPLIT), SPLIT ? 4 : (sizeof(TB) == 8 ? 2 : 3)) k_gs_sub(Batch b, GsArgs<TB> a) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char gs_sm[];
  __shared__ double xs[SPLIT ? kChain * 32 : 1];   // w'' of the row, [chain index][lane]
  __shared__ double rowsum[SPLIT ? 1 : kRows][kMaxRestart + 1];
  __shared__ double coef[kMaxRestart];
  constexpr int NM = SPLIT ? 1 : 4;                // quads of a lane
  const Chunk ch = b.chunks[blockIdx.x];
  if (!case_live(b, ch.cs, a.need)) return;
  const CaseDev cs = b.cases[ch.cs];
  const size_t base = 4 * cs.cell_off + ch.begin;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, len = ch.len;
  const int r = SPLIT ? blockIdx.y : warp, m0 = SPLIT ? warp : 0;
  const TB* V = a.V + base;
  Ring<TB> ring = ring_of<TB>(gs_sm, V, a, r, len);
  if constexpr (!SPLIT) ring.start();
  coefficients<SPLIT>(a, cs, ch.cs, b.ncases, ch.begin == 0 && (!SPLIT || r == 0), coef, true);
  double x[NM][4];
#pragma unroll
  for (int m = 0; m < NM; ++m) load_w<TB>(a.w + base, r, m0 + m, lane, len, x[m]);
  if constexpr (SPLIT) {
    subtract<TB>(a.nq, [&](Quad<TB>& v, int q) { v.load(V + (size_t)q * a.vstride, r, warp, lane, len); }, coef, x[0]);
  } else {
    subtract_ring(ring, coef, x);
  }
#pragma unroll
  for (int m = 0; m < NM; ++m) store_quad(a.Vout + base, r, m0 + m, lane, len, x[m]);
  double n[1] = {0.0};
  if constexpr (SPLIT) {
#pragma unroll
    for (int t = 0; t < 4; ++t) xs[(4 * warp + t) * 32 + lane] = x[0][t];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int i = 0; i < kChain; ++i) {
        const double y = xs[i * 32 + lane];
        n[0] = fma(y, y, n[0]);
      }
    }
  } else {
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
      for (int t = 0; t < 4; ++t) n[0] = fma(x[m][t], x[m][t], n[0]);
  }
  if (!SPLIT || warp == 0) {
    const double s = warp_tree<1>(n);
    if (lane == 0) rowsum[SPLIT ? 0 : r][0] = s;
  }
  store_chunk<SPLIT>(a.part_norm + blockIdx.x, rowsum, 1);
}

// the end of Arnoldi step a.k, by one warp: the Hessenberg column and the new vector's scale
__device__ __forceinline__ void close_step(const GsCloseArgs& a, int ncases, int cs_id, double hn, double wn0,
                                           const double* h1, const double* h2) {
  const int lane = threadIdx.x & 31, k = a.k;
  CaseCtl& c = a.ctl[cs_id];
  const bool use = hn > DBL_EPSILON * wn0;
  double* H = a.H + (size_t)cs_id * kMaxRestart * (kMaxRestart + 1) + (size_t)k * (kMaxRestart + 1);
  for (int q = lane; q <= k; q += 32) H[q] = h1[q] + h2[q];
  if (lane == 0) {
    H[k + 1] = use ? hn : 0.0;
    a.scale[(size_t)(k + 1) * ncases + cs_id] = use ? 1.0 / hn : 0.0;
    c.k_used = k + 1;
    if (!use) a.live[cs_id] &= ~kLiveKrylov;
  }
}

// a whole Arnoldi step of a small case --------------------------------------------
// With few rows the four launches are latency: each starts up, fetches the basis or the sums of the
// last, reduces.  Here a case is a cluster.  A row of a chunk belongs to a team of four warps,
// which copies its entries of every vector (1 KB each) into shared memory once and runs all three
// passes from there; a row's sums go to every CTA of the cluster as they are formed (st.async,
// counted on an mbarrier there), and each CTA adds them up itself, in the order of the passes
// above, so the results are theirs to the bit.  What is left is latency, and the conversions of the
// entries to FP64.  One 128x48 case, 25 vectors on average: the four launches 29.5 us, this 17;
// 16 cases of 128x32, 13 vectors: 24 and 14.  FP64 rows are too large for the shared memory.
using CaseBasis = __nv_bfloat16;
constexpr int kTeams = 5;                // rows of a CTA at most
struct CaseSmem {
  int tile, wp, msg, norm, rowsum, coef, scale, h1, h2, wn0, bar, bytes;   // offsets
  __host__ __device__ CaseSmem(int teams, int rows, int nq) {
    int o = 0;
    auto take = [&](int n) {
      const int at = o;
      o += n;
      return at;
    };
    tile = take(teams * nq * 1024);                     // [team][vector][quad m][lane]
    wp = take(teams * kChain * 32 * 8);                 // [team][chain index][lane]
    msg = take(2 * rows * (nq + 1) * 8);                // [pass][row][vector]
    norm = take(rows * 8);
    rowsum = take(teams * (kMaxRestart + 1) * 8);
    coef = take(kMaxRestart * 8);
    scale = take(kMaxRestart * 8);
    h1 = take(kMaxRestart * 8);
    h2 = take(kMaxRestart * 8);
    wn0 = take(8);
    bar = take(3 * 8);
    bytes = o;
  }
};
constexpr int kCaseMaxSmem = 227 * 1024;

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");
}
__device__ __forceinline__ void peer_store1(uint32_t addr, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
               "r"(bar)
               : "memory");
}

template <int TEAMS>
__global__ void __launch_bounds__(128 * TEAMS, TEAMS == 2 ? 3 : 1) k_gs_case(Batch b, GsArgs<CaseBasis> a, GsCloseArgs c, uint32_t* err,
                                                          int rows_max) {
  grid_wait();
  using TB = CaseBasis;
  extern __shared__ __align__(16) unsigned char gs_sm[];
  const uint32_t size = cluster_size(), rank = cluster_rank();
  const int cs_id = blockIdx.x / size;
  if (!case_live(b, cs_id, a.need)) return;   // the whole cluster leaves
  const CaseDev cs = b.cases[cs_id];
  const int nq = a.nq, stride = nq + 1, rows = cs.nchunks * kRows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int team = warp >> 2, m = warp & 3, nwarps = blockDim.x >> 5;
  const CaseSmem sm(blockDim.x >> 7, rows_max, nq);
  uint2* tile = reinterpret_cast<uint2*>(gs_sm + sm.tile) + (size_t)team * nq * 128;
  double* wp = reinterpret_cast<double*>(gs_sm + sm.wp) + team * kChain * 32;
  double* msg = reinterpret_cast<double*>(gs_sm + sm.msg);
  double* norm = reinterpret_cast<double*>(gs_sm + sm.norm);
  double* rs = reinterpret_cast<double*>(gs_sm + sm.rowsum) + team * (kMaxRestart + 1);
  double* coef = reinterpret_cast<double*>(gs_sm + sm.coef);
  double* scale = reinterpret_cast<double*>(gs_sm + sm.scale);
  double* h1 = reinterpret_cast<double*>(gs_sm + sm.h1);
  double* h2 = reinterpret_cast<double*>(gs_sm + sm.h2);
  double* wn0 = reinterpret_cast<double*>(gs_sm + sm.wn0);
  uint64_t* bar = reinterpret_cast<uint64_t*>(gs_sm + sm.bar);
  if (threadIdx.x == 0) {
    for (int q = 0; q < 3; ++q) mbar_init(bar + q, 1);
    mbar_init_fence();
    mbar_arrive_expect(bar, rows * stride * 8);
    mbar_arrive_expect(bar + 1, rows * nq * 8);
    mbar_arrive_expect(bar + 2, rank == 0 ? rows * 8 : 0);
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  const int row = team * (int)size + (int)rank;
  const bool have = row < rows;               // the same for a team
  const Chunk ch = b.chunks[cs.chunk0 + (have ? row / kRows : 0)];
  const int r = row % kRows, len = ch.len;
  const size_t base = 4 * cs.cell_off + ch.begin;
  double w0[4] = {0.0, 0.0, 0.0, 0.0};
  if (have) {
    const int e = Quad<TB>::at(r, m, lane);
    const uint32_t bytes = e < len ? 8u : 0u;
    const TB* src = a.V + base + (e < len ? e : 0);
    uint32_t dst = smem_u32(tile + m * 32 + lane);
#pragma unroll 4
    for (int q = 0; q < nq; ++q) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
      dst += 128 * sizeof(uint2);
      src += a.vstride;
    }
    load_w<TB>(a.w + base, r, m, lane, len, w0);
#pragma unroll
    for (int t = 0; t < 4; ++t) wp[(4 * m + t) * 32 + lane] = w0[t];
  }
  for (int q = threadIdx.x; q < nq; q += blockDim.x) scale[q] = a.scale[(size_t)q * b.ncases + cs_id];
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every CTA's mbarriers exist

  auto whole = [&](Quad<TB>& v, int q, int k) { v.raw = tile[(size_t)q * 128 + k * 32 + lane]; };
  auto mine = [&](Quad<TB>& v, int q) { v.raw = tile[(size_t)q * 128 + m * 32 + lane]; };
  // the row's first n sums to every CTA
  auto publish = [&](int pass, int n) {
    for (int v = threadIdx.x & 127; v < n * (int)size; v += 128) {
      const int q = v / (int)size;
      const uint32_t peer = v - q * (int)size;
      peer_store1(peer_addr(msg + ((size_t)pass * rows_max + row) * stride + q, peer), rs[q], peer_addr(bar + pass, peer));
    }
  };
  // project the row in wp on the basis and publish; pass 0 also its w . w
  auto project = [&](int pass) {
    double wv[kChain];
#pragma unroll
    for (int i = 0; i < kChain; ++i) wv[i] = wp[i * 32 + lane];
    if (pass == 0 && m == 0) {
      double n[1] = {0.0};
#pragma unroll
      for (int i = 0; i < kChain; ++i) n[0] = fma(wv[i], wv[i], n[0]);
      const double s = warp_tree<1>(n);
      if (lane == 0) rs[nq] = s;
    }
    project_row<TB>(nq, m, 4, whole, wv, rs);
    team_sync(team);
    publish(pass, pass == 0 ? nq + 1 : nq);
  };
  // a pass's sums over the case's chunks, and the coefficients of the next subtraction
  auto fold = [&](int pass) {
    bool ok = wait_cluster(bar + pass, 0);
    const int n = pass == 0 ? nq + 1 : nq;
    if (ok) {
#pragma unroll 2
      for (int q = warp; q < n; q += nwarps) {
        double s = 0.0;
        if (lane < cs.nchunks) {
          const double* v = msg + ((size_t)pass * rows_max + lane * kRows) * stride + q;
#pragma unroll
          for (int k = 0; k < kRows; ++k) s += v[k * stride];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
          if (q < nq) {
            const double sc = scale[q];
            const double h = __dmul_rn(s, sc);
            (pass == 0 ? h1 : h2)[q] = h;
            const double hh = pass == 0 ? h : __dadd_rn(h1[q], h);
            coef[q] = hh * sc;
          } else {
            *wn0 = sqrt(s);
          }
        }
      }
    }
    return __syncthreads_and(ok) != 0;
  };

  if (have) project(0);
  bool ok = fold(0);
  if (ok) {
    if (have) {
      double x[4] = {w0[0], w0[1], w0[2], w0[3]};
      subtract<TB>(nq, mine, coef, x);
#pragma unroll
      for (int t = 0; t < 4; ++t) wp[(4 * m + t) * 32 + lane] = x[t];
      team_sync(team);
      project(1);
    }
    ok = fold(1);
  }
  if (ok) {
    if (have) {
      double x[4] = {w0[0], w0[1], w0[2], w0[3]};
      subtract<TB>(nq, mine, coef, x);
      store_quad(a.Vout + base, r, m, lane, len, x);
#pragma unroll
      for (int t = 0; t < 4; ++t) wp[(4 * m + t) * 32 + lane] = x[t];
      team_sync(team);
      if (m == 0) {
        double n[1] = {0.0};
#pragma unroll
        for (int i = 0; i < kChain; ++i) {
          const double y = wp[i * 32 + lane];
          n[0] = fma(y, y, n[0]);
        }
        const double s = warp_tree<1>(n);
        if (lane == 0) peer_store1(peer_addr(norm + row, 0), s, peer_addr(bar + 2, 0));
      }
    }
    if (rank == 0 && warp == 0) {
      ok = wait_cluster(bar + 2, 0);
      if (ok) {
        double s = 0.0;
        if (lane < cs.nchunks) {
#pragma unroll
          for (int k = 0; k < kRows; ++k) s += norm[lane * kRows + k];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        close_step(c, b.ncases, cs_id, sqrt(s), *wn0, h1, h2);
      }
    }
  }
  if (!ok) {
    if (lane == 0 && err != nullptr) atomicExch(err, 1u);
    __syncwarp();
    cluster_sync();   // the other threads of the cluster finish, or give up and come here too, first
  }
}

// start vector: V_raw[0] = r and its squared norm ------------------------------
constexpr int kGB = 256;                 // threads per block
constexpr int kGE = kChunk / kGB;        // entries per thread

__device__ __forceinline__ void ldv(const double* p, double (&v)[4]) {
  const double2 t0 = *reinterpret_cast<const double2*>(p);
  const double2 t1 = *reinterpret_cast<const double2*>(p + 2);
  v[0] = t0.x; v[1] = t0.y; v[2] = t1.x; v[3] = t1.y;
}
__device__ __forceinline__ void stv(double* p, const double (&v)[4]) {
  *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void stv(__nv_bfloat16* p, const double (&v)[4]) {
  __nv_bfloat162 lo = __floats2bfloat162_rn((float)v[0], (float)v[1]);
  __nv_bfloat162 hi = __floats2bfloat162_rn((float)v[2], (float)v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

template <typename TB>
__global__ void __launch_bounds__(kGB) k_gs_start(Batch b, GsArgs<TB> a) {
  grid_wait();
  const Chunk ch = b.chunks[blockIdx.x];
  if (!case_live(b, ch.cs, a.need)) return;
  const CaseDev cs = b.cases[ch.cs];
  const size_t base = 4 * cs.cell_off + ch.begin;
  __shared__ double scratch[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double nrm = 0.0;
#pragma unroll
  for (int s = 0; s < kGE / 4; ++s) {
    const int e = 4 * (threadIdx.x + s * kGB);
    if (e < ch.len) {
      double x[4];
      ldv(a.w + base + e, x);
      stv(a.Vout + base + e, x);
#pragma unroll
      for (int u = 0; u < 4; ++u) nrm += x[u] * x[u];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nrm += __shfl_down_sync(0xffffffffu, nrm, o);
  if (lane == 0) scratch[warp] = nrm;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kGB / 32; ++w) s += scratch[w];
    a.part_norm[blockIdx.x] = s;
  }
}

// per-case close of an Arnoldi step (k >= 0) or of the start vector (k = -1),
// one warp per case ----
__global__ void __launch_bounds__(32) k_gs_close(Batch b, GsCloseArgs a) {
  grid_wait();
  const int cs_id = blockIdx.x;
  if ((a.live[cs_id] & a.need) != a.need) return;
  const CaseDev cs = b.cases[cs_id];
  const int lane = threadIdx.x;
  const double hn = sqrt(warp_chunk_sum(a.part_norm + cs.chunk0, 1, cs.nchunks));
  CaseCtl& c = a.ctl[cs_id];
  if (a.k < 0) {
    if (lane != 0) return;
    // _safe_normalize of the preconditioned residual: threshold eps
    const bool use = hn > DBL_EPSILON;
    const double beta = use ? hn : 0.0;
    a.scale[cs_id] = use ? 1.0 / hn : 0.0;
    c.beta = beta;
    c.k_used = 0;
    const bool run = beta > c.ptol && c.bnorm > 0.0;
    if (run) a.live[cs_id] |= kLiveKrylov;
    else a.live[cs_id] &= ~kLiveKrylov;
    return;
  }
  close_step(a, b.ncases, cs_id, hn, a.wn0[cs_id], a.h1 + (size_t)cs_id * kHStride, a.h2 + (size_t)cs_id * kHStride);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// whether the rows of a chunk go to CTAs of their own, eight CTAs for one: with at most half the
// SMs' number of chunks the GPU is idle otherwise (27 vectors, BF16, passes 1 / 2 / 3 in us,
// split against whole: 48 chunks 8 / 14 / 12 against 10 / 21 / 15; 128 chunks 13 / 25 / 23
// against 10 / 21 / 17, every CTA reducing the coefficients once more)
static bool gs_split(int nchunks) { return nchunks <= 148 / 2; }

// a pass over every chunk: with the chunks' rows on CTAs of their own (whole = false), the rows
// of a chunk are a cluster
template <typename TB>
static void launch_pass(void (*split)(Batch, GsArgs<TB>), void (*whole)(Batch, GsArgs<TB>), size_t split_smem,
                        const Batch& b, const GsArgs<TB>& a, cudaStream_t s) {
  if (!b.nchunks) return;
  if (!gs_split(b.nchunks)) {
    launch(whole, b.nchunks, 32 * warps_of(false), kRows * Ring<TB>::kBytes, s, b, a);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(b.nchunks, kRows);
  cfg.blockDim = dim3(32 * warps_of(true));
  cfg.dynamicSmemBytes = split_smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = kRows;
  at[0].val.clusterDim.z = 1;
  at[1] = dependent_launch();
  cfg.attrs = at;
  cfg.numAttrs = 2;
  (void)cudaLaunchKernelEx(&cfg, split, b, a);   // as <<<>>>: see cudaGetLastError
}
template <typename TB>
void launch_gs_dots(const Batch& b, const GsArgs<TB>& a, cudaStream_t s) {
  launch_pass<TB>(k_gs_dots<TB, true>, k_gs_dots<TB, false>, 0, b, a, s);
}
template <typename TB>
void launch_gs_project(const Batch& b, const GsArgs<TB>& a, cudaStream_t s) {
  launch_pass<TB>(k_gs_project<TB, true>, k_gs_project<TB, false>, gs_tile_bytes<TB>(a.nq), b, a, s);
}
template <typename TB>
void launch_gs_finish(const Batch& b, const GsArgs<TB>& a, cudaStream_t s) {
  launch_pass<TB>(k_gs_sub<TB, true>, k_gs_sub<TB, false>, 0, b, a, s);
}
template <typename TB>
void launch_gs_start(const Batch& b, const GsArgs<TB>& a, cudaStream_t s) {
  if (b.nchunks) launch(k_gs_start<TB>, b.nchunks, kGB, 0, s, b, a);
}
void launch_gs_close(const Batch& b, const GsCloseArgs& a, cudaStream_t s) {
  if (b.ncases) launch(k_gs_close, b.ncases, 32, 0, s, b, a);
}

// the launch of k_gs_case for all cases of up to `rows` rows
struct CaseLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  void (*kernel)(Batch, GsArgs<CaseBasis>, GsCloseArgs, uint32_t*, int);
  CaseLaunch(int ncases, int cluster, int rows, int nq, cudaStream_t s) {
    const int teams = (rows + cluster - 1) / cluster;
    // two teams at most: room for three CTAs on an SM, which a batch of 16 cases of 32 rows needs
    kernel = teams <= 2 ? k_gs_case<2> : k_gs_case<kTeams>;
    cfg.gridDim = dim3((unsigned)(ncases * cluster));
    cfg.blockDim = dim3((unsigned)(128 * teams));
    cfg.dynamicSmemBytes = CaseSmem(teams, rows, nq).bytes;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1] = dependent_launch();
    cfg.attrs = at;
    cfg.numAttrs = 2;
  }
};
int gs_case_vectors(int ncases, int cluster, int max_chunks, int nq) {
  const int rows = max_chunks * kRows;
  if (rows > kTeams * cluster || max_chunks > 32) return 0;
  if (ncases * cluster > 148 * (rows <= 2 * cluster ? 3 : 1)) return 0;   // more CTAs than run at once
  auto fits = [&](int q) {
    CaseLaunch l(ncases, cluster, rows, q, nullptr);
    if (l.cfg.dynamicSmemBytes > kCaseMaxSmem) return false;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, l.kernel, &l.cfg) == cudaSuccess) return n >= ncases;
    (void)cudaGetLastError();
    return false;
  };
  if (!fits(1)) return 0;
  while (!fits(nq)) --nq;
  return nq;
}
void launch_gs_case(const Batch& b, const GsArgs<CaseBasis>& a, const GsCloseArgs& c, uint32_t* err, int cluster,
                    int max_chunks, cudaStream_t s) {
  CaseLaunch l(b.ncases, cluster, max_chunks * kRows, a.nq, s);
  (void)cudaLaunchKernelEx(&l.cfg, l.kernel, b, a, c, err, max_chunks * kRows);   // as <<<>>>: see cudaGetLastError
}

#define A2D_GS_INST(TB)                                                                 \
  template void launch_gs_dots<TB>(const Batch&, const GsArgs<TB>&, cudaStream_t);     \
  template void launch_gs_project<TB>(const Batch&, const GsArgs<TB>&, cudaStream_t);  \
  template void launch_gs_finish<TB>(const Batch&, const GsArgs<TB>&, cudaStream_t);   \
  template void launch_gs_start<TB>(const Batch&, const GsArgs<TB>&, cudaStream_t);
A2D_GS_INST(double)
A2D_GS_INST(__nv_bfloat16)
#undef A2D_GS_INST

cudaError_t gs_init() {
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* f, size_t bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  for (auto f : {k_gs_case<2>, k_gs_case<kTeams>}) {
    set(reinterpret_cast<const void*>(f), kCaseMaxSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }
  set(reinterpret_cast<const void*>(&k_gs_project<__nv_bfloat16, true>), gs_tile_bytes<__nv_bfloat16>(kMaxRestart));
#define A2D_GS_ATTR(TB)                                                                       \
  set(reinterpret_cast<const void*>(&k_gs_dots<TB, false>), kRows * Ring<TB>::kBytes);       \
  set(reinterpret_cast<const void*>(&k_gs_project<TB, false>), kRows * Ring<TB>::kBytes);    \
  set(reinterpret_cast<const void*>(&k_gs_sub<TB, false>), kRows * Ring<TB>::kBytes);
  A2D_GS_ATTR(double)
  A2D_GS_ATTR(__nv_bfloat16)
#undef A2D_GS_ATTR
  return e;
}

}  // namespace a2d
