// The whole line preconditioner x = M^-1 r in one launch: every line-Jacobi sweep of
// a case (aero2d/implicit.py:130-157; the mathematics is in sweep.cu) by one thread-block
// cluster, a CTA per 32-line group.
//
// What bounds it.  Separate launches per sweep read the factors P, Q, G, C (128 B a
// cell in FP16) from HBM in every sweep, send e0 and x' through L2 between launches, and put a
// row's coupling products and its recurrence step one after the other in the same warps; a
// small batch then waits on the length of a step, a large one on both.  Here
//   * the coupling e_j = e0_j + P_j x'[i-1]_j - Q_j x'[i+1]_j, which no row needs another
//     row for, is formed by kHelpers warps, a row of 32 lines per warp at a time (P and Q
//     straight from global memory, kAhead rows in flight), into shared memory, following the
//     back substitution of the sweep before outward from the twist row;
//   * two warps run the recurrences alone, from the wall and from the far field (a lane per
//     line, all four rows of a block in the lane: no barrier and no exchange in a step),
//     with G and C arriving through a ring of bulk copies that two service warps keep full,
//     also across sweeps;
//   * e_j, d_j and x_j of a line group live in one shared-memory array, each in place of
//     the one before; only the group's first and last line go to the neighbouring CTAs, by
//     asynchronous stores into their shared memory that count their bytes on an mbarrier
//     there (release fences in their place cost 7 us a sweep).
// A cluster's factors come from HBM in its first sweeps and from L2 after: residency is two
// CTAs per SM, about 37 cases of 256 x 64 (2 MB of FP16 factors each) on the 126 MB L2.
// What is left is the recurrence's length (about 215 cycles a row of one warp, of which the
// dependent products are 20) and, past 37 cases, the second wave.
// Measured (B200, four sweeps, mixed, 256 x 64): 1 case 85 -> 39 us, 16 cases 99 -> 54, 64
// cases 180 -> 137; 384 x 96, 12 cases 131 -> 88; FP64 256 x 64, 1 case 178 -> 63.
//
// The arithmetic of every row and its order are those of the per-sweep kernels
// (sweep.cu, sweep_rows.cu, sweep_pairs.cu), so results are bitwise the same.  Every wait is
// bounded (tma.cuh); a wait that runs out records an error, and its CTA stays until
// the other CTAs of the cluster are done or have given up too, so none of them
// stores into the shared memory of a CTA that has gone.  A warp leaves as a whole (waits.cuh):
// helper and service warps by their waits' vote, which costs 1 to 2 % of an application in the
// recurrence warps; there a lane whose wait runs out is no longer `alive`, waits for nothing
// further and signals nothing, and the warp votes once, at the end.  No cluster multicast.
#include <algorithm>
#include <type_traits>

#include "batch.cuh"
#include "cluster.cuh"
#include "kernels.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace a2d {
namespace lines {

constexpr int kHelpers = 8;                       // coupling warps (a multiple of 2: alternating halves)
constexpr int kStep = kHelpers / 2;               // rows of a half between two rows of one helper
constexpr int kService0 = 2 + kHelpers;          // warps: 0 wall, 1 far field, helpers, service
constexpr int kThreads = 32 * (kService0 + 2);
constexpr int kBlockEntries = 16 * kLanes;        // one 4x4 block for the 32 lines of a group
constexpr int kPack = 4;                          // blocks per ring stage, rows per step of the recurrence loops
constexpr int kBatch = kStep;                     // rows of a half signalled together, one per helper
static_assert(kBatch == kPack, "a forward pack is one batch of e rows");
constexpr int kMaxCluster = 16;                   // CTAs: lines of up to 512 cells round the airfoil
constexpr int kMaxSmem = 227 * 1024;

template <typename TI> struct Types;
template <> struct Types<float> {
  using TF = __half;
  using TC = float;
  static constexpr int kAhead = 2;                // rows a helper keeps in flight
  static constexpr int kStages = 4;               // ring stages per half
  static constexpr int kCtas = 2;                 // resident per SM
};
template <> struct Types<double> {
  using TF = double;
  using TC = double;
  static constexpr int kAhead = 1;
  static constexpr int kStages = 2;
  static constexpr int kCtas = 1;
};

// shared memory of a CTA for lines of up to `rows` cells
template <typename TI>
struct Smem {
  using TC = typename Types<TI>::TC;
  using TF = typename Types<TI>::TF;
  static constexpr int kStages = Types<TI>::kStages;
  static constexpr uint32_t kBlk = kBlockEntries * sizeof(TF);
  static constexpr uint32_t kRow = kLanes * 4 * sizeof(TC);
  static constexpr uint32_t kRing = 2 * kStages * kPack * kBlk;
  static constexpr uint32_t kEdge = 4 * sizeof(TC);
  // ring, rows, x_k, edges [parity][side][row], mbarriers
  __host__ __device__ static uint32_t off_rows() { return kRing; }
  __host__ __device__ static uint32_t off_xk(int rows) { return off_rows() + (uint32_t)rows * kRow; }
  __host__ __device__ static uint32_t off_edge(int rows) { return off_xk(rows) + kRow; }
  __host__ __device__ static uint32_t off_bars(int rows) { return off_edge(rows) + 4u * rows * kEdge; }
  __host__ __device__ static int batches(int rows) { return rows / 2 / kBatch + 2; }   // per half
  // full, empty [half][stage]; meet [2]; then per half and batch: ready, edge [parity]; row k's
  // edge [parity]
  __host__ __device__ static int bars(int rows) { return 4 * kStages + 2 + 6 * batches(rows) + 2; }
  __host__ __device__ static uint32_t bytes(int rows) { return off_bars(rows) + 8u * bars(rows); }
};

// ---- loads ----
__device__ __forceinline__ uint2 ldg_stream(const __half* p) {
  uint2 r;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ float4 ldg_stream(const float* p) {
  float4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
               : "l"(p));
  return r;
}
struct Raw4d {
  double2 a, b;
};
__device__ __forceinline__ Raw4d ldg_stream(const double* p) {
  Raw4d r;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(r.a.x), "=d"(r.a.y) : "l"(p));
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(r.b.x), "=d"(r.b.y) : "l"(p + 2));
  return r;
}
__device__ __forceinline__ void widen(const uint2& raw, float (&v)[4]) {
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void widen(const float4& t, float (&v)[4]) {
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void widen(const Raw4d& t, double (&v)[4]) {
  v[0] = t.a.x; v[1] = t.a.y; v[2] = t.b.x; v[3] = t.b.y;
}
template <typename T> struct RawOf;
template <> struct RawOf<__half> { using type = uint2; };
template <> struct RawOf<float> { using type = float4; };
template <> struct RawOf<double> { using type = Raw4d; };

// four entries of a block row from shared memory
__device__ __forceinline__ uint2 lds_raw(const __half* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ Raw4d lds_raw(const double* p) {
  return Raw4d{*reinterpret_cast<const double2*>(p), *reinterpret_cast<const double2*>(p + 2)};
}

// the 4-vector of one lane in a row of the line array: FP32 one 16-byte entry per
// lane; FP64 two halves of 16 bytes (no bank conflicts either way)
__device__ __forceinline__ void row_load(const float* row, int l, float (&v)[4]) {
  const float4 t = reinterpret_cast<const float4*>(row)[l];
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void row_store(float* row, int l, const float (&v)[4]) {
  reinterpret_cast<float4*>(row)[l] = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void row_load(const double* row, int l, double (&v)[4]) {
  const double2 a = reinterpret_cast<const double2*>(row)[l], b = reinterpret_cast<const double2*>(row)[kLanes + l];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void row_store(double* row, int l, const double (&v)[4]) {
  reinterpret_cast<double2*>(row)[l] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(row)[kLanes + l] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void edge_load(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void edge_load(const double* p, double (&v)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// e0 of one lane, read back by the thread that stored it (plain accesses: the compiler may
// move a __ldcg over the store)
__device__ __forceinline__ void e0_load(const float* p, float (&v)[4]) { widen(*reinterpret_cast<const float4*>(p), v); }
__device__ __forceinline__ void e0_store(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void e0_load(const double* p, double (&v)[4]) {
  widen(Raw4d{reinterpret_cast<const double2*>(p)[0], reinterpret_cast<const double2*>(p)[1]}, v);
}
__device__ __forceinline__ void e0_store(double* p, const double (&v)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// one row of a block times a 4-vector, as the per-sweep kernels write it (the compiler
// contracts both the same way)
template <typename T>
__device__ __forceinline__ T dot4(const T (&a)[4], const T (&b)[4]) {
  T s = a[0] * b[0];
#pragma unroll
  for (int q = 1; q < 4; ++q) s += a[q] * b[q];
  return s;
}
template <typename T>
__device__ __forceinline__ T add_dot4(T s, const T (&a)[4], const T (&b)[4]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) s += a[q] * b[q];
  return s;
}

// one 4-vector into another CTA's shared memory, its bytes counted on an mbarrier there: the
// waiter needs no fence or arrival of ours (a cluster fence takes longer than a pack's rows)
__device__ __forceinline__ void peer_store(uint32_t addr, const float (&v)[4], uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
      "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void peer_store(uint32_t addr, const double (&v)[4], uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "d"(v[0]), "d"(v[1]), "r"(bar)
               : "memory");
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr + 16),
               "d"(v[2]), "d"(v[3]), "r"(bar)
               : "memory");
}
extern __shared__ __align__(128) unsigned char lines_sm[];

// the CTA's view of its lines; everything shared is addressed from lines_sm, so that the
// compiler sees shared memory and not a generic pointer
template <typename TI>
struct Cta {
  using TC = typename Types<TI>::TC;
  using TF = typename Types<TI>::TF;
  using SM = Smem<TI>;
  static constexpr int S = Types<TI>::kStages;
  int rows_cap;      // rows that the shared arrays hold
  int ni, nc, k;     // k: the twist row
  int n;             // lines of the group
  __device__ __forceinline__ int count(int h) const { return h == 0 ? k + 1 : nc - 1 - k; }   // e rows of a half
  __device__ __forceinline__ int row_of(int h, int t) const { return h == 0 ? t : nc - 1 - t; }
  __device__ __forceinline__ unsigned char* stage(int h, int s) const {
    return lines_sm + (uint32_t)(h * S + s) * kPack * SM::kBlk;
  }
  // e, d, x of row j: [lane][4], see row_load
  __device__ __forceinline__ TC* row(int j) const {
    return reinterpret_cast<TC*>(lines_sm + SM::off_rows() + (uint32_t)j * SM::kRow);
  }
  // x_k of the wall half, for the far half
  __device__ __forceinline__ TC* xk() const { return reinterpret_cast<TC*>(lines_sm + SM::off_xk(rows_cap)); }
  // x of the line before the group (side 0) and after it (side 1), by sweep parity
  __device__ __forceinline__ TC* edge_at(int parity, int side, int j) const {
    return reinterpret_cast<TC*>(lines_sm + SM::off_edge(rows_cap) +
                                 (uint32_t)((parity * 2 + side) * rows_cap + j) * SM::kEdge);
  }
  __device__ __forceinline__ uint64_t* bar(int q) const {
    return reinterpret_cast<uint64_t*>(lines_sm + SM::off_bars(rows_cap)) + q;
  }
  __device__ __forceinline__ uint64_t* full(int h, int s) const { return bar(h * S + s); }
  __device__ __forceinline__ uint64_t* empty(int h, int s) const { return bar(2 * S + h * S + s); }
  // [0] d'_{k+1} of the far half, [1] x_k of the wall half
  __device__ __forceinline__ uint64_t* meet(int q) const { return bar(4 * S + q); }
  __device__ __forceinline__ uint64_t* batch_bar(int kind, int h, int q) const {
    return bar(4 * S + 2 + (kind * 2 + h) * SM::batches(rows_cap) + q);
  }
  // a forward batch of a half's e rows is in place (rows counted inward from the half's end)
  __device__ __forceinline__ uint64_t* ready(int h, int q) const { return batch_bar(0, h, q); }
  // a back pack of a half's x rows (counted outward from row k) is in place, and the
  // neighbours' lines of it, and the rows may be overwritten; by sweep parity
  __device__ __forceinline__ uint64_t* edge_bar(int parity, int h, int q) const {
    return batch_bar(1 + parity, h, q);
  }
  // the same for row k
  __device__ __forceinline__ uint64_t* k_edge(int parity) const {
    return bar(4 * S + 2 + 6 * SM::batches(rows_cap)) + parity;
  }
};

// ======================= service warp of half h =======================
// Keeps the half's ring full: the stages of one sweep are forward packs of up to kPack G
// blocks, the wall half's (G, H) of the twist row, back packs of up to kPack C blocks
// (consecutive rows: one copy); the same again for the next sweep.  And, as the recurrence
// gives back the stage of a back pack (or of the twist row), whose x rows are then in
// place: stores the group's first and last line of those rows into the neighbouring CTAs.
__host__ __device__ __forceinline__ int packs(int rows) { return (rows + kPack - 1) / kPack; }

template <typename TI>
__device__ __forceinline__ bool serve(const Cta<TI> c, const SweepArgs& a, size_t blk0, int sweeps, int h, int lane,
                                      uint32_t prev, uint32_t next) {
  using TF = typename Types<TI>::TF;
  using TC = typename Types<TI>::TC;
  constexpr int S = Types<TI>::kStages;
  constexpr uint32_t kBlk = Smem<TI>::kBlk;
  const TF* G = static_cast<const TF*>(a.PQG) + 3 * blk0 + 2 * kBlockEntries;   // row j at j * 3 blocks
  const TF* C = static_cast<const TF*>(a.CF) + blk0;
  const int nf = h == 0 ? c.k : c.nc - 1 - c.k;
  const int np = packs(nf), mid = h == 0 ? 1 : 0, per = 2 * np + mid;
  const int total = per * sweeps;
  int fq = 0;                      // pack of its sweep that the next fill brings
  auto fill = [&](int s) {
    if (lane == 0) {
      unsigned char* dst = c.stage(h, s);
      uint64_t* full = c.full(h, s);
      if (fq < np) {
        const int t = fq * kPack, cnt = min(kPack, nf - t);
        mbar_arrive_expect(full, cnt * kBlk);
        for (int u = 0; u < cnt; ++u)
          bulk_load(dst + u * kBlk, G + (size_t)c.row_of(h, t + u) * (3 * kBlockEntries), kBlk, full);
      } else if (fq < np + mid) {
        mbar_arrive_expect(full, 2 * kBlk);
        bulk_load(dst, G + (size_t)c.k * (3 * kBlockEntries), kBlk, full);
        bulk_load(dst + kBlk, C + (size_t)c.k * kBlockEntries, kBlk, full);
      } else {
        const int t = (fq - np - mid) * kPack, cnt = min(kPack, nf - t);
        const int low = h == 0 ? c.k - t - cnt : c.k + 1 + t;   // the pack's lowest row
        mbar_arrive_expect(full, cnt * kBlk);
        bulk_load(dst, C + (size_t)low * kBlockEntries, cnt * kBlk, full);
      }
    }
    if (++fq == per) fq = 0;
  };
  for (int p = 0; p < min(S, total); ++p) fill(p);
  int s = 0, uq = 0, sw = 0;       // stage given back, its pack and sweep
  uint32_t ph = 0;
#pragma unroll 1
  for (int p = 0; p < total; ++p) {
    if (!mbar_wait_warp(c.empty(h, s), ph)) {
      // the recurrence stopped: the copies in flight get a bounded time to land
      for (int u = p; u < min(p + S, total); ++u) (void)mbar_wait(c.full(h, u % S), (u / S) & 1);
      return false;
    }
    if (uq >= np && sw + 1 < sweeps) {
      const int par = sw & 1;
      const bool twist = uq < np + mid;
      const int t = (uq - np - mid) * kPack, cnt = twist ? 1 : min(kPack, nf - t);
      const int j0 = twist ? c.k : (h == 0 ? c.k - t - cnt : c.k + 1 + t);
      uint64_t* eb = twist ? c.k_edge(par) : c.edge_bar(par, h, t / kPack);
      // the group's first line is the line after the previous group's last one, its last the
      // line before the next group's first
      const int side = lane & 1, j = j0 + (lane >> 1);
      const uint32_t to = side == 0 ? prev : next;
      if (lane < 2 * cnt) {
        TC v[4];
        row_load(c.row(j), side == 0 ? 0 : c.n - 1, v);
        peer_store(peer_addr(c.edge_at(par, 1 - side, j), to), v, peer_addr(eb, to));
      }
      __syncwarp();
      // read, so that the rows may be overwritten; and as many bytes come from the neighbours
      if (lane == 0) mbar_arrive_expect(eb, 2 * cnt * Smem<TI>::kEdge);
    }
    if (p + S < total) fill(s);
    if (++uq == per) {
      uq = 0;
      ++sw;
    }
    if (++s == S) {
      s = 0;
      ph ^= 1;
    }
  }
  return true;
}

// ======================= helper warp: e rows =======================
template <typename TI, bool FIRST> struct Pre;
template <typename TI> struct Pre<TI, true> {
  typename RawOf<TI>::type inv[4];
  double r[4];
};
template <typename TI> struct Pre<TI, false> {
  typename RawOf<typename Types<TI>::TF>::type p[4], q[4];
  typename Types<TI>::TC e0[4];
};

// rows of helper hw (its half hw & 1): in the first sweep from the half's end inward, in
// the order the recurrence takes them; later from row k outward, in the order the back
// substitution before completes their x (the wall half's row k last), so that all but the
// last pack of e rows is formed while that back substitution still runs
template <typename TI, bool FIRST>
__device__ __forceinline__ bool couple(const Cta<TI> c, const SweepArgs& a, size_t blk0, size_t vbase, int i,
                                       int sweep, int sweeps, int hw, int lane) {
  using TF = typename Types<TI>::TF;
  using TC = typename Types<TI>::TC;
  constexpr int U = Types<TI>::kAhead;
  const int h = hw & 1, q0 = hw >> 1;
  const int nf = h == 0 ? c.k : c.nc - 1 - c.k;
  // the helper's rows are the same in every sweep (its e0 is read back by the thread that
  // wrote it): v counts rows outward from row k, congruent to q0 modulo kStep; row k itself is
  // v = -1, taken last
  const int first_v = FIRST ? ((nf - 1 - q0) % kStep + kStep) % kStep : q0;
  const int tail = h == 0 && q0 == kStep - 1 ? 1 : 0;
  const int cnt = FIRST ? c.count(h) : nf + (tail ? (q0 - nf % kStep + kStep) % kStep + 1 : 0);
  const int comp = c.nc * c.ni;
  const TI* INV = static_cast<const TI*>(a.INV) + blk0 + lane * 4;
  const TF* PQ = static_cast<const TF*>(a.PQG) + 3 * blk0 + lane * 4;
  TC* e0v = reinterpret_cast<TC*>(a.e0) + blk0 / 4 + lane * 4;   // [row][lane][4], as the blocks are
  const double* rv = a.r + vbase + i;
  auto row_at = [&](int v) {
    if (FIRST) return c.row_of(h, v);
    return h == 0 ? (v < nf ? c.k - 1 - v : c.k) : c.k + 1 + v;
  };
  Pre<TI, FIRST> pre[U];
  auto load = [&](Pre<TI, FIRST>& p, int v) {
    if (v >= cnt) return;
    const int j = row_at(v);
    if constexpr (FIRST) {
#pragma unroll
      for (int r = 0; r < 4; ++r) p.inv[r] = ldg_stream(INV + (size_t)j * kBlockEntries + r * kLanes * 4);
#pragma unroll
      for (int r = 0; r < 4; ++r) p.r[r] = __ldcg(rv + r * comp + j * c.ni);
    } else {
      const TF* b = PQ + (size_t)j * (3 * kBlockEntries);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        p.p[r] = ldg_stream(b + r * kLanes * 4);
        p.q[r] = ldg_stream(b + kBlockEntries + r * kLanes * 4);
      }
      e0_load(e0v + (size_t)j * (kLanes * 4), p.e0);
    }
  };
#pragma unroll
  for (int u = 0; u < U; ++u) load(pre[u], first_v + u * kStep);
  const uint32_t par = (sweep - 1) & 1;              // parity of the sweep whose x is read
  const uint32_t ph = ((sweep - 1) >> 1) & 1;        // and the phase of that parity's barriers
#pragma unroll 1
  for (int vb = first_v; vb < cnt; vb += U * kStep) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = vb + u * kStep;
      if (v < cnt) {
        const int j = row_at(v);
        TC* row = c.row(j);
        TC e[4];
        if constexpr (FIRST) {
          TC rr[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) rr[r] = TC(pre[u].r[r]);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            TC iv[4];
            widen(pre[u].inv[r], iv);
            e[r] = dot4(iv, rr);
          }
          if (sweeps > 1) e0_store(e0v + (size_t)j * (kLanes * 4), e);
        } else {
          const bool twist = v >= nf;
          uint64_t* eb = twist ? c.k_edge(par) : c.edge_bar(par, h, v / kPack);
          TC xm[4], xp[4];
          if (!wait_cluster(eb, ph)) return false;
          row_load(row, lane == 0 ? 0 : lane - 1, xm);
          row_load(row, lane == kLanes - 1 ? lane : lane + 1, xp);
          if (lane == 0) edge_load(c.edge_at(par, 0, j), xm);
          if (lane == c.n - 1) edge_load(c.edge_at(par, 1, j), xp);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            TC pv[4], qv[4];
            widen(pre[u].p[r], pv);
            widen(pre[u].q[r], qv);
            e[r] = pre[u].e0[r] + dot4(pv, xm) - dot4(qv, xp);
          }
          __syncwarp();   // every lane has read its neighbours' x before the row is overwritten
        }
        load(pre[u], v + U * kStep);
        row_store(row, lane, e);
        __syncwarp();
        if (lane == 0) mbar_arrive(c.ready(h, (h == 0 ? j : c.nc - 1 - j) / kBatch));
      }
    }
  }
  return true;
}

// ======================= recurrence warp of half h =======================
template <typename TI>
__device__ __forceinline__ bool recur(const Cta<TI> c, const SweepArgs& a, size_t vbase, int i, bool owner, int sweeps, int h,
                      int lane) {
  using TC = typename Types<TI>::TC;
  using TF = typename Types<TI>::TF;
  using Raw = typename RawOf<TF>::type;
  constexpr int S = Types<TI>::kStages;
  constexpr uint32_t kBlk = Smem<TI>::kBlk;
  const int k = c.k, nc = c.nc;
  const int nf = h == 0 ? k : nc - 1 - k;
  const int comp = nc * c.ni;
  double* xg = a.x + vbase + i;
  const int dir = h == 0 ? 1 : -1;
  int s = 0;              // ring stage
  uint32_t sph = 0;       // and its phase
  bool alive = true;
  // block u of the stage, this lane's four rows
  auto block = [&](int u, Raw(&raw)[4]) {
    const TF* b = reinterpret_cast<const TF*>(c.stage(h, s) + u * kBlk) + lane * 4;
#pragma unroll
    for (int r = 0; r < 4; ++r) raw[r] = lds_raw(b + r * kLanes * 4);
  };
  // the stage is used up: called after the store of a value computed from its last block,
  // so that its loads have returned (an arrival alone does not wait for them) before it is
  // overwritten
  auto retire = [&]() {
    __syncwarp();
    if (lane == 0 && alive) mbar_arrive(c.empty(h, s));
    if (++s == S) {
      s = 0;
      sph ^= 1;
    }
  };
  // a try at the next stage (and forward batch), made before a pack is worked on, so that its
  // result is there when the pack is done: a wait that succeeds at once still takes ~90 cycles
  auto try_next = [&]() { return s + 1 == S ? mbar_test(c.full(h, 0), sph ^ 1) : mbar_test(c.full(h, s + 1), sph); };
  bool have = false, have_e = false;
  // N rows of a pack, two in flight: `in(u)` the row and block of step u, `out(u, v)` stores
  // its result; step: result from (block, row vector, v), v the result of the step before
  auto walk = [&](auto count, auto in, auto step, auto out, TC(&v)[4]) {
    constexpr int N = decltype(count)::value, W = N < 2 ? N : 2;
    Raw raw[W][4];
    TC y[W][4];
#pragma unroll
    for (int u = 0; u < W; ++u) in(u, y[u], raw[u]);
#pragma unroll
    for (int u = 0; u < N; ++u) {
      TC z[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        TC g[4];
        widen(raw[u % W][r], g);
        z[r] = step(g, y[u % W][r], v);
      }
      if (u + W < N) in(u + W, y[u % W], raw[u % W]);
      out(u, z);
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] = z[r];
    }
  };
  using Full = std::integral_constant<int, kPack>;
  using One = std::integral_constant<int, 1>;
#pragma unroll 1
  for (int sw = 0; sw < sweeps; ++sw) {
    const bool last = sw == sweeps - 1;
    const uint32_t ph = sw & 1;
    // forward: d_j = e_j + G_j d_{j-1}, a pack of rows at a time
    TC d[4] = {TC(0), TC(0), TC(0), TC(0)};
    have_e = false;
    auto fstep = [](const TC(&g)[4], TC e, const TC(&v)[4]) { return add_dot4(e, g, v); };
#pragma unroll 1
    for (int t = 0; t < nf; t += kPack) {
      const int j = c.row_of(h, t);
      alive = alive && (have || mbar_wait(c.full(h, s), sph));
      alive = alive && (have_e || mbar_wait(c.ready(h, t / kBatch), ph));
      have = try_next();
      have_e = t + kPack < nf && mbar_test(c.ready(h, t / kBatch + 1), ph);
      int u0 = 0;
      auto in = [&](int u, TC(&y)[4], Raw(&raw)[4]) {
        row_load(c.row(j + (u0 + u) * dir), lane, y);
        block(u0 + u, raw);
      };
      auto out = [&](int u, const TC(&z)[4]) { row_store(c.row(j + (u0 + u) * dir), lane, z); };
      if (nf - t >= kPack) {
        walk(Full(), in, fstep, out, d);
      } else {
#pragma unroll 1
        for (; u0 < nf - t; ++u0) walk(One(), in, fstep, out, d);
      }
      retire();
    }
    // the halves meet at row k
    TC x[4];
    if (h == 0) {
      alive = alive && mbar_wait(c.ready(0, k / kBatch), ph);
      alive = alive && (have || mbar_wait(c.full(h, s), sph));
      alive = alive && mbar_wait(c.meet(0), ph);
      have = try_next();
      TC e[4], dp[4] = {TC(0), TC(0), TC(0), TC(0)};
      row_load(c.row(k), lane, e);
      if (nc - 1 - k > 0) row_load(c.row(k + 1), lane, dp);   // d'_{k+1}
      Raw raw[4];
      block(0, raw);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        TC g[4];
        widen(raw[r], g);
        x[r] = add_dot4(e[r], g, d);
      }
      block(1, raw);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        TC g[4];
        widen(raw[r], g);
        x[r] = add_dot4(x[r], g, dp);
      }
      row_store(c.xk(), lane, x);
      if (!last) row_store(c.row(k), lane, x);
      __syncwarp();
      if (lane == 0 && alive) mbar_arrive(c.meet(1));
      retire();
      if (last && owner) {
#pragma unroll
        for (int r = 0; r < 4; ++r) xg[r * comp + k * c.ni] = (double)x[r];
      }
    } else {
      __syncwarp();
      if (lane == 0 && alive) mbar_arrive(c.meet(0));
      // also without rows of its own: a half runs at most one sweep ahead of the other
      alive = alive && mbar_wait(c.meet(1), ph);
      row_load(c.xk(), lane, x);
    }
    // back substitution outward from row k: x_j = d_j - C_j x_{j+-1}
    auto bstep = [](const TC(&g)[4], TC y, const TC(&v)[4]) { return y - dot4(g, v); };
#pragma unroll 1
    for (int t = 0; t < nf; t += kPack) {
      const int j = h == 0 ? k - 1 - t : k + 1 + t;
      const int top = min(kPack, nf - t) - 1;    // the wall half walks down the pack's rows
      alive = alive && (have || mbar_wait(c.full(h, s), sph));
      have = try_next();
      int u0 = 0;
      auto in = [&](int u, TC(&y)[4], Raw(&raw)[4]) {
        row_load(c.row(j - (u0 + u) * dir), lane, y);
        block(h == 0 ? top - u0 - u : u0 + u, raw);
      };
      auto out = [&](int u, const TC(&z)[4]) {
        const int jj = j - (u0 + u) * dir;
        if (!last) {
          row_store(c.row(jj), lane, z);
        } else if (owner) {
#pragma unroll
          for (int r = 0; r < 4; ++r) xg[r * comp + jj * c.ni] = (double)z[r];
        }
      };
      if (nf - t >= kPack) {
        walk(Full(), in, bstep, out, x);
      } else {
#pragma unroll 1
        for (; u0 < nf - t; ++u0) walk(One(), in, bstep, out, x);
      }
      retire();
    }
  }
  return warp_all(alive);
}

template <typename TI>
__global__ void __launch_bounds__(kThreads, Types<TI>::kCtas) k_lines(Batch b, SweepArgs a, const int* cases, int sweeps,
                                                       int rows_cap) {
  grid_wait();
  using SM = Smem<TI>;
  constexpr int S = Types<TI>::kStages;
  const uint32_t size = cluster_size(), rank = cluster_rank();
  const int cs_id = cases[blockIdx.x / size];
  if (!case_live(b, cs_id, a.need)) return;    // the whole cluster leaves
  const CaseDev cs = b.cases[cs_id];
  const Group grp = b.groups[cs.group0 + (int)rank];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Cta<TI> c;
  c.rows_cap = rows_cap;
  c.ni = cs.g.ni;
  c.nc = cs.g.nc;
  c.k = c.nc / 2;
  c.n = grp.n;
  const int nbatch = SM::batches(rows_cap);
  for (int q = threadIdx.x; q < SM::bars(rows_cap); q += kThreads) {
    uint32_t arrivals = 1;
    const int u = q - (4 * S + 2);
    if (u >= 0 && u < 2 * nbatch) {
      const int left = c.count(u / nbatch) - u % nbatch * kBatch;   // ready: a helper per row of the batch
      arrivals = left < 1 ? 1 : min(left, kBatch);
    }
    mbar_init(c.bar(q), arrivals);
  }
  mbar_init_fence();
  __syncthreads();
  if (sweeps > 1) cluster_sync();   // the neighbours' mbarriers exist before anything is stored there

  const size_t blk0 = lbidx(cs.rows_nc, c.nc, grp.g, 0, 0, 0);
  const size_t vbase = 4 * (size_t)cs.cell_off;
  const bool owner = lane < grp.n;             // lanes past the group's last line only compute
  const int i = grp.i0 + (owner ? lane : grp.n - 1);
  const uint32_t prev = rank == 0 ? size - 1 : rank - 1, next = rank + 1 == size ? 0 : rank + 1;
  bool ok = true;
  if (warp < 2) {
    ok = recur<TI>(c, a, vbase, i, owner, sweeps, warp, lane);
  } else if (warp < kService0) {
    ok = couple<TI, true>(c, a, blk0, vbase, i, 0, sweeps, warp - 2, lane);
#pragma unroll 1
    for (int sw = 1; sw < sweeps && ok; ++sw)
      ok = couple<TI, false>(c, a, blk0, vbase, i, sw, sweeps, warp - 2, lane);
  } else {
    ok = serve<TI>(c, a, blk0, sweeps, warp - kService0, lane, prev, next);
  }
  if (!ok) {
    if (lane == 0 && a.err != nullptr) atomicExch(a.err, 1u);
    __syncwarp();
    // the other threads of the cluster finish, or give up and come here too, first
    cluster_sync();
  }
}

}  // namespace lines

// the launch of `count` clusters of `groups` CTAs, for lines of up to `rows` cells
template <typename TI>
struct LinesLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  LinesLaunch(int count, int groups, int rows, cudaStream_t s) {
    cfg.gridDim = dim3((unsigned)(count * groups));
    cfg.blockDim = dim3(lines::kThreads);
    cfg.dynamicSmemBytes = lines::Smem<TI>::bytes(rows);
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)groups;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1] = dependent_launch();
    cfg.attrs = at;
    cfg.numAttrs = 2;
  }
};

template <typename TI>
bool lines_take(int groups, int rows) {
  return groups <= lines::kMaxCluster && lines::Smem<TI>::bytes(rows) <= (uint32_t)lines::kMaxSmem;
}

template <typename TI>
int lines_clusters(int groups, int rows) {
  if (!lines_take<TI>(groups, rows)) return 0;
  LinesLaunch<TI> l(1, groups, rows, nullptr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, lines::k_lines<TI>, &l.cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

template <typename TI>
void launch_lines(const Batch& b, const SweepArgs& a, const int* cases, int count, int groups, int rows, int sweeps,
                  cudaStream_t s) {
  if (count == 0) return;
  LinesLaunch<TI> l(count, groups, rows, s);
  (void)cudaLaunchKernelEx(&l.cfg, lines::k_lines<TI>, b, a, cases, sweeps, rows);   // as <<<>>>: see cudaGetLastError
}

cudaError_t lines_init() {
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* f) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, lines::kMaxSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  };
  set(reinterpret_cast<const void*>(&lines::k_lines<float>));
  set(reinterpret_cast<const void*>(&lines::k_lines<double>));
  return e;
}

template bool lines_take<float>(int, int);
template bool lines_take<double>(int, int);
template int lines_clusters<float>(int, int);
template int lines_clusters<double>(int, int);
template void launch_lines<float>(const Batch&, const SweepArgs&, const int*, int, int, int, int, cudaStream_t);
template void launch_lines<double>(const Batch&, const SweepArgs&, const int*, int, int, int, int, cudaStream_t);

}  // namespace a2d
