// How a bounded wait decides: tries alone first, then tries between readings of a clock.
#pragma once

namespace a2d {

#ifdef __CUDACC__
#define A2D_WAIT_HD __host__ __device__ __forceinline__
#else
#define A2D_WAIT_HD inline
#endif

constexpr unsigned long long kWaitLimitNs = 1000000000ull;   // 1 s

// tries before a wait starts to read the clock: most waits are over by then, and a
// %globaltimer read takes longer than they do
constexpr int kWaitTries = 64;

// Whether done() came true within the limit.  all(flag) makes one verdict of several lanes': each
// lane tries and reads the clock at its own time, so a phase that completes at the limit is seen by some of
// a warp's lanes and not by others, and lanes that give up while others go on to the warp's next
// vote, shuffle or barrier leave these waiting for ever.  One lane alone passes all(flag) = flag.
template <class Done, class Now, class All>
A2D_WAIT_HD bool bounded_wait(Done done, Now now_ns, All all) {
#ifdef __CUDACC__
#pragma unroll 1
#endif
  for (int q = 0; q < kWaitTries; ++q)
    if (all(done())) return true;
  const unsigned long long t0 = now_ns();
  while (!all(done())) {
    if (!all(now_ns() - t0 <= kWaitLimitNs)) return false;
  }
  return true;
}

}  // namespace a2d
