// Arrival counts of strips that several CTAs share, for kernels in which whoever delivers a strip's last partial sums finishes it.
//
// The counts lie in the caller's scratch, beside the partial sums, so that launches share them exactly where they share
// those: never in two streams, threads or graphs at a time.  Nothing clears scratch before a launch, and a launch of its own for that would
// cost more than the whole hand-over.  So a count carries the tag of the launch it belongs to: every contributor first opens
// the counts it will need (arrivals_open, once the kernels in front are done with the scratch), which replaces whatever else lies
// there by the tag and zero arrivals, and adds itself when its sums are written (arrivals_last).  The last one leaves a zero: a graph's replays
// have the same tag each time.
//
// Tags are 54 bits wide, never handed out twice and spread over all values, so that neither an earlier launch's words nor data
// that happened to lie there (2^-54 per word) look like an opened count.
//
// A contributor that gives up on a wait leaves counts half full, which a replay of its graph would take for its own.  So the tags are
// mixed with a word of the device that umma_reset_status() changes: what was left before the reset is another launch's after it.
// (Arrivals made good on the way out instead cost w4_stream.cu's main loop registers: decoder layer of one token 1.4 us of 125.)
#pragma once
#include <atomic>
#include "common.cuh"

namespace b2q {

using Arrivals = unsigned long long;
constexpr int ARRIVALS_BITS = 10, ARRIVALS_MAX = (1 << ARRIVALS_BITS) - 1;      // contributors to a strip

inline Arrivals arrivals_tag() {
  static std::atomic<unsigned long long> launches{0};
  return (launches.fetch_add(1, std::memory_order_relaxed) + 1) * 0x9E3779B97F4A7C15ull << ARRIVALS_BITS;      // odd factor: one to one
}

const Arrivals* arrivals_epoch();      // the current device's; umma_gemm.cu

#ifdef __CUDACC__
__device__ __forceinline__ void arrivals_open(Arrivals* count, Arrivals tag, const Arrivals* epoch) {
  const Arrivals v = *reinterpret_cast<volatile Arrivals*>(count), t = tag ^ *reinterpret_cast<const volatile Arrivals*>(epoch) << ARRIVALS_BITS;
  if ((v ^ t) >> ARRIVALS_BITS) atomicCAS(count, v, t);                // where it fails, another contributor has just opened the count
}
// Whether this contributor is the last of others + 1.
__device__ __forceinline__ bool arrivals_last(Arrivals* count, int others) {
  const bool last = (int)(atomicAdd(count, 1ull) & ARRIVALS_MAX) == others;
  if (last) *reinterpret_cast<volatile Arrivals*>(count) = 0;
  return last;
}
#endif

}  // namespace b2q
