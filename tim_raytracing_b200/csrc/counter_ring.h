// counter_ring.h -- the work counters of tim_rt_trace_dev's launches, one slot a call.
#pragma once
#include <cstdint>

namespace timrt {

// Calls in flight at once, over all streams. A call takes two words, one for each kind of
// ray; the ring is not charged to the context's memory budget.
constexpr uint32_t kRingCalls = 4096, kRingWords = 2u * kRingCalls;
inline uint32_t ring_word(uint32_t call) { return 2u * (call % kRingCalls); }

}  // namespace timrt
