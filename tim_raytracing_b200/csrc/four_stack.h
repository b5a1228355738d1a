// four_stack.h -- the stack of an any-hit ray's walk on the 4-wide tree (trace_any.cuh).
//
// A reference of an inner node is its index and, from bit 25 up, the levels of inner nodes
// below it at most. An entered node's slots go onto the stack one word each while the rest
// of the walk is sure of one word for every level below: a walk at a node with `below`
// levels under it and `used` words on its stack then keeps
//   used + below + 1 <= words - 1   (word 0 is the end marker)
// Pushing slots leaves three more words at a level less, and writes the word above them;
// it is done where used + below <= words - 5. Otherwise the node waits as a whole, in one
// word (its index and the slots yet to visit), from which its references are read again
// one by one: one more word at a level less. So no walk runs out of words, and a tree whose
// slots fit, 3 words a level, never has a node wait.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TIMRT_HD __host__ __device__ __forceinline__
#else
#define TIMRT_HD inline
#endif

namespace timrt {

constexpr uint32_t kFourBelowShift = 25, kFourIndexMask = (1u << kFourBelowShift) - 1u;
constexpr uint32_t kFourWaiting = 1u << 30;   // a waiting node: index << 4 | slots

// Most stack words of an any-hit ray, but for trees of more levels. 24 against 18 words:
// the frame's any-hit rays the same, a probe update in 1M triangles 3.24 against 3.43 ms,
// 20,000 rays among 20,000 crossing needles, of which nearly every node waits, 9.1 against
// 11.6 ms (31 when a ray out of words began again on the binary tree, on its lane alone;
// half of the rays closest-hit ones 127, now 10.9).
constexpr int kAnyStack = 24;

// Stack words for a tree of `levels` levels of inner nodes.
TIMRT_HD int four_words(int levels) {
    const int all = 3 * levels + 2, least = levels + 2;
    const int words = all < 6 ? 6 : (all > kAnyStack ? kAnyStack : all);
    return words < least ? least : words;
}

// Whether the slots of the node `ref` may be pushed: top is the address of the stack's top
// word, bottom that of word 0, step the distance of two words. False for every waiting
// node: kFourWaiting stands for 32 levels, and no stack has that many words.
TIMRT_HD bool four_fits(uint32_t top, uint32_t ref, uint32_t bottom, int words, uint32_t step) {
    return top + (ref >> kFourBelowShift) * step <= bottom + (uint32_t)(words - 5) * step;
}
// Below this address of the top word every node's slots fit, in trees of at most `levels`
// levels, and no node waits: one comparison tells, at most visits (four_fits at each of
// them took 0.4 to 2.2 % of a launch).
TIMRT_HD uint32_t four_near(uint32_t bottom, int words, int levels, uint32_t step) {
    const int spare = words - 5 - (levels - 1) + 1;
    return bottom + (spare > 0 ? (uint32_t)spare : 0u) * step;
}

TIMRT_HD uint32_t four_waiting(uint32_t ref, uint32_t slots) { return kFourWaiting | (ref & kFourIndexMask) << 4 | slots; }

}  // namespace timrt
