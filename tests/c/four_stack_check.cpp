// Walks trees of 1 to 32 levels by the stack rule of four_stack.h, as any_advance
// (trace_any.cuh) does, with entered slots from none to all: every entered slot has to be
// visited once, in the order of a stack without end, and no word past the stack touched.
#include <cstdio>
#include <vector>
#include "four_stack.h"
using namespace timrt;

static uint64_t g_s = 88172645463325252ull;
static uint32_t rnd() {
    g_s ^= g_s << 13; g_s ^= g_s >> 7; g_s ^= g_s << 17;
    return (uint32_t)(g_s >> 32);
}

constexpr uint32_t kLeaf = 0x80000000u, kIdle = 0xFFFFFFFFu, kStep = 1024u, kBottom = 2052u;
struct Node { uint32_t ref[4], slots; };   // slots: the entered ones

// Nodes in preorder: the walk's own order does not depend on the numbering.
static uint32_t grow(std::vector<Node>& nodes, int level, int levels, int kind, uint32_t& leaf) {
    const uint32_t me = (uint32_t)nodes.size();
    nodes.push_back({});
    Node n{};
    const int spine = (int)(rnd() & 3u);
    for (int k = 0; k < 4; ++k) {
        const bool inner = level + 1 < levels && (k == spine || (nodes.size() < 3000u && rnd() % 8u < 2u));
        n.ref[k] = inner ? grow(nodes, level + 1, levels, kind, leaf) | (uint32_t)(levels - 2 - level) << kFourBelowShift
                         : kLeaf | leaf++;
    }
    n.slots = kind == 0 ? 15u : (kind == 1 ? rnd() & 15u : (rnd() | rnd()) & 15u);
    nodes[me] = n;
    return me;
}

static void plain(const std::vector<Node>& nodes, uint32_t ref, std::vector<uint32_t>& out) {
    if (ref & kLeaf) { out.push_back(ref); return; }
    const Node& n = nodes[ref & kFourIndexMask];
    for (int k = 3; k >= 0; --k)
        if (n.slots >> k & 1u) plain(nodes, n.ref[k], out);
}

int main() {
    long walks = 0, waits = 0, bad = 0;
    for (int levels = 1; levels <= 32; ++levels)
        for (int i = 0; i < 60; ++i) {
            std::vector<Node> nodes;
            uint32_t leaf = 0;
            grow(nodes, 0, levels, i % 3, leaf);
            // a launch's words are those of its deepest tree, at least this tree's own
            const int most = i & 1 ? levels : levels + (int)(rnd() % (uint32_t)(33 - levels)), words = four_words(most);
            std::vector<uint32_t> want, got, mem((size_t)words, 0xABABABABu);
            plain(nodes, (uint32_t)(levels - 1) << kFourBelowShift, want);
            const uint32_t near = four_near(kBottom, words, most, kStep);
            uint32_t top = kBottom, node = (uint32_t)(levels - 1) << kFourBelowShift;
            mem[0] = kIdle;
            auto push = [&](uint32_t v, bool keep) {   // writes above the top whether it keeps it or not
                const uint32_t k = (top - kBottom) / kStep + 1u;
                if (k >= (uint32_t)words) { ++bad; return; }
                mem[k] = v;
                if (keep) top += kStep;
            };
            auto pop = [&] { const uint32_t v = mem[(top - kBottom) / kStep]; top -= kStep; return v; };
            while (node != kIdle && !bad) {
                if (node & kLeaf) { got.push_back(node); node = pop(); continue; }
                if (node & kFourWaiting) {
                    const uint32_t slot = 31u - (uint32_t)__builtin_clz(node & 15u), rest = node & ~(1u << slot);
                    push(rest, rest & 15u);
                    node = nodes[(node >> 4) & kFourIndexMask].ref[slot];
                    continue;
                }
                const Node& n = nodes[node & kFourIndexMask];
                if (top < near || four_fits(top, node, kBottom, words, kStep)) {
                    if (!four_fits(top, node, kBottom, words, kStep)) ++bad;
                    for (int k = 0; k < 4; ++k) push(n.ref[k], n.slots >> k & 1u);
                    node = pop();
                } else {
                    ++waits;
                    if (3 * levels + 2 <= words) ++bad;   // such a tree's slots always fit
                    node = n.slots ? four_waiting(node, n.slots) : pop();
                }
            }
            ++walks;
            if (got != want || top + kStep != kBottom) ++bad;
        }
    std::printf("walks %ld bad %ld waits %s\n", walks, bad, waits > 1000 ? "many" : "few");
    return bad != 0;
}
