// 4,096 calls in a row, from any call on (the count wraps), have words of their own.
#include <cstdio>
#include <vector>
#include "counter_ring.h"

int main() {
    int bad = 0;
    for (uint32_t start : {0u, 1u, 2047u, 4095u, 123456u, 0xFFFFF000u, 0xFFFFFFFFu}) {
        std::vector<int> taken(timrt::kRingWords, 0);
        for (uint32_t k = 0; k < 4096u; ++k)
            for (uint32_t w = 0; w < 2u; ++w) {
                const uint32_t at = timrt::ring_word(start + k) + w;
                if (at >= timrt::kRingWords || taken[at]++) ++bad;
            }
    }
    std::printf("bad %d\n", bad);
    return bad != 0;
}
