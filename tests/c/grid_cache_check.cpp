// Calls GridCache (csrc/grid_cache.h) for every stack size a launcher can ask for on the
// first, a middle and the last device; each size's value has to stay its own.
#include <cstdio>
#include "grid_cache.h"

static int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }

int main() {
    using namespace timrt;
    static GridCache cache;
    const int devices[] = {0, 1, 30, GridCache::kDevices - 1}, most = kWalkStack + kWalkBeside;
    int calls = 0, wrong = 0;
    for (int round = 0; round < 2; ++round)
        for (int d : devices)
            for (int depth = 0; depth <= most; ++depth) {
                device = d;
                const int want = 1 + 1000 * d + depth;
                wrong += cache.get(depth, [&](int dev) { ++calls; return dev == d ? want : -1; }) != want;
            }
    // every size computed once; a size beyond them is computed, not kept
    wrong += calls != 4 * (most + 1);
    wrong += cache.get(most + 1, [](int) { return 7; }) != 7 || cache.get(most + 1, [](int) { return 8; }) != 8;
    std::printf("sizes %d wrong %d\n", most + 1, wrong);
    return wrong != 0;
}
