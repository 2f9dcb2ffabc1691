// Host check of the index arithmetic of grids with a warp per item: the item
// numbers at and beyond 2^27, where the thread's own number passes 32 bits;
// of the stroker's slots per node and lane, from 2^28 nodes on; and of the
// chunks of a row of up to 2^31 - 1 pixels.
#include <cstdint>
#include <cstdio>

#include "fill.cuh"
#include "stroke_gpu.cuh"

using namespace z2dg;

int main() {
    long long wrong = 0;
    for (uint32_t threads : {128u, 256u})
        for (long long item : {0ll, 1ll, (1ll << 27) - 1, 1ll << 27, (1ll << 27) + 5, 1ll << 30, (1ll << 31) - 1}) {
            const uint32_t per = threads / 32;
            const uint32_t block = (uint32_t)(item / per), first = (uint32_t)(item % per) * 32;
            for (uint32_t lane : {0u, 31u}) wrong += warp_number(block, threads, first + lane) != item;
        }
    for (int g : {0, 3, 5})
        for (int32_t node : {0, 1, (1 << 26) - 1, 1 << 28, (1 << 28) + 3, 0x7FFFFFFF})
            wrong += lane_slot(node, g) != (long long)node * (1 << g);
    for (int32_t n : {1, 127, 128, 129, 0x7FFFFFFF - 128, 0x7FFFFFFF - 127, 0x7FFFFFFF})
        wrong += row_chunks(n, 128) != (int32_t)(((long long)n + 127) / 128);
    printf("wrong %lld\n", wrong);
    return wrong ? 1 : 0;
}
