// sl_fits: stepping through a segment that ends at the largest admitted position,
// in 32 bits and by the largest step of the lists' kernels, ends; one that ends
// just below 2^32 would wrap around.
#include <cstdio>
#include <cstdlib>

#include "../../within_b200/csrc/segbook.hpp"

using namespace wgpu;

// steps that sl_sum takes from a to b, or -1 when the position wraps
static int steps(uint32_t a, uint32_t b, uint32_t step) {
    int n = 0;
    for (uint32_t q = a; q < b; q += step, ++n)
        if (q + step < q) return -1;
    return n;
}

int main() {
    uint64_t limit = 0;   // the largest admitted position count
    for (uint64_t bit = 1ull << 32; bit; bit >>= 1)
        if (sl_fits(limit + bit)) limit += bit;
    if (!sl_fits(limit) || sl_fits(limit + 1) || sl_fits(UINT32_MAX)) return std::printf("limit\n"), 1;
    for (uint32_t step = 1; step <= SL_STEP; step *= 2)
        for (uint32_t off = 1; off < 3 * SL_STEP; off += 61)
            if (steps((uint32_t)limit - off, (uint32_t)limit, step) != (int)((off + step - 1) / step))
                return std::printf("step %u offset %u\n", step, off), 1;
    if (steps(UINT32_MAX - 100, UINT32_MAX, SL_STEP) != -1) return std::printf("no wrap\n"), 1;
    std::printf("ok\n");
    return 0;
}
