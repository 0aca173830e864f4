// SegBook: every position of every problem lies in exactly one short segment,
// medium segment or piece; pieces of a split segment are consecutive.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../within_b200/csrc/segbook.hpp"

using namespace wgpu;

#define CHECK(c)                                              \
    do {                                                      \
        if (!(c)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #c);       \
            std::exit(1);                                     \
        }                                                     \
    } while (0)

int main() {
    std::mt19937 rng(5);
    SegBook b;
    const uint32_t edges[] = {0, 1, SL_SHORT, SL_SHORT + 1, SL_MEDIUM, SL_MEDIUM + 1, 2 * SL_MEDIUM, 5000, 200000};
    for (int trial = 0; trial < 60; ++trial) {
        const uint32_t n = 1 + rng() % 50, kind = trial % 3;
        std::vector<uint32_t> ptr(1, rng() % 7);
        for (uint32_t s = 0; s < n; ++s)
            ptr.push_back(ptr.back() + (kind == 0 ? rng() % (SL_SHORT + 1) : kind == 1 ? edges[rng() % 9] : rng() % 3000));
        const uint32_t first = rng() % n, n_seg = n - first;
        const SLPart P = b.add(ptr.data(), first, n_seg, 1 + rng() % 900);
        std::vector<int> seen(ptr.back() + 1, 0);
        std::vector<int> segs(n, 0);
        for (uint32_t i = 0; i < P.n_short; ++i) {
            const uint32_t s = P.all_short ? P.first + i : b.short_ids[P.short_off + i];
            CHECK(ptr[s + 1] - ptr[s] <= SL_SHORT);
            ++segs[s];
            for (uint32_t q = ptr[s]; q < ptr[s + 1]; ++q) ++seen[q];
        }
        for (uint32_t i = P.medium_lo; i < P.medium_hi; ++i) {
            const uint32_t s = b.medium_ids[i], len = ptr[s + 1] - ptr[s];
            CHECK(len > SL_SHORT && len <= SL_MEDIUM);
            ++segs[s];
            for (uint32_t q = ptr[s]; q < ptr[s + 1]; ++q) ++seen[q];
        }
        for (uint32_t r = P.piece_lo; r < P.piece_hi; ++r) {
            const SLPiece& pc = b.pieces[r];
            CHECK(ptr[pc.seg + 1] - ptr[pc.seg] > SL_MEDIUM && pc.p0 < pc.p1);
            if (pc.p0 == ptr[pc.seg]) ++segs[pc.seg];
            for (uint32_t q = pc.p0; q < pc.p1; ++q) ++seen[q];
            if (pc.split < 0) {
                CHECK(pc.p0 == ptr[pc.seg] && pc.p1 == ptr[pc.seg + 1]);
            } else {
                const SLSplit& sp = b.splits[pc.split];
                CHECK(sp.r0 <= r && r <= sp.r1 && sp.r1 < P.piece_hi);
                CHECK(b.pieces[sp.r0].p0 == ptr[pc.seg] && b.pieces[sp.r1].p1 == ptr[pc.seg + 1]);
                if (r > sp.r0) CHECK(b.pieces[r - 1].p1 == pc.p0 && b.pieces[r - 1].seg == pc.seg);
            }
        }
        for (uint32_t s = 0; s < n; ++s) CHECK(segs[s] == (s >= first ? 1 : 0));
        for (uint32_t q = 0; q < ptr.back(); ++q) CHECK(seen[q] == (q >= ptr[first] ? 1 : 0));
    }
    std::printf("ok\n");
    return 0;
}
