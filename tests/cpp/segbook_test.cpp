// SegBook: every position of every problem lies in exactly one short segment,
// medium segment or piece; pieces of a split segment are consecutive.
// NarrowRounds: every row once, its entries in its lanes, aligned passes.
#include <cmath>
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
    const uint32_t lens[] = {0, 1, RP_LANES, RP_LANES + 1, 17, 45, RP_ENTRIES / 32 * RP_LANES};
    for (int trial = 0; trial < 40; ++trial) {
        const uint32_t n = trial < 3 ? trial : 1 + rng() % 700, zero = 100000;
        std::vector<uint32_t> ptr(1, rng() % 5), col, id;
        std::vector<double> val;
        for (uint32_t r = 0; r < n; ++r) {
            ptr.push_back(ptr.back() + lens[rng() % (trial % 4 == 0 ? 7 : 6)]);
            id.push_back(5000 + r);
        }
        for (uint32_t e = 0; e < ptr.back(); ++e) {
            col.push_back(rng() % 5000);
            val.push_back(1.0 + e);
        }
        NarrowRounds N;
        const uint32_t cut = n ? rng() % (n + 1) : 0;   // two rounds
        CHECK(N.add(ptr.data(), col.data(), val.data(), id.data(), 0, cut, zero));
        const size_t first_pass2 = N.pass.size();
        CHECK(N.add(ptr.data(), col.data(), val.data(), id.data(), cut, n, zero));
        CHECK(N.val.size() == N.col.size() && N.row.size() == N.slice.size() * RP_SLICE);
        std::vector<double> sum(n, 0.0), want(n, 0.0);
        std::vector<int> seen(n, 0);
        for (uint32_t r = 0; r < n; ++r)
            for (uint32_t e = ptr[r]; e < ptr[r + 1]; ++e) want[r] += val[e] * (1.0 + col[e]);
        for (size_t p = 0; p < N.pass.size(); ++p) {
            const RPass& P = N.pass[p];
            CHECK(P.n_slice >= 1 && P.n_slice <= RP_WARPS && P.n_ent <= RP_ENTRIES && P.n_ent % 32 == 0);
            CHECK(P.e0 % 32 == 0 && P.s0 % 2 == 0 && P.s0 + P.n_slice <= N.slice.size());
            for (uint32_t q = 0; q < P.n_slice; ++q) {
                const RSlice& sl = N.slice[P.s0 + q];
                CHECK(sl.first + sl.width * 32 <= P.n_ent);
                for (uint32_t l = 0; l < 32; ++l) {
                    const uint32_t row = N.row[(P.s0 + q) * RP_SLICE + l / RP_LANES];
                    if (row != zero && l % RP_LANES == 0) {
                        ++seen[row - 5000];
                        CHECK((row - 5000 < cut) == (p < first_pass2));
                    }
                    for (uint32_t j = 0; j < sl.width; ++j) {
                        const size_t at = (size_t)P.e0 + sl.first + j * 32 + l;
                        if (N.col[at] == zero) CHECK(N.val[at] == 0.0);
                        else sum[row - 5000] += N.val[at] * (1.0 + N.col[at]);
                    }
                }
            }
        }
        for (uint32_t r = 0; r < n; ++r) CHECK(seen[r] == 1 && std::abs(sum[r] - want[r]) <= 1e-12 * want[r]);
        std::vector<uint32_t> wide = {0, RP_ENTRIES / 32 * RP_LANES + 1};
        CHECK(!N.add(wide.data(), col.data(), val.data(), id.data(), 0, 1, zero));
    }
    std::printf("ok\n");
    return 0;
}
