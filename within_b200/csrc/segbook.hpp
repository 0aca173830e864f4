// segbook.hpp -- work lists of the piece engine (seglist.cuh), built once per
// segment pointer array on the host and shared by every column count.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace wgpu {

// Segments of at most this many positions are summed by one group of lanes
// each.  A longer one gives a whole warp (or several pieces) enough positions
// to have its loads in flight at once.
constexpr uint32_t SL_SHORT = 32;

struct SLPiece {
    uint32_t seg, p0, p1;   // positions [p0, p1) of segment seg
    int32_t split;          // split id when the segment has several pieces, else -1
};

struct SLSplit {
    uint32_t r0, r1;        // pieces r0..r1 (global ids), in position order
};

// One problem's share of the book: segments [first, first + n_seg).
struct SLPart {
    uint32_t first = 0;
    uint32_t n_short = 0;
    uint32_t ids_off = 0;       // entries of short_ids, unless every segment is short
    bool all_short = true;      // short segment i is first + i
    uint32_t piece_lo = 0, piece_hi = 0;
};

struct SegBook {
    std::vector<uint32_t> short_ids;
    std::vector<SLPiece> pieces;
    std::vector<SLSplit> splits;

    // Segment s of the problem spans ptr[s] .. ptr[s + 1], s in [first, first + n_seg).
    // target_warps: pieces the problem's long segments are cut into, about.
    SLPart add(const uint32_t* ptr, uint32_t first, uint32_t n_seg, uint32_t target_warps) {
        SLPart P;
        P.first = first;
        P.ids_off = (uint32_t)short_ids.size();
        P.piece_lo = (uint32_t)pieces.size();
        uint64_t long_pos = 0;
        for (uint32_t s = first; s < first + n_seg; ++s) {
            const uint32_t len = ptr[s + 1] - ptr[s];
            if (len > SL_SHORT) long_pos += len;
        }
        P.all_short = long_pos == 0;
        if (P.all_short) {
            P.n_short = n_seg;
            P.piece_hi = P.piece_lo;
            return P;
        }
        uint64_t len = (long_pos + target_warps - 1) / std::max<uint32_t>(1, target_warps);
        len = std::min<uint64_t>(4096, std::max<uint64_t>(512, (len + 127) / 128 * 128));
        for (uint32_t s = first; s < first + n_seg; ++s) {
            const uint32_t a = ptr[s], b = ptr[s + 1];
            if (b - a <= SL_SHORT) {
                short_ids.push_back(s);
                ++P.n_short;
                continue;
            }
            const uint32_t np = (uint32_t)((b - a + len - 1) / len);
            int32_t split = -1;
            if (np > 1) {
                split = (int32_t)splits.size();
                splits.push_back(SLSplit{(uint32_t)pieces.size(), (uint32_t)pieces.size() + np - 1});
            }
            for (uint32_t q = 0; q < np; ++q)
                pieces.push_back(SLPiece{s, (uint32_t)(a + q * len), (uint32_t)std::min<uint64_t>(b, a + (q + 1) * len),
                                         split});
        }
        P.piece_hi = (uint32_t)pieces.size();
        return P;
    }
};

}  // namespace wgpu
