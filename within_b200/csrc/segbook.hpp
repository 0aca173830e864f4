// segbook.hpp -- work lists of the list engine (seglist.cuh), built once per
// segment pointer array on the host and shared by every column count.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace wgpu {

// Segments of at most SL_SHORT positions are summed by one group of lanes each,
// longer ones of at most SL_MEDIUM by one warp, the rest in pieces by blocks.
// SL_SHORT: what one group of lanes sums in a few batches of loads (eight positions
// at a time, two in k_segshort).  SL_MEDIUM:
// at eight columns a warp takes eight positions per step, so 512 positions are
// eight batches of eight steps; a block would leave most of its warps idle.
constexpr uint32_t SL_SHORT = 32;
constexpr uint32_t SL_MEDIUM = 512;

// The lists' kernels step through positions in 32 bits, at most eight batches of
// a block's 256 lanes beyond a segment's end: a plan whose positions come closer
// to 2^32 would wrap around there, and stays on the tile and range engines.
constexpr uint32_t SL_STEP = 8 * 256;
constexpr bool sl_fits(uint64_t positions) { return positions + 2 * SL_STEP <= UINT32_MAX; }

struct SLPiece {
    uint32_t seg, p0, p1;   // positions [p0, p1) of segment seg
    int32_t split;          // split id when the segment has several pieces, else -1
};

struct SLSplit {
    uint32_t r0, r1;        // pieces r0..r1, in position order
};

// One problem's share of the book: segments [first, first + n_seg).
struct SLPart {
    uint32_t first = 0;
    uint32_t n_short = 0;
    uint32_t short_off = 0;                 // entries of short_ids, unless every segment is short
    bool all_short = true;                  // short segment i is first + i
    uint32_t medium_lo = 0, medium_hi = 0;  // entries of medium_ids
    uint32_t piece_lo = 0, piece_hi = 0;
};

struct SegBook {
    std::vector<uint32_t> short_ids, medium_ids;
    std::vector<SLPiece> pieces;
    std::vector<SLSplit> splits;

    // Segment s of the problem spans ptr[s] .. ptr[s + 1], s in [first, first + n_seg).
    // target_blocks: pieces the problem's long segments are cut into, about.
    SLPart add(const uint32_t* ptr, uint32_t first, uint32_t n_seg, uint32_t target_blocks) {
        SLPart P;
        P.first = first;
        P.short_off = (uint32_t)short_ids.size();
        P.medium_lo = P.medium_hi = (uint32_t)medium_ids.size();
        P.piece_lo = P.piece_hi = (uint32_t)pieces.size();
        uint64_t long_pos = 0;
        for (uint32_t s = first; s < first + n_seg; ++s) {
            const uint32_t len = ptr[s + 1] - ptr[s];
            if (len > SL_SHORT) P.all_short = false;
            if (len > SL_MEDIUM) long_pos += len;
        }
        if (P.all_short) {
            P.n_short = n_seg;
            return P;
        }
        uint64_t len = (long_pos + target_blocks - 1) / std::max<uint32_t>(1, target_blocks);
        len = std::min<uint64_t>(16384, std::max<uint64_t>(SL_MEDIUM, (len + 127) / 128 * 128));
        for (uint32_t s = first; s < first + n_seg; ++s) {
            const uint32_t a = ptr[s], b = ptr[s + 1];
            if (b - a <= SL_SHORT) {
                short_ids.push_back(s);
                ++P.n_short;
                continue;
            }
            if (b - a <= SL_MEDIUM) {
                medium_ids.push_back(s);
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
        P.medium_hi = (uint32_t)medium_ids.size();
        P.piece_hi = (uint32_t)pieces.size();
        return P;
    }
};

// Slices of the narrow rounds of a triangular solve (k_rounds, seglist.cuh).
constexpr uint32_t RP_THREADS = 992, RP_WARPS = RP_THREADS / 32;
constexpr uint32_t RP_LANES = 4;              // lanes per row
constexpr uint32_t RP_SLICE = 32 / RP_LANES;  // rows per warp
constexpr uint32_t RP_ENTRIES = 4096;         // most entries of one pass (padding counted)
constexpr uint32_t RP_STAGES = 3;

struct RPass {
    uint32_t e0, n_ent;       // entries [e0, e0 + n_ent) of val / col
    uint32_t s0, n_slice;     // slices [s0, s0 + n_slice); slice lists start at even s0
};
struct RSlice {
    uint32_t first, width;    // first entry relative to the pass, entries per lane
};

struct NarrowRounds {
    std::vector<double> val;
    std::vector<uint32_t> col, row;
    std::vector<RSlice> slice;
    std::vector<RPass> pass;

    // Appends one round: rows [lo, hi) of the factor (ptr, col, val in CSR, id[r]
    // the reduced slot of row r).  Padding entries and rows name slot `zero`.
    // false (nothing appended): a row alone is wider than a pass.
    bool add(const uint32_t* ptr, const uint32_t* c, const double* v, const uint32_t* id, uint32_t lo, uint32_t hi,
             uint32_t zero) {
        std::vector<uint32_t> order(hi - lo);
        for (uint32_t i = 0; i < hi - lo; ++i) order[i] = lo + i;
        auto len = [&](uint32_t r) { return ptr[r + 1] - ptr[r]; };
        std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return len(a) > len(b); });
        if (!order.empty() && (len(order[0]) + RP_LANES - 1) / RP_LANES * 32 > RP_ENTRIES) return false;
        for (uint32_t i = 0; i < order.size();) {
            RPass P{(uint32_t)val.size(), 0, (uint32_t)slice.size(), 0};
            while (i < order.size() && P.n_slice < RP_WARPS) {
                const uint32_t w = (len(order[i]) + RP_LANES - 1) / RP_LANES;   // the slice's longest row
                if (P.n_ent + w * 32 > RP_ENTRIES) break;
                slice.push_back(RSlice{P.n_ent, w});
                val.resize(val.size() + (size_t)w * 32, 0.0);
                col.resize(col.size() + (size_t)w * 32, zero);
                for (uint32_t q = 0; q < RP_SLICE; ++q) {
                    const bool on = i + q < order.size();
                    row.push_back(on ? id[order[i + q]] : zero);
                    for (uint32_t e = 0; on && e < len(order[i + q]); ++e) {
                        const size_t at = (size_t)P.e0 + P.n_ent + (e / RP_LANES) * 32 + q * RP_LANES + e % RP_LANES;
                        val[at] = v[ptr[order[i + q]] + e];
                        col[at] = c[ptr[order[i + q]] + e];
                    }
                }
                P.n_ent += w * 32;
                ++P.n_slice;
                i += RP_SLICE;
            }
            if (slice.size() % 2) {   // the next pass's slices start 16-byte aligned
                slice.push_back(RSlice{0, 0});
                row.insert(row.end(), RP_SLICE, zero);
            }
            pass.push_back(P);
        }
        return true;
    }
};

}  // namespace wgpu
