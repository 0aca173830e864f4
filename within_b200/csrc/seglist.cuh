// seglist.cuh -- the list engine: deterministic segmented reduction from work
// lists of short, medium and long segments (segbook.hpp), the default for every
// FP64 plan of the Schwarz apply and of the adjoint's rest.
//
// What bounds the sums: 12 bytes of index and value per non-zero and one
// gathered operand.  The scan engines (segreduce.cuh, segsweep.cuh) find segment
// boundaries inside a tile of mixed segments, which costs tens of instructions
// per position in scans, shuffles and barriers.  Knowing each segment's length
// beforehand, no scan is needed:
//   - a short segment (at most SL_SHORT positions) is summed in position order
//     by one group of lanes;
//   - a medium one (at most SL_MEDIUM) by one warp, whose lanes stride over it
//     and end in one shuffle tree;
//   - a long one in pieces, one block each; the last block to arrive (an atomic
//     counter, not a wait) adds the pieces' partials.
// What is left is latency: index, then operand, then the emit's own loads.  So
// every lane takes SL_BATCH positions at a time, all indices before any operand
// (positions past the end re-read the last one and add zero), and a segment's
// emit loads are requested before its sum.  The K columns of a position lie
// across K / 2 lanes (two columns per lane, one 16-byte access).  Every sum has
// one fixed order: results are bitwise reproducible, with no floating-point
// atomics.
//
// 10,000,000-row panel, one column, against the scan engines: C^T 80 -> 49 us,
// restrict 26 -> 15, means 22 -> 12.5, kept sums 11 -> 6, the run combine 25 ->
// 21; eight columns: C^T 498 -> 116 us, restrict 148 -> 52, means 114 -> 44, run
// combine 138 -> 51.  With four loads per lane requested at once C^T took 64 us
// and eight-column restrict 150 us (there mostly the one warp that added the
// 1700 partials of a segment cut for warps, hence pieces for blocks).
#pragma once
#include "pdl.cuh"
#include <cstdint>

#include "bulk.cuh"
#include "kernels.cuh"
#include "segbook.hpp"

namespace wgpu {

constexpr int SL_THREADS = 256;
constexpr int SL_WARPS = SL_THREADS / 32;
constexpr int SL_BATCH = 8;
static_assert(SL_BATCH * SL_THREADS <= (int)SL_STEP, "a step past the end stays below the wrap");

// device view of one problem's lists; blocks [0, pieces) take the pieces, then
// the medium segments (one warp each), then the short ones
struct SLDev {
    const uint32_t* ptr;          // segment pointers
    const uint32_t* short_ids;
    const uint32_t* medium_ids;
    uint32_t n_short, n_medium, n_piece, medium_blocks;
    const SLPiece* pieces;        // of this problem
    uint32_t piece_lo;            // its first piece's id
    const SLSplit* splits;
    double* part;                 // K per piece
    unsigned* counters;           // one per split
};

// F provides (W = fl_w<K>() columns from column c0):
//   struct Ctx; Ctx ctx(uint32_t seg) const;       what every position of a segment shares
//   struct Idx; Idx index(uint32_t pos) const;     a position's index and factor
//   V value(const Ctx&, uint32_t pos, const Idx&, int c0, bool valid) const;
//   struct Pre; Pre pre(uint32_t seg, int c0) const;   what emit reads
//   void emit(uint32_t seg, int c0, const Pre&, const V& s) const;
// PF: the next batch's indices are requested before this batch's operands.
template <class F, int K, int NB, bool PF>
__device__ __forceinline__ FlVec<fl_w<K>()> sl_sum(const F& f, const typename F::Ctx& cx, uint32_t a, uint32_t b,
                                                   uint32_t stride, int c0) {
    constexpr int W = fl_w<K>();
    FlVec<W> s;
#pragma unroll
    for (int i = 0; i < W; ++i) s.q[i] = 0.0;
    if constexpr (PF) {
        if (a >= b) return s;
        typename F::Idx ix[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) ix[j] = f.index(min(a + j * stride, b - 1));
        for (uint32_t q = a; q < b; q += NB * stride) {
            typename F::Idx nx[NB];   // the next batch's indices, requested before this one's operands
#pragma unroll
            for (int j = 0; j < NB; ++j) nx[j] = f.index(min(q + (NB + j) * stride, b - 1));
            FlVec<W> v[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) v[j] = f.value(cx, min(q + j * stride, b - 1), ix[j], c0, q + j * stride < b);
#pragma unroll
            for (int j = 0; j < NB; ++j)
#pragma unroll
                for (int i = 0; i < W; ++i) s.q[i] += q + j * stride < b ? v[j].q[i] : 0.0;
#pragma unroll
            for (int j = 0; j < NB; ++j) ix[j] = nx[j];
        }
    } else {
        for (uint32_t q = a; q < b; q += NB * stride) {
            typename F::Idx ix[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) ix[j] = f.index(min(q + j * stride, b - 1));
            FlVec<W> v[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) v[j] = f.value(cx, min(q + j * stride, b - 1), ix[j], c0, q + j * stride < b);
#pragma unroll
            for (int j = 0; j < NB; ++j)
#pragma unroll
                for (int i = 0; i < W; ++i) s.q[i] += q + j * stride < b ? v[j].q[i] : 0.0;
        }
    }
    return s;
}

// Block `block` of one problem.  LISTED: the short segments are those of
// short_ids; else every short segment i is segment first + i.
template <class F, int K, bool LISTED>
__device__ __forceinline__ void seglist_block(const F& f, const SLDev& L, uint32_t block, uint32_t first) {
    constexpr int W = fl_w<K>(), P = fl_per_row<K>(), S = 32 / P;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g = lane / P, c0 = (lane % P) * W;
    auto tree = [&](FlVec<W>& s) {
#pragma unroll
        for (int o = P; o < 32; o <<= 1)
#pragma unroll
            for (int i = 0; i < W; ++i) s.q[i] += __shfl_xor_sync(FULL, s.q[i], o);
    };
    if (block >= L.n_piece + L.medium_blocks) {   // short segments
        const uint32_t t = (block - L.n_piece - L.medium_blocks) * SL_THREADS + threadIdx.x;
        const uint32_t i = t / P;
        if (i >= L.n_short) return;
        const uint32_t seg = LISTED || L.short_ids ? __ldg(L.short_ids + i) : first + i;
        const uint32_t a = __ldg(L.ptr + seg), b = __ldg(L.ptr + seg + 1);
        const typename F::Pre pre = f.pre(seg, c0);
        f.emit(seg, c0, pre, sl_sum<F, K, F::BATCH, false>(f, f.ctx(seg), a, b, 1, c0));
        return;
    }
    if (block >= L.n_piece) {   // medium segments
        const uint32_t i = (block - L.n_piece) * SL_WARPS + wid;
        if (i >= L.n_medium) return;   // whole warps
        const uint32_t seg = __ldg(L.medium_ids + i);
        const uint32_t a = __ldg(L.ptr + seg), b = __ldg(L.ptr + seg + 1);
        const typename F::Pre pre = f.pre(seg, c0);
        FlVec<W> s = sl_sum<F, K, F::BATCH, F::PREFETCH>(f, f.ctx(seg), a + g, b, S, c0);
        tree(s);
        if (lane < P) f.emit(seg, c0, pre, s);
        return;
    }
    __shared__ __align__(16) double sm[SL_WARPS][K];
    __shared__ int last;
    const SLPiece pc = L.pieces[block];
    FlVec<W> s = sl_sum<F, K, F::BATCH, F::PREFETCH>(f, f.ctx(pc.seg), pc.p0 + wid * S + g, pc.p1, SL_WARPS * S, c0);
    tree(s);
    if (lane < P) fl_st<W>(&sm[wid][c0], s);
    __syncthreads();
    if (pc.split >= 0) {
        const SLSplit sp = L.splits[pc.split];
        if (threadIdx.x < K) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < SL_WARPS; ++w) t += sm[w][threadIdx.x];
            L.part[(size_t)(L.piece_lo + block) * K + threadIdx.x] = t;
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(&L.counters[pc.split], 1u) == sp.r1 - sp.r0 ? 1 : 0;
        __syncthreads();
        if (!last) return;
        __threadfence();
#pragma unroll
        for (int i = 0; i < W; ++i) s.q[i] = 0.0;
        for (uint32_t q = sp.r0 + wid * S + g; q <= sp.r1; q += SL_WARPS * S)
#pragma unroll
            for (int i = 0; i < W; ++i) s.q[i] += __ldcg(L.part + (size_t)q * K + c0 + i);
        tree(s);
        if (lane < P) fl_st<W>(&sm[wid][c0], s);
        if (threadIdx.x == 0) L.counters[pc.split] = 0;
        __syncthreads();
    }
    if (wid == 0 && lane < P) {
#pragma unroll
        for (int i = 0; i < W; ++i) {
            s.q[i] = 0.0;
#pragma unroll
            for (int w = 0; w < SL_WARPS; ++w) s.q[i] += sm[w][c0 + i];
        }
        f.emit(pc.seg, c0, f.pre(pc.seg, c0), s);
    }
}

template <class F, int K>
__device__ __forceinline__ void seglist_body(const F& f, const SLDev& L, const int* __restrict__ skip) {
    pdl_wait();
    pdl_launch_dependents();
    if (skip && *skip) return;
    seglist_block<F, K, true>(f, L, blockIdx.x, 0);
}

template <class F, int K>
__global__ void __launch_bounds__(SL_THREADS)
k_seglist(F f, SLDev L, const int* __restrict__ skip) {
    seglist_body<F, K>(f, L, skip);
}
// the same held to 32 registers, eight blocks per SM (F::FULL)
template <class F, int K>
__global__ void __launch_bounds__(SL_THREADS, 8)
k_seglist_full(F f, SLDev L, const int* __restrict__ skip) {
    seglist_body<F, K>(f, L, skip);
}

// Every segment short (the rows of C, the prolongation, most rounds): one group
// of lanes per segment, in position order.  Nothing but resident warps hides the
// two or three dependent loads of so little work, so the kernel is held to 32
// registers (eight blocks per SM) and asks for two positions at a time: C of the
// 10,000,000-row panel (10.4 M non-zeros in rows of about five) takes 62 us with
// one column and 146 to 152 us over runs with eight; 236 us with eight positions at a time in 64
// registers, 183 us with four in 40, 66 us (one column) with the values of a
// warp's segments staged in shared memory.
constexpr int SL_SHORT_BATCH = 2;

template <class F, int K>
__global__ void __launch_bounds__(SL_THREADS, 8)
k_segshort(F f, const uint32_t* __restrict__ ptr, uint32_t first, uint32_t n_seg, const int* __restrict__ skip) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int W = fl_w<K>(), P = fl_per_row<K>();
    if (skip && *skip) return;
    const uint32_t t = blockIdx.x * SL_THREADS + threadIdx.x;
    const uint32_t i = t / P;
    const int c0 = (int)(t % P) * W;
    if (i >= n_seg) return;
    const uint32_t seg = first + i;
    const uint32_t a = __ldg(ptr + seg), b = __ldg(ptr + seg + 1);
    const typename F::Pre pre = f.pre(seg, c0);
    f.emit(seg, c0, pre, sl_sum<F, K, SL_SHORT_BATCH, false>(f, f.ctx(seg), a, b, 1, c0));
}

// ---------------------------------------------------------------------------
// The steps of the Schwarz apply and the adjoint's rest on this engine; the
// sums are those of the functors of the same name in kernels.cuh, FP64.
template <int K>
struct SlBase {
    // medium and long segments: positions a lane requests at once, whether the
    // next batch's indices come before this batch's operands, and whether the
    // kernel is held to eight blocks per SM.  With indices ahead C^T
    // went from 126 to 116 us at eight columns and from 27 to 22 at four, the
    // forward rounds from 40 to 17 and from 14 to 9.
    static constexpr int BATCH = SL_BATCH;
    static constexpr bool PREFETCH = true, FULL = false;
    static constexpr int W = fl_w<K>();
    using V = FlVec<W>;
    struct Ctx {};
    struct Idx {
        uint32_t i;
        double f;
    };
    SchwarzDev S;
    __device__ Ctx ctx(uint32_t) const { return {}; }
    static __device__ __forceinline__ V scaled(const V& a, double f) {
        V r;
#pragma unroll
        for (int i = 0; i < W; ++i) r.q[i] = a.q[i] * f;
        return r;
    }
    static __device__ __forceinline__ V ld(const double* p, size_t row, int c0) { return fl_ld<W>(p + row * K + c0); }
    static __device__ __forceinline__ void st(double* p, size_t row, int c0, const V& v) {
        fl_st<W>(p + row * K + c0, v);
    }
    // solution of kept index (reduced slot u of subdomain s) after the gauge / cover read-back
    __device__ __forceinline__ V kept(uint32_t u, uint32_t s, int m, int c0) const {
        V o = ld(S.xv, u, c0);
        if (m != 0) {
            const V q = ld(S.xv, m == 1 ? S.red_off[s] + S.n_kept[s] : u + S.n_kept[s], c0);
#pragma unroll
            for (int i = 0; i < W; ++i) o.q[i] = m == 1 ? o.q[i] - q.q[i] : 0.5 * (o.q[i] - q.q[i]);
        }
        return o;
    }
    __device__ __forceinline__ V reduced(uint32_t u, int c0) const {
        const uint32_t s = S.red_sub[u];
        V b = ld(S.rb, u, c0);
        const V m = ld(S.m2, s, c0);
#pragma unroll
        for (int i = 0; i < W; ++i) b.q[i] -= m.q[i];
        return b;
    }
    // mean of a floating subdomain's sum, 0 for the others
    struct MeanPre {
        double inv;   // 0: not floating
    };
    __device__ __forceinline__ MeanPre mean_pre(uint32_t sub) const {
        return MeanPre{S.mode[sub] == 0 ? 1.0 / (double)(S.loc_ptr[sub + 1] - S.loc_ptr[sub]) : 0.0};
    }
    static __device__ __forceinline__ V mean(const MeanPre& p, const V& s) {
        V o;
#pragma unroll
        for (int i = 0; i < W; ++i) o.q[i] = p.inv != 0.0 ? s.q[i] * p.inv : 0.0;
        return o;
    }
};

#define SL_TYPES                     \
    using B = SlBase<K>;             \
    using V = typename B::V;         \
    using Idx = typename B::Idx;     \
    using B::S

template <int K>
struct SlRestrict : SlBase<K> {
    // it streams: resident warps are worth more than loads per lane (71 -> 52 us at
    // eight columns, 14 -> 10 at four), and than the few registers that spill for
    // it at four and eight columns (24 bytes of stack)
    static constexpr int BATCH = 4;
    static constexpr bool PREFETCH = false, FULL = true;
    SL_TYPES;
    using Ctx = typename B::Ctx;
    using Pre = typename B::MeanPre;
    const double* r;
    __device__ Idx index(uint32_t j) const { return {__ldg(S.glob + j), __ldg(S.scale + j)}; }
    __device__ V value(const Ctx&, uint32_t j, const Idx& x, int c0, bool valid) const {
        const V v = B::scaled(B::ld(r, x.i, c0), x.f);
        if (valid) B::st(S.rl, j, c0, v);
        return v;
    }
    __device__ Pre pre(uint32_t sub, int) const { return this->mean_pre(sub); }
    __device__ void emit(uint32_t sub, int c0, const Pre& p, const V& s) const { B::st(S.m1, sub, c0, B::mean(p, s)); }
};

template <int K>
struct SlCt : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        uint32_t red, cover;   // cover: reduced slot of the negated copy, ~0 = none
        double rsum;
        V m, rl;
    };
    __device__ Idx index(uint32_t a) const { return {__ldg(S.ct_col + a), __ldg(S.ct_val + a)}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        return B::scaled(B::ld(S.rl, x.i, c0), x.f);
    }
    __device__ Pre pre(uint32_t row, int c0) const {
        const uint32_t slot = S.ct_row_slot[row], sub = S.slot_sub[slot], red = S.ct_row_red[row];
        return Pre{red, S.mode[sub] == 2 ? red + S.n_kept[sub] : 0xffffffffu, S.ct_rowsum[row], B::ld(S.m1, sub, c0),
                   B::ld(S.rl, slot, c0)};
    }
    __device__ void emit(uint32_t, int c0, const Pre& p, const V& s) const {
        V val, neg;
#pragma unroll
        for (int i = 0; i < B::W; ++i) {
            val.q[i] = (p.rl.q[i] - p.m.q[i]) + (s.q[i] - p.m.q[i] * p.rsum);
            neg.q[i] = -val.q[i];
        }
        B::st(S.rb, p.red, c0, val);
        if (p.cover != 0xffffffffu) B::st(S.rb, p.cover, c0, neg);
    }
};

template <int K>
struct SlKeptSum : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        int mode;
        double rn;
        uint32_t ground;
    };
    __device__ Idx index(uint32_t q) const { return {__ldg(S.ct_row_red + q), 1.0}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const { return B::ld(S.rb, x.i, c0); }
    __device__ Pre pre(uint32_t sub, int) const {
        return Pre{S.mode[sub], (double)S.red_n[sub], S.red_off[sub] + S.n_kept[sub]};
    }
    __device__ void emit(uint32_t sub, int c0, const Pre& p, const V& s) const {
        V o, neg;
#pragma unroll
        for (int i = 0; i < B::W; ++i) {
            o.q[i] = p.mode == 0 ? s.q[i] / p.rn : 0.0;
            neg.q[i] = -s.q[i];
        }
        if (p.mode == 1) B::st(S.rb, p.ground, c0, neg);
        B::st(S.m2, sub, c0, o);
    }
};

template <int K>
struct SlDense : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        uint32_t u;
    };
    __device__ Idx index(uint32_t a) const { return {__ldg(S.dense_col + a), __ldg(S.dense_val + a)}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        return B::scaled(this->reduced(x.i, c0), x.f);
    }
    __device__ Pre pre(uint32_t row, int) const { return Pre{S.dense_row_slot[row]}; }
    __device__ void emit(uint32_t, int c0, const Pre& p, const V& s) const { B::st(S.xv, p.u, c0, s); }
};

template <int K>
struct SlFwd : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        uint32_t u;
        double di;
        V b;
    };
    __device__ Idx index(uint32_t a) const { return {__ldg(S.fwd_col + a), __ldg(S.fwd_val + a)}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        return B::scaled(B::ld(S.yv, x.i, c0), x.f);
    }
    __device__ Pre pre(uint32_t row, int c0) const {
        const uint32_t u = S.fwd_row[row];
        return Pre{u, S.dinv[u], this->reduced(u, c0)};
    }
    __device__ void emit(uint32_t, int c0, const Pre& p, const V& s) const {
        V y, x;
#pragma unroll
        for (int i = 0; i < B::W; ++i) {
            y.q[i] = p.b.q[i] - s.q[i];
            x.q[i] = y.q[i] * p.di;
        }
        B::st(S.yv, p.u, c0, y);
        B::st(S.xv, p.u, c0, x);
    }
};

template <int K>
struct SlCore : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        uint32_t u;
    };
    __device__ Idx index(uint32_t a) const { return {__ldg(S.core_col + a), __ldg(S.core_val + a)}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        return B::scaled(B::ld(S.yv, x.i, c0), x.f);
    }
    __device__ Pre pre(uint32_t row, int) const { return Pre{S.core_row_slot[row]}; }
    __device__ void emit(uint32_t, int c0, const Pre& p, const V& s) const { B::st(S.xv, p.u, c0, s); }
};

template <int K>
struct SlBwd : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        uint32_t v;
        V x;
    };
    __device__ Idx index(uint32_t a) const { return {__ldg(S.bwd_col + a), __ldg(S.bwd_val + a)}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        return B::scaled(B::ld(S.xv, x.i, c0), x.f);
    }
    __device__ Pre pre(uint32_t row, int c0) const {
        const uint32_t v = S.bwd_row[row];
        return Pre{v, B::ld(S.xv, v, c0)};
    }
    __device__ void emit(uint32_t, int c0, const Pre& p, const V& s) const {
        V x;
#pragma unroll
        for (int i = 0; i < B::W; ++i) x.q[i] = p.x.q[i] - s.q[i];
        B::st(S.xv, p.v, c0, x);
    }
};

template <int K>
struct SlC : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {
        uint32_t e;
        V first;   // D_e^-1 (rhs - mean)
    };
    __device__ Idx index(uint32_t a) const { return {__ldg(S.c_col + a), __ldg(S.c_val + a)}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        if (!(x.i & 0x80000000u)) return B::scaled(B::ld(S.xv, x.i, c0), x.f);
        const uint32_t u = x.i & 0x7fffffffu, s = S.red_sub[u];
        return B::scaled(this->kept(u, s, S.mode[s], c0), x.f);
    }
    __device__ Pre pre(uint32_t row, int c0) const {
        const uint32_t e = S.elim_slot[row], sub = S.slot_sub[e];
        const double ie = S.inv_e[e];
        const V rl = B::ld(S.rl, e, c0), m = B::ld(S.m1, sub, c0);
        Pre p{e, {}};
#pragma unroll
        for (int i = 0; i < B::W; ++i) p.first.q[i] = (rl.q[i] - m.q[i]) * ie;
        return p;
    }
    __device__ void emit(uint32_t, int c0, const Pre& p, const V& s) const {
        V o;
#pragma unroll
        for (int i = 0; i < B::W; ++i) o.q[i] = p.first.q[i] + s.q[i];
        B::st(S.sl, p.e, c0, o);
    }
};

template <int K>
struct SlMean : SlBase<K> {
    static constexpr bool PREFETCH = false;
    SL_TYPES;
    using Pre = typename B::MeanPre;
    struct Ctx {
        uint32_t sub, elim_end, red0;   // slots below elim_end are eliminated; red0 + j is kept slot j's reduced slot
        int mode;
    };
    __device__ Ctx ctx(uint32_t s) const {
        const uint32_t e = S.loc_ptr[s] + S.n_elim[s];
        return Ctx{s, e, S.red_off[s] - e, S.mode[s]};
    }
    __device__ Idx index(uint32_t j) const { return {j, 1.0}; }
    __device__ V value(const Ctx& cx, uint32_t j, const Idx&, int c0, bool valid) const {
        if (j < cx.elim_end) return B::ld(S.sl, j, c0);
        const V v = this->kept(cx.red0 + j, cx.sub, cx.mode, c0);
        if (valid) B::st(S.sl, j, c0, v);
        return v;
    }
    __device__ Pre pre(uint32_t sub, int) const { return this->mean_pre(sub); }
    __device__ void emit(uint32_t sub, int c0, const Pre& p, const V& s) const { B::st(S.m3, sub, c0, B::mean(p, s)); }
};

template <int K>
struct SlProlong : SlBase<K> {
    SL_TYPES;
    using Ctx = typename B::Ctx;
    struct Pre {};
    double* z;
    __device__ Idx index(uint32_t a) const { return {__ldg(S.dof_slot + a), 1.0}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        const uint32_t s = __ldg(S.slot_sub + x.i);
        const double sc = __ldg(S.scale + x.i);
        V v = B::ld(S.sl, x.i, c0);
        const V m = B::ld(S.m3, s, c0);
#pragma unroll
        for (int i = 0; i < B::W; ++i) v.q[i] = sc * (v.q[i] - m.q[i]);
        return v;
    }
    __device__ Pre pre(uint32_t, int) const { return {}; }
    __device__ void emit(uint32_t dof, int c0, const Pre&, const V& s) const { B::st(z, dof, c0, s); }
};
#undef SL_TYPES

// ---------------------------------------------------------------------------
// The narrow rounds of the factor's triangular solves in one launch per
// direction: one block per column keeps that column's reduced vector in shared
// memory and walks the rounds, one block barrier per pass.  A round of a few
// hundred rows of ten entries is 2 us of latency (index, operand, emit, each
// from L2) and 2 us of launch for 20 ns of traffic; here the entries are copied
// into shared memory RP_STAGES - 1 passes ahead, right-hand sides are formed
// before the first pass and results written after the last, so a pass touches
// shared memory only.  What bounds it then is the one SM's issue rate, so the
// host packs the rows into slices (NarrowRounds, segbook.hpp): the rows of a
// round sorted by length, RP_SLICE rows per warp, RP_LANES lanes per row, padded
// to the slice's longest row -- no row pointers, no bounds, conflict-free reads
// of index and value.  33 rounds of a factor of 4,368 vertices and 47,000 entries
// (1,000,000-row design with a 4,348-level factor), per direction: 200 us as
// launches, 40 us forward and 32 us backward here (0.9 us per pass: barrier,
// index, operand, sum and write-back in sequence).  Reading the rows' entries
// from L2 one pass ahead took 56 us, copying them with every thread 50 us.
struct RStage {
    double val[RP_ENTRIES];
    uint32_t col[RP_ENTRIES];
    uint32_t row[RP_WARPS * RP_SLICE];
    uint2 slice[RP_WARPS + RP_WARPS % 2];   // copied in pairs
};
static_assert(sizeof(RStage) % 16 == 0 && RP_WARPS * 32 == RP_THREADS, "16-byte aligned stages, one slice per warp");

// device arrays of a NarrowRounds
struct RDev {
    const double* val;
    const uint32_t *col, *row;
    const uint2* slice;
    const RPass* pass;
    uint32_t n_pass;
};

// BACKWARD false: y_u = b_u - sum L[u, v] y_v and z_u = y_u / d_u for the factor
// rows [row_lo, row_hi) (the y of earlier rows from memory);
// true: x_v = z_v - sum L[u, v] x_u.
template <int K, bool BACKWARD>
__global__ void __launch_bounds__(RP_THREADS + 32)
k_rounds(SchwarzDev S, RDev R, uint32_t row_lo, uint32_t row_hi, uint32_t n_red, int* err,
         const int* __restrict__ skip) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char rp_smem[];
    if (skip && *skip) return;
    const int k = blockIdx.x;   // this block's column
    const unsigned FULL = 0xffffffffu;
    const uint32_t tid = threadIdx.x, wid = tid >> 5, lane = tid & 31u;
    const uint32_t* __restrict__ rows = BACKWARD ? S.bwd_row : S.fwd_row;
    RStage* stage = reinterpret_cast<RStage*>(rp_smem);
    RPass* pass = reinterpret_cast<RPass*>(rp_smem + RP_STAGES * sizeof(RStage));
    double* vec = reinterpret_cast<double*>(pass + R.n_pass);   // n_red values and a zero for the padding
    __shared__ __align__(8) uint64_t bar[RP_STAGES];
    // an earlier wait that has timed out: this launch's result is not used, and its waits
    // would run out as well (looked at with the first pass: at the start it cost 0.6 us)
    const int earlier = tid == 0 ? *(const volatile int*)err : 0;
    for (uint32_t i = tid; i < R.n_pass; i += RP_THREADS + 32) pass[i] = R.pass[i];
    if (tid == 0) {
        for (uint32_t i = 0; i < RP_STAGES; ++i) mbar_init(&bar[i], 1);
        fence_mbar_init();
    }
    __syncthreads();
    // the last warp's first lane has the passes copied (sizes are multiples of 16 bytes), the others sum
    const bool copies = tid == RP_THREADS;
    auto issue = [&](uint32_t p) {
        if (p >= R.n_pass) return;
        const RPass q = pass[p];
        RStage& G = stage[p % RP_STAGES];
        uint64_t* bp = &bar[p % RP_STAGES];
        const uint32_t sb = (q.n_slice + 1) / 2 * 16, rb = q.n_slice * RP_SLICE * 4;
        mbar_arrive_expect_tx(bp, q.n_ent * 12 + sb + rb);
        if (q.n_ent) {
            bulk_g2s(G.val, R.val + q.e0, q.n_ent * 8, bp);
            bulk_g2s(G.col, R.col + q.e0, q.n_ent * 4, bp);
        }
        bulk_g2s(G.row, R.row + q.s0 * RP_SLICE, rb, bp);
        bulk_g2s(G.slice, R.slice + q.s0, sb, bp);
    };
    if (copies)
        for (uint32_t i = 0; i + 1 < RP_STAGES; ++i) issue(i);
    // the column's values, eight per thread in flight
    for (uint32_t u0 = tid; wid < RP_WARPS && u0 < n_red; u0 += 8 * RP_THREADS) {
        double x[8];
        uint32_t sub[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t u = min(u0 + j * RP_THREADS, n_red - 1);
            x[j] = (BACKWARD ? S.xv : S.rb)[(size_t)u * K + k];
            sub[j] = BACKWARD ? 0u : __ldg(S.red_sub + u);
        }
        if constexpr (!BACKWARD) {
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] -= S.m2[(size_t)sub[j] * K + k];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (u0 + j * RP_THREADS < n_red) vec[u0 + j * RP_THREADS] = x[j];
    }
    if (tid == 0) vec[n_red] = 0.0;
    if (!BACKWARD && row_lo > 0) {   // rounds that ran as launches of their own
        __syncthreads();
        for (uint32_t r = tid; wid < RP_WARPS && r < row_lo; r += RP_THREADS) {
            const uint32_t u = __ldg(rows + r);
            vec[u] = S.yv[(size_t)u * K + k];
        }
    }
    bool failed = false;
    uint32_t p = 0;
    for (; p < R.n_pass; ++p) {
        const bool landed = mbar_wait_bounded(&bar[p % RP_STAGES], (p / RP_STAGES) & 1u);
        // pass p's copies and the previous pass's sums are visible to every thread
        if (__syncthreads_or(!landed || earlier != 0)) {
            failed = true;
            break;
        }
        if (copies) {   // into the stage of pass p - 1, which every warp has left
            fence_proxy_async_smem();
            issue(p + RP_STAGES - 1);
        }
        if (wid == RP_WARPS) continue;
        if (wid >= pass[p].n_slice) continue;   // whole warps
        const RStage& G = stage[p % RP_STAGES];
        const uint2 sl = G.slice[wid];   // first entry in the pass, entries per lane
        const uint32_t row = G.row[wid * RP_SLICE + lane / RP_LANES];   // padding rows: the zero
        const double* gv = G.val + sl.x + lane;
        const uint32_t* gc = G.col + sl.x + lane;
        double s = 0.0;
        for (uint32_t j0 = 0; j0 < sl.y; j0 += 4) {
            double v[4], x[4];
            uint32_t c[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {   // past the width: the last entry again, not added
                const uint32_t i = min(j0 + j, sl.y - 1) * 32;
                c[j] = gc[i];
                v[j] = gv[i];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = vec[c[j]];
#pragma unroll
            for (int j = 0; j < 4; ++j) s += j0 + j < sl.y ? v[j] * x[j] : 0.0;
        }
#pragma unroll
        for (int o = 1; o < (int)RP_LANES; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane % RP_LANES == 0) vec[row] -= s;
    }
    if (failed) {   // record it, then wait (bounded) for the copies still in flight
        if (tid == 0) atomicExch(err, ERR_WAIT_TIMEOUT);
        for (uint32_t q = p; q < R.n_pass && q + 1 < p + RP_STAGES; ++q)
            (void)mbar_wait_bounded(&bar[q % RP_STAGES], (q / RP_STAGES) & 1u);
        return;
    }
    __syncthreads();
    if (wid == RP_WARPS) return;
    for (uint32_t r0 = row_lo + tid; r0 < row_hi; r0 += 8 * RP_THREADS) {
        uint32_t u[8];
        double di[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] = __ldg(rows + min(r0 + j * RP_THREADS, row_hi - 1));
        if constexpr (!BACKWARD) {
#pragma unroll
            for (int j = 0; j < 8; ++j) di[j] = __ldg(S.dinv + u[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (r0 + j * RP_THREADS >= row_hi) continue;
            const double y = vec[u[j]];
            if constexpr (BACKWARD) {
                S.xv[(size_t)u[j] * K + k] = y;
            } else {
                S.yv[(size_t)u[j] * K + k] = y;
                S.xv[(size_t)u[j] * K + k] = y * di[j];
            }
        }
    }
}

// one (term, column) problem of A^T u: run sums by run ordinal, or the rows
// of the term's level-sorted order
template <int K>
struct SlScatter {
    static constexpr int BATCH = SL_BATCH;
    static constexpr bool PREFETCH = true, FULL = false;
    static constexpr int W = fl_w<K>();
    using V = FlVec<W>;
    struct Ctx {};
    struct Idx {
        uint32_t i;
    };
    struct Pre {};
    ScatterProb pr;
    const double* u;
    const double* sqrt_w;
    double* out;
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ Idx index(uint32_t pos) const { return {pr.order ? __ldg(pr.order + pos) : pos}; }
    __device__ V value(const Ctx&, uint32_t, const Idx& x, int c0, bool) const {
        if (pr.run_sum) return fl_ld<W>(pr.run_sum + ((size_t)x.i * pr.ncol + pr.col) * K + c0);
        double f = pr.load ? __ldg(pr.load + x.i) : 1.0;
        if (sqrt_w) f *= __ldg(sqrt_w + x.i);
        V v = fl_ld<W>(u + (size_t)x.i * K + c0);
#pragma unroll
        for (int k = 0; k < W; ++k) v.q[k] *= f;
        return v;
    }
    __device__ Pre pre(uint32_t, int) const { return {}; }
    __device__ void emit(uint32_t seg, int c0, const Pre&, const V& s) const {
        fl_st<W>(out + ((size_t)pr.out_off + seg) * K + c0, s);
    }
};

// Several problems of A^T u in one launch: a design of many terms has one per
// term and column, most of them a few microseconds of work, and a launch each
// cost more than the sums: solves of one column with eight terms of 2,000 levels on
// 20,000 rows 1.67 -> 0.74 ms (20 iterations), with eight terms of 300 levels on
// 1,000,000 rows 0.99 -> 0.75 ms (6 iterations).  A block finds its problem by its
// index; the sums are those of a launch each, to the bit.
constexpr int SL_GROUP = 8;   // problems of one launch: about 1.3 KB of kernel parameters
// A problem of short segments only that fills the GPU on its own keeps its own
// launch of k_segshort, whose blocks are eight per SM: eight terms of 100,000 levels
// on 1,000,000 rows, 20 iterations, four columns (782 blocks each) 5.46 ms alone and
// 5.65 grouped, one column (391 blocks each) 3.39 alone and 2.80 grouped.
constexpr uint32_t SL_ALONE_BLOCKS = 148 * 4;
struct SlGroup {
    ScatterProb pr[SL_GROUP];
    SLDev L[SL_GROUP];
    uint32_t first[SL_GROUP];   // problems of short segments only: the first one
    uint32_t block0[SL_GROUP];  // first block of each problem
    int n;
};

template <int K>
__global__ void __launch_bounds__(SL_THREADS)
k_seggroup(const __grid_constant__ SlGroup G, const double* u, const double* sqrt_w, double* out,
           const int* __restrict__ skip) {
    pdl_wait();
    pdl_launch_dependents();
    if (skip && *skip) return;
    int q = 0;
#pragma unroll
    for (int i = 1; i < SL_GROUP; ++i)
        if (i < G.n && blockIdx.x >= G.block0[i]) q = i;
    const SlScatter<K> f{G.pr[q], u, sqrt_w, out};
    seglist_block<SlScatter<K>, K, false>(f, G.L[q], blockIdx.x - G.block0[q], G.first[q]);
}

}  // namespace wgpu
