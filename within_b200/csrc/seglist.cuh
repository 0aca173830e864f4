// seglist.cuh -- the piece engine: deterministic segmented reduction from work
// lists of short segments and of pieces of long ones (segbook.hpp), the
// default for every FP64 plan of the Schwarz apply and of the adjoint's rest.
//
// What bounds the sums: 12 bytes of index and value per non-zero and one
// gathered operand.  The scan engines (segreduce.cuh, segsweep.cuh) find segment
// boundaries inside a tile of mixed segments, which costs tens of instructions
// per position in scans, shuffles and barriers: 2.4 warp instructions per
// non-zero for C^T at one column, and 500 us at eight.  Knowing each segment's
// length beforehand, no scan is needed:
//   - a long segment (more than SL_SHORT positions) is cut into pieces of 512 to
//     4096 positions; a warp strides over its piece, every lane keeps one
//     partial, and one shuffle tree ends it.  Several pieces of one segment are
//     added in piece order by the last warp to arrive (an atomic counter, not a
//     wait);
//   - a short segment is summed in position order by one group of lanes.
// The K columns of a position lie across K / 2 lanes (two columns per lane, one
// 16-byte access), so at K = 8 a warp step covers eight positions with 64-byte
// operand reads, and no lane holds K accumulators.  Every sum has one fixed
// order: results are bitwise reproducible, with no floating-point atomics.
#pragma once
#include "pdl.cuh"
#include <cstdint>

#include "kernels.cuh"
#include "segbook.hpp"

namespace wgpu {

constexpr int SL_THREADS = 256;
constexpr int SL_WARPS = SL_THREADS / 32;

// device view of one problem's lists
struct SLDev {
    const uint32_t* ptr;          // segment pointers
    const uint32_t* short_ids;    // nullptr: short segment i is first + i
    uint32_t first, n_short;
    uint32_t short_blocks;
    const SLPiece* pieces;
    uint32_t piece_lo, piece_hi;
    const SLSplit* splits;
    double* part;                 // K per piece
    unsigned* counters;           // one per split
};

// F provides (W = fl_w<K>() columns from column c0):
//   struct Ctx; Ctx ctx(uint32_t seg) const;             what every position of a segment shares
//   FlVec<W> value(const Ctx&, uint32_t pos, int c0) const;
//   void emit(uint32_t seg, int c0, const FlVec<W>& s) const;
template <class F, int K>
__device__ __forceinline__ FlVec<fl_w<K>()> sl_sum(const F& f, const typename F::Ctx& cx, uint32_t a, uint32_t b,
                                                   uint32_t stride, int c0) {
    constexpr int W = fl_w<K>();
    constexpr int U = 4;   // values requested before any is added
    FlVec<W> s;
#pragma unroll
    for (int i = 0; i < W; ++i) s.q[i] = 0.0;
    uint32_t q = a;
    for (; q + (U - 1) * stride < b; q += U * stride) {
        FlVec<W> v[U];
#pragma unroll
        for (int j = 0; j < U; ++j) v[j] = f.value(cx, q + j * stride, c0);
#pragma unroll
        for (int j = 0; j < U; ++j)
#pragma unroll
            for (int i = 0; i < W; ++i) s.q[i] += v[j].q[i];
    }
    for (; q < b; q += stride) {
        const FlVec<W> v = f.value(cx, q, c0);
#pragma unroll
        for (int i = 0; i < W; ++i) s.q[i] += v.q[i];
    }
    return s;
}

template <class F, int K>
__global__ void __launch_bounds__(SL_THREADS)
k_seglist(F f, SLDev L, const int* __restrict__ skip) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int W = fl_w<K>(), P = fl_per_row<K>(), S = 32 / P;
    if (skip && *skip) return;
    if (blockIdx.x < L.short_blocks) {
        const uint32_t t = blockIdx.x * SL_THREADS + threadIdx.x;
        const uint32_t i = t / P;
        const int c0 = (int)(t % P) * W;
        if (i >= L.n_short) return;
        const uint32_t seg = L.short_ids ? __ldg(L.short_ids + i) : L.first + i;
        const uint32_t a = __ldg(L.ptr + seg), b = __ldg(L.ptr + seg + 1);
        f.emit(seg, c0, sl_sum<F, K>(f, f.ctx(seg), a, b, 1, c0));
        return;
    }
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t r = L.piece_lo + (blockIdx.x - L.short_blocks) * SL_WARPS + (threadIdx.x >> 5);
    if (r >= L.piece_hi) return;   // whole warps
    const SLPiece pc = L.pieces[r];
    const int g = lane / P, c0 = (lane % P) * W;
    FlVec<W> s = sl_sum<F, K>(f, f.ctx(pc.seg), pc.p0 + g, pc.p1, S, c0);
#pragma unroll
    for (int o = P; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < W; ++i) s.q[i] += __shfl_xor_sync(FULL, s.q[i], o);
    if (pc.split < 0) {
        if (lane < P) f.emit(pc.seg, c0, s);
        return;
    }
    if (lane < P) {
        fl_st<W>(L.part + (size_t)r * K + c0, s);
        __threadfence();
    }
    __syncwarp();
    const SLSplit sp = L.splits[pc.split];
    unsigned last = 0;
    if (lane == 0) last = atomicAdd(&L.counters[pc.split], 1u) == sp.r1 - sp.r0 ? 1u : 0u;
    if (!__shfl_sync(FULL, last, 0)) return;
    __threadfence();
#pragma unroll
    for (int i = 0; i < W; ++i) s.q[i] = 0.0;
    for (uint32_t q = sp.r0 + g; q <= sp.r1; q += S)
#pragma unroll
        for (int i = 0; i < W; ++i) s.q[i] += __ldcg(L.part + (size_t)q * K + c0 + i);
#pragma unroll
    for (int o = P; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < W; ++i) s.q[i] += __shfl_xor_sync(FULL, s.q[i], o);
    if (lane < P) f.emit(pc.seg, c0, s);
    if (lane == 0) L.counters[pc.split] = 0;
}

// One column, every segment short: a warp's 32 segments are 32 consecutive runs
// of positions, so the warp computes their values with coalesced reads into
// shared memory and every lane then adds its own segment's in position order
// (the sum of one lane reading them from memory, bit for bit).  A lane that
// walks its row in memory takes one L1 wavefront per element and array: C on
// the 10,000,000-row panel (10.4 M non-zeros, rows of about ten) took 70 us
// for 20 us of traffic that way.
constexpr uint32_t SL_STAGE = 512;   // values staged per warp; wider groups read memory directly

template <class F>
__global__ void __launch_bounds__(SL_THREADS)
k_segstage(F f, const uint32_t* __restrict__ ptr, uint32_t first, uint32_t n_seg, const int* __restrict__ skip) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ double sm[SL_WARPS][SL_STAGE];
    if (skip && *skip) return;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t i0 = (blockIdx.x * SL_WARPS + wid) * 32u;
    if (i0 >= n_seg) return;   // whole warps
    const bool mine = i0 + lane < n_seg;
    const uint32_t seg = first + (mine ? i0 + lane : n_seg - 1);
    const uint32_t b = __ldg(ptr + seg + 1), a = mine ? __ldg(ptr + seg) : b;
    const uint32_t w0 = __shfl_sync(FULL, a, 0), w1 = __shfl_sync(FULL, b, 31);
    const typename F::Ctx cx = f.ctx(seg);
    FlVec<1> s;
    if (w1 - w0 <= SL_STAGE) {
        uint32_t q = w0 + lane;
        for (; q + 96 < w1; q += 128) {
            FlVec<1> v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = f.value(cx, q + 32 * j, 0);
#pragma unroll
            for (int j = 0; j < 4; ++j) sm[wid][q + 32 * j - w0] = v[j].q[0];
        }
        for (; q < w1; q += 32) sm[wid][q - w0] = f.value(cx, q, 0).q[0];
        __syncwarp();
        s.q[0] = 0.0;
        for (uint32_t p = a; p < b; ++p) s.q[0] += sm[wid][p - w0];
    } else {
        s = sl_sum<F, 1>(f, cx, a, b, 1, 0);
    }
    if (mine) f.emit(seg, 0, s);
}

// ---------------------------------------------------------------------------
// The steps of the Schwarz apply and the adjoint's rest on this engine; the
// sums are those of the functors of the same name in kernels.cuh, FP64.
template <int K>
struct SlBase {
    static constexpr bool STAGED = false;   // one column, short segments only: k_segstage
    static constexpr int W = fl_w<K>();
    using V = FlVec<W>;
    SchwarzDev S;
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
};

template <int K>
struct SlRestrict : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    const double* r;
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t j, int c0) const {
        const uint32_t g = __ldg(this->S.glob + j);
        const V v = B::scaled(B::ld(r, g, c0), __ldg(this->S.scale + j));
        B::st(this->S.rl, j, c0, v);
        return v;
    }
    __device__ void emit(uint32_t sub, int c0, const V& s) const {
        const bool fl = this->S.mode[sub] == 0;
        const double inv = 1.0 / (double)(this->S.loc_ptr[sub + 1] - this->S.loc_ptr[sub]);
        V o;
#pragma unroll
        for (int i = 0; i < B::W; ++i) o.q[i] = fl ? s.q[i] * inv : 0.0;
        B::st(this->S.m1, sub, c0, o);
    }
};

template <int K>
struct SlCt : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        return B::scaled(B::ld(this->S.rl, __ldg(this->S.ct_col + a), c0), __ldg(this->S.ct_val + a));
    }
    __device__ void emit(uint32_t row, int c0, const V& s) const {
        const SchwarzDev& S = this->S;
        const uint32_t slot = S.ct_row_slot[row], rbi = S.ct_row_red[row];
        const uint32_t sub = S.slot_sub[slot];
        const double rsum = S.ct_rowsum[row];
        const V m = B::ld(S.m1, sub, c0), rlv = B::ld(S.rl, slot, c0);
        V val, neg;
#pragma unroll
        for (int i = 0; i < B::W; ++i) {
            val.q[i] = (rlv.q[i] - m.q[i]) + (s.q[i] - m.q[i] * rsum);
            neg.q[i] = -val.q[i];
        }
        B::st(S.rb, rbi, c0, val);
        if (S.mode[sub] == 2) B::st(S.rb, rbi + S.n_kept[sub], c0, neg);
    }
};

template <int K>
struct SlKeptSum : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t q, int c0) const {
        return B::ld(this->S.rb, __ldg(this->S.ct_row_red + q), c0);
    }
    __device__ void emit(uint32_t sub, int c0, const V& s) const {
        const SchwarzDev& S = this->S;
        const int m = S.mode[sub];
        const double rn = (double)S.red_n[sub];
        V o, neg;
#pragma unroll
        for (int i = 0; i < B::W; ++i) {
            o.q[i] = m == 0 ? s.q[i] / rn : 0.0;
            neg.q[i] = -s.q[i];
        }
        if (m == 1) B::st(S.rb, S.red_off[sub] + S.n_kept[sub], c0, neg);
        B::st(S.m2, sub, c0, o);
    }
};

template <int K>
struct SlDense : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        return B::scaled(this->reduced(__ldg(this->S.dense_col + a), c0), __ldg(this->S.dense_val + a));
    }
    __device__ void emit(uint32_t row, int c0, const V& s) const {
        B::st(this->S.xv, this->S.dense_row_slot[row], c0, s);
    }
};

template <int K>
struct SlFwd : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        return B::scaled(B::ld(this->S.yv, __ldg(this->S.fwd_col + a), c0), __ldg(this->S.fwd_val + a));
    }
    __device__ void emit(uint32_t row, int c0, const V& s) const {
        const uint32_t u = this->S.fwd_row[row];
        const V b = this->reduced(u, c0);
        const double di = this->S.dinv[u];
        V y, x;
#pragma unroll
        for (int i = 0; i < B::W; ++i) {
            y.q[i] = b.q[i] - s.q[i];
            x.q[i] = y.q[i] * di;
        }
        B::st(this->S.yv, u, c0, y);
        B::st(this->S.xv, u, c0, x);
    }
};

template <int K>
struct SlCore : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        return B::scaled(B::ld(this->S.yv, __ldg(this->S.core_col + a), c0), __ldg(this->S.core_val + a));
    }
    __device__ void emit(uint32_t row, int c0, const V& s) const {
        B::st(this->S.xv, this->S.core_row_slot[row], c0, s);
    }
};

template <int K>
struct SlBwd : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        return B::scaled(B::ld(this->S.xv, __ldg(this->S.bwd_col + a), c0), __ldg(this->S.bwd_val + a));
    }
    __device__ void emit(uint32_t row, int c0, const V& s) const {
        const uint32_t v = this->S.bwd_row[row];
        V x = B::ld(this->S.xv, v, c0);
#pragma unroll
        for (int i = 0; i < B::W; ++i) x.q[i] -= s.q[i];
        B::st(this->S.xv, v, c0, x);
    }
};

template <int K>
struct SlC : SlBase<K> {
    static constexpr bool STAGED = true;
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        const uint32_t cc = __ldg(this->S.c_col + a);
        const double c = __ldg(this->S.c_val + a);
        if (!(cc & 0x80000000u)) return B::scaled(B::ld(this->S.xv, cc, c0), c);
        const uint32_t u = cc & 0x7fffffffu, s = this->S.red_sub[u];
        return B::scaled(this->kept(u, s, this->S.mode[s], c0), c);
    }
    __device__ void emit(uint32_t row, int c0, const V& s) const {
        const uint32_t e = this->S.elim_slot[row];
        const uint32_t sub = this->S.slot_sub[e];
        const double ie = this->S.inv_e[e];
        const V rlv = B::ld(this->S.rl, e, c0), m = B::ld(this->S.m1, sub, c0);
        V o;
#pragma unroll
        for (int i = 0; i < B::W; ++i) o.q[i] = (rlv.q[i] - m.q[i]) * ie + s.q[i];
        B::st(this->S.sl, e, c0, o);
    }
};

template <int K>
struct SlMean : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {
        uint32_t sub, elim_end, red0;   // slots below elim_end are eliminated; red0 + j is kept slot j's reduced slot
        int mode;
    };
    __device__ Ctx ctx(uint32_t s) const {
        const uint32_t e = this->S.loc_ptr[s] + this->S.n_elim[s];
        return Ctx{s, e, this->S.red_off[s] - e, this->S.mode[s]};
    }
    __device__ V value(const Ctx& cx, uint32_t j, int c0) const {
        if (j < cx.elim_end) return B::ld(this->S.sl, j, c0);
        const V v = this->kept(cx.red0 + j, cx.sub, cx.mode, c0);
        B::st(this->S.sl, j, c0, v);
        return v;
    }
    __device__ void emit(uint32_t sub, int c0, const V& s) const {
        const bool fl = this->S.mode[sub] == 0;
        const double inv = 1.0 / (double)(this->S.loc_ptr[sub + 1] - this->S.loc_ptr[sub]);
        V o;
#pragma unroll
        for (int i = 0; i < B::W; ++i) o.q[i] = fl ? s.q[i] * inv : 0.0;
        B::st(this->S.m3, sub, c0, o);
    }
};

template <int K>
struct SlProlong : SlBase<K> {
    using B = SlBase<K>;
    using V = typename B::V;
    struct Ctx {};
    double* z;
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t a, int c0) const {
        const uint32_t j = __ldg(this->S.dof_slot + a);
        const uint32_t s = __ldg(this->S.slot_sub + j);
        const double sc = __ldg(this->S.scale + j);
        V v = B::ld(this->S.sl, j, c0);
        const V m = B::ld(this->S.m3, s, c0);
#pragma unroll
        for (int i = 0; i < B::W; ++i) v.q[i] = sc * (v.q[i] - m.q[i]);
        return v;
    }
    __device__ void emit(uint32_t dof, int c0, const V& s) const { B::st(z, dof, c0, s); }
};

// one (term, column) problem of A^T u: run sums by run ordinal, or the rows
// of the term's level-sorted order
template <int K>
struct SlScatter {
    static constexpr bool STAGED = false;
    static constexpr int W = fl_w<K>();
    using V = FlVec<W>;
    struct Ctx {};
    ScatterProb pr;
    const double* u;
    const double* sqrt_w;
    double* out;
    __device__ Ctx ctx(uint32_t) const { return {}; }
    __device__ V value(const Ctx&, uint32_t pos, int c0) const {
        const uint32_t i = pr.order ? __ldg(pr.order + pos) : pos;
        if (pr.run_sum) return fl_ld<W>(pr.run_sum + ((size_t)i * pr.ncol + pr.col) * K + c0);
        double f = pr.load ? __ldg(pr.load + i) : 1.0;
        if (sqrt_w) f *= __ldg(sqrt_w + i);
        V v = fl_ld<W>(u + (size_t)i * K + c0);
#pragma unroll
        for (int k = 0; k < W; ++k) v.q[k] *= f;
        return v;
    }
    __device__ void emit(uint32_t seg, int c0, const V& s) const {
        fl_st<W>(out + ((size_t)pr.out_off + seg) * K + c0, s);
    }
};

}  // namespace wgpu
