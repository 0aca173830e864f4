// csweep.cuh -- the column-lane row sweep: the fused row sweep of rowsweep.cuh
// for several right-hand sides (K = 2, 4, 8) of intercept-only designs of at
// most three terms.
//
// What bounds it: one row carries 8 K bytes of u in and out (16 K with K
// columns of FP64) against 4 bytes per code, so the LSMR step is a stream of
// 1.4 GB at K = 8 on a 10,000,000-row panel.  The scan layout of rowsweep.cuh
// (a lane holds R rows and all K columns) spends its time elsewhere: a
// five-step shuffle scan per column and run term, and a match loop per row for
// the histogram term.  Here the K columns of a row lie across LPR = K / 2
// lanes (two columns per lane, one 16-byte access each), a warp holds S =
// 32 / LPR independent streams of consecutive rows, and every stream walks its
// own fixed range of rows in order.  A run is then a register accumulator that
// is written when the code changes -- no shuffle, no scan -- and a histogram
// term is one private shared-memory bin per lane and level, conflict-free
// whatever the levels (lane l owns bytes [16 l, 16 l + 16) of every bin row).
// The next four rows' codes, u and sqrt(w) are requested before the current
// four are used.  10,000,000-row panel, eight columns: the LSMR step 1272 ->
// 431 us (1.4 GB: 3.3 of 6.5 TB/s), the adjoint 823 -> 205 us; 2,000,000 rows,
// weighted, four columns: 145 -> 76 us.  Four rows per step because each
// stream then reads 256 consecutive bytes of u per request (with two rows the
// same kernel took 501 us); three blocks per SM because the registers of four
// (128 per thread) spill.  The weighted step of four and eight columns spills all
// the same at 168 registers (about 100 bytes a thread; weights cost 20 us of 119 at
// eight columns).  What is left is latency at low occupancy: 12 warps per SM,
// 18 % of the warp slots, waiting for u and for gathered coefficients (long
// scoreboard), DRAM at 39 % with eight columns and 16 % with two.
//
// The private bins take 2 KB per level and block, so a histogram term of more
// than 35 levels leaves two blocks per SM and one of more than 53 a single one,
// and at two columns every lane walks a range of its own.  It is taken there too:
// LSMR step of 2,000,000 rows against the scan sweep, us (weighted in brackets):
//   bins      two columns          four columns           eight columns
//     20   69 -> 46  (72 -> 52)  146 ->  65 (149 ->  78)  331 -> 100 (332 -> 120)
//     35   82 -> 66  (88 -> 82)  159 -> 102 (160 -> 113)  353 -> 137 (356 -> 142)
//     50   89 -> 72  (94 -> 88)  182 -> 111 (185 -> 131)  408 -> 143 (412 -> 175)
//     64   95 -> 61 (100 -> 79)  203 -> 113 (205 -> 138)  447 -> 198 (448 -> 242)
// and 1.3 to 7 times as fast on 200,000 rows.
//
// The ranges are those of rowsweep.cuh with one range per stream: a run that
// crosses ranges leaves a tail partial and head partials, which k_cs_finish
// adds in range order; it also adds the block partials of the norms and of the
// bins, one warp per sum, so the sweep has no serial last block.  Every sum has
// one fixed order: results are bitwise reproducible.
#pragma once
#include "pdl.cuh"
#include <type_traits>

#include "rowsweep.cuh"

namespace wgpu {

constexpr int CS_THREADS = 128;
constexpr int CS_WARPS = CS_THREADS / 32;
constexpr int CS_MAXQ = 3;
constexpr int CS_ROWS = 4;            // rows per step and stream
constexpr uint32_t CS_MIN_RANGE = 16; // rows of the shortest range
constexpr int CS_BLOCKS_PER_SM = 3;   // by registers (168 per thread)
constexpr size_t CS_SMEM_PER_SM = 216 * 1024;

template <int K>
__host__ __device__ constexpr int cs_lpr() { return K / 2; }
template <int K>
__host__ __device__ constexpr int cs_streams() { return 32 / cs_lpr<K>(); }

// bins: one double2 per lane, warp and bucket
__host__ __device__ constexpr size_t cs_smem_bytes(int n_buckets) {
    return (size_t)CS_WARPS * n_buckets * 32 * sizeof(double2);
}
// resident blocks per SM the bins leave room for
inline int cs_blocks_per_sm(int n_buckets) {
    const size_t sm = cs_smem_bytes(n_buckets) + 1024;
    const size_t fit = CS_SMEM_PER_SM / sm;
    return fit < 1 ? 1 : (fit > (size_t)CS_BLOCKS_PER_SM ? CS_BLOCKS_PER_SM : (int)fit);
}

// class of every term: 0 left to the segmented reduction, 1 run term
// (slot = index into RwParams::run), 2 histogram term (slot = its bucket0)
struct CsTerms {
    int nq;
    int cls[CS_MAXQ];
    int slot[CS_MAXQ];
};

// one step's inputs of a stream: R full rows from `row`
template <int R, bool WTD>
struct CsRows {
    uint32_t cd[CS_MAXQ][R];
    double2 in[R];           // u (modes 0, 1) or the right-hand side (mode 3)
    double w[WTD ? R : 1];
};

template <int K, int R, bool WTD>
__device__ __forceinline__ void cs_load(const OpParams& p, const CsTerms& ct, const double* in, uint32_t row, int c2,
                                        CsRows<R, WTD>& B) {
#pragma unroll
    for (int t = 0; t < CS_MAXQ; ++t) {
        if (t >= ct.nq) continue;
        if constexpr (R == CS_ROWS) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(p.codes[t] + row));
            B.cd[t][0] = q.x;
            B.cd[t][1] = q.y;
            B.cd[t][2] = q.z;
            B.cd[t][3] = q.w;
        } else {
            B.cd[t][0] = __ldg(p.codes[t] + row);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) B.in[r] = *reinterpret_cast<const double2*>(in + (size_t)(row + r) * K + c2);
    if constexpr (WTD) {
#pragma unroll
        for (int r = 0; r < R; ++r) B.w[r] = __ldg(p.sqrt_w + row + r);
    }
}

// a run term of one stream: the open run's sum, its code, the ordinal of the
// next run (terms summed by run ordinal) and whether its head lies in this range
struct CsRun {
    double2 acc;
    uint32_t code, next;
    bool started;
};

template <int K, int MODE, bool WTD>
__global__ void __launch_bounds__(CS_THREADS, CS_BLOCKS_PER_SM)
k_csweep(OpParams p, RwParams rw, CsTerms ct, const double* __restrict__ v, double* __restrict__ u, ColState* cur,
         Ctl* ctl, const int* skip, int store, const double* __restrict__ rhs) {
    pdl_wait();
    pdl_launch_dependents();
    static_assert(MODE == 0 || MODE == 1 || MODE == 3, "FP64 modes only");
    constexpr int LPR = cs_lpr<K>(), S = cs_streams<K>();
    constexpr bool NORM = MODE == 1 || MODE == 3;
    extern __shared__ double2 cs_bins[];
    __shared__ double red[CS_WARPS][K];
    if (MODE == 1 && ctl->all_done) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->k5_skip = 1;
        return;
    }
    if (MODE != 1 && skip && *skip) return;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int sub = lane / LPR, c2 = (lane % LPR) * 2;
    const int nb = rw.n_buckets;
    double2* bins = cs_bins + (size_t)wid * nb * 32 + lane;
    for (int i = 0; i < nb; ++i) bins[i * 32] = make_double2(0.0, 0.0);

    bool act0 = false, act1 = false;
    double sc0 = 0.0, sc1 = 0.0;
    if (MODE == 1) {
        act0 = !cur[c2].done;
        act1 = !cur[c2 + 1].done;
        sc0 = -(cur[c2].alpha * cur[c2].beta_prev_inv);
        sc1 = -(cur[c2 + 1].alpha * cur[c2 + 1].beta_prev_inv);
    }
    double2 accn = make_double2(0.0, 0.0);

    const uint32_t g = ((uint32_t)blockIdx.x * CS_WARPS + wid) * S + sub;
    const uint64_t r0w = (uint64_t)g * rw.rows_per_range;
    const uint32_t r0 = (uint32_t)min(r0w, (uint64_t)p.n);
    const uint32_t r1 = (uint32_t)min(r0w + rw.rows_per_range, (uint64_t)p.n);
    const double* in = MODE == 3 ? rhs : u;
    double* atu = reinterpret_cast<double*>(rw.atu);

    // run terms: dst is where the open run's sum goes when the run ends -- A^T u
    // by level (sorted term), the run-sum array by ordinal, or the range's head
    // partial when the run started in an earlier range
    CsRun run[CS_MAXQ];
    char* dst[CS_MAXQ];
#pragma unroll
    for (int t = 0; t < CS_MAXQ; ++t) {
        run[t] = CsRun{make_double2(0.0, 0.0), 0u, 0u, false};
        dst[t] = nullptr;
        if (t < ct.nq && ct.cls[t] == 1 && r0 < r1) {
            const RwRun& RR = rw.run[ct.slot[t]];
            const uint32_t c0 = __ldg(p.codes[t] + r0);
            run[t].code = c0;
            run[t].started = r0 == 0 || __ldg(p.codes[t] + r0 - 1) != c0;
            if (!RR.direct) run[t].next = __ldg(RR.range_base + g) + (run[t].started ? 1u : 0u);
            if (!run[t].started) dst[t] = reinterpret_cast<char*>(RR.head + (size_t)g * K + c2);
            else if (RR.direct) dst[t] = reinterpret_cast<char*>(atu + ((size_t)p.off[t] + c0) * K + c2);
            else dst[t] = reinterpret_cast<char*>(RR.run_sum + (size_t)(run[t].next - 1) * K + c2);
        }
    }

    // R rows whose inputs are in B; x: their coefficients (modes 1 to 3)
    auto step = [&](auto RC, uint32_t row, const auto& B, const auto& x) {
        constexpr int R = decltype(RC)::value;
        double2 b[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            double2 val;
            if constexpr (MODE == 0) {
                val = B.in[r];
            } else {
                double2 av = make_double2(0.0, 0.0);
#pragma unroll
                for (int t = 0; t < CS_MAXQ; ++t) {   // terms in term order, as in k_rowsweep
                    if (t >= ct.nq) continue;
                    av.x += x[t][r].x;
                    av.y += x[t][r].y;
                }
                if constexpr (WTD) {
                    av.x *= B.w[r];
                    av.y *= B.w[r];
                }
                if constexpr (MODE == 1) {
                    val.x = act0 ? av.x + sc0 * B.in[r].x : B.in[r].x;
                    val.y = act1 ? av.y + sc1 * B.in[r].y : B.in[r].y;
                } else {
                    val.x = B.in[r].x - av.x;
                    val.y = B.in[r].y - av.y;
                }
                if constexpr (NORM) {
                    accn.x += val.x * val.x;
                    accn.y += val.y * val.y;
                }
                if (MODE == 1 || store) *reinterpret_cast<double2*>(u + (size_t)(row + r) * K + c2) = val;
            }
            b[r] = WTD ? make_double2(B.w[WTD ? r : 0] * val.x, B.w[WTD ? r : 0] * val.y) : val;
        }
#pragma unroll
        for (int t = 0; t < CS_MAXQ; ++t) {
            if (t >= ct.nq || ct.cls[t] == 0) continue;
            if (ct.cls[t] == 2) {
                double2* bt = bins + ct.slot[t] * 32;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    double2* q = bt + B.cd[t][r] * 32;
                    double2 o = *q;
                    o.x += b[r].x;
                    o.y += b[r].y;
                    *q = o;
                }
                continue;
            }
            const RwRun& RR = rw.run[ct.slot[t]];
            const bool direct = RR.direct != 0;
            char* base = direct ? reinterpret_cast<char*>(atu + (size_t)p.off[t] * K + c2)
                                : reinterpret_cast<char*>(RR.run_sum + c2);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint32_t c = B.cd[t][r];
                const bool head = c != run[t].code;
                if (head) {   // the open run ends; the next one starts
                    *reinterpret_cast<double2*>(dst[t]) = run[t].acc;
                    const uint32_t idx = direct ? c : run[t].next;
                    ++run[t].next;
                    dst[t] = base + (size_t)idx * (K * sizeof(double));
                    run[t].started = true;
                    run[t].code = c;
                }
                run[t].acc.x = head ? b[r].x : run[t].acc.x + b[r].x;
                run[t].acc.y = head ? b[r].y : run[t].acc.y + b[r].y;
            }
        }
    };
    auto gather = [&](auto RC, const auto& B, auto& x) {
        constexpr int R = decltype(RC)::value;
        if constexpr (MODE != 0) {
#pragma unroll
            for (int t = 0; t < CS_MAXQ; ++t) {
                if (t >= ct.nq) continue;
                const double* vt = v + (size_t)p.off[t] * K + c2;
#pragma unroll
                for (int r = 0; r < R; ++r) x[t][r] = __ldg(reinterpret_cast<const double2*>(vt + (size_t)B.cd[t][r] * K));
            }
        }
    };
    if (r0 < r1) {
        using RS = std::integral_constant<int, CS_ROWS>;
        using R1 = std::integral_constant<int, 1>;
        const uint32_t steps = (r1 - r0) / CS_ROWS;
        uint32_t row = r0;
        if (steps) {
            CsRows<CS_ROWS, WTD> C, N;
            cs_load<K, CS_ROWS, WTD>(p, ct, in, row, c2, N);
            for (uint32_t s = 0; s < steps; ++s, row += CS_ROWS) {
                C = N;
                double2 x[CS_MAXQ][CS_ROWS];
                gather(RS{}, C, x);
                // the next rows' streams, requested before this step's sums
                if (s + 1 < steps) cs_load<K, CS_ROWS, WTD>(p, ct, in, row + CS_ROWS, c2, N);
                step(RS{}, row, C, x);
            }
        }
        for (; row < r1; ++row) {   // the ragged end of the data
            CsRows<1, WTD> C;
            double2 x[CS_MAXQ][1];
            cs_load<K, 1, WTD>(p, ct, in, row, c2, C);
            gather(R1{}, C, x);
            step(R1{}, row, C, x);
        }
        // range end: the open run -- complete when it started here and ends
        // exactly at the range end, else the tail or (started earlier) a head partial
#pragma unroll
        for (int t = 0; t < CS_MAXQ; ++t) {
            if (t >= ct.nq || ct.cls[t] != 1) continue;
            const bool cont = r1 < p.n && __ldg(p.codes[t] + r1) == run[t].code;
            double* out = run[t].started && cont ? rw.run[ct.slot[t]].tail + (size_t)g * K + c2
                                                 : reinterpret_cast<double*>(dst[t]);
            *reinterpret_cast<double2*>(out) = run[t].acc;
        }
    }
    __syncwarp();
    // ---- block partials: the streams of each warp by a fixed xor tree, then the warps in order.
    // Layout [sum][block], so that k_cs_finish reads consecutive blocks.
    const unsigned nblk = gridDim.x;
    if constexpr (NORM) {
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1) {
            accn.x += __shfl_xor_sync(FULL, accn.x, o);
            accn.y += __shfl_xor_sync(FULL, accn.y, o);
        }
        if (lane < LPR) {
            red[wid][c2] = accn.x;
            red[wid][c2 + 1] = accn.y;
        }
    }
    for (int i = 0; i < nb; ++i) {
        double2 q = bins[i * 32];
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1) {
            q.x += __shfl_xor_sync(FULL, q.x, o);
            q.y += __shfl_xor_sync(FULL, q.y, o);
        }
        if (lane < LPR) bins[i * 32] = q;
    }
    __syncthreads();
    if (NORM && threadIdx.x < K) {
        double a = 0.0;
#pragma unroll
        for (int w = 0; w < CS_WARPS; ++w) a += red[w][threadIdx.x];
        rw.part[(size_t)threadIdx.x * nblk + blockIdx.x] = a;
    }
    const double* fb = reinterpret_cast<const double*>(cs_bins);
    for (int i = threadIdx.x; i < nb * K; i += CS_THREADS) {
        const int bk = i / K, k = i % K;
        double a = 0.0;
#pragma unroll
        for (int w = 0; w < CS_WARPS; ++w) a += fb[((size_t)(w * nb + bk) * 32) * 2 + k];
        rw.part[(size_t)(K + i) * nblk + blockIdx.x] = a;
    }
}

// After the sweep: blocks [0, fix_blocks) add the partials of the runs that
// cross ranges (tail of range g0 + heads of g0+1..g1, in range order; one
// thread per run and column), the others the block partials (one warp per
// norm or bin): beta (mode 1) or ||r||^2 (mode 3), and the bins into A^T u.
constexpr int CS_FIN_THREADS = 256;
template <int K, int MODE>
__global__ void __launch_bounds__(CS_FIN_THREADS)
k_cs_finish(OpParams p, RwParams rw, CsTerms ct, unsigned nblk, unsigned fix_blocks, ColState* cur,
            const Ctl* ctl, const int* skip, double* sq_out, int sq_stride) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr bool NORM = MODE == 1 || MODE == 3;
    if (MODE == 1 && ctl->all_done) return;
    if (MODE != 1 && skip && *skip) return;
    double* atu = reinterpret_cast<double*>(rw.atu);
    if (blockIdx.x < fix_blocks) {
        const uint32_t i = blockIdx.x * CS_FIN_THREADS + threadIdx.x;
        const uint32_t f = i / K, k = i % K;
        if (f >= rw.n_fix) return;
        const RwFix fx = rw.fix[f];
        const RwRun& RR = rw.run[fx.run];
        double a = __ldcg(&RR.tail[(size_t)fx.g0 * K + k]);
        for (uint32_t h = fx.g0 + 1; h <= fx.g1; ++h) a += __ldcg(&RR.head[(size_t)h * K + k]);
        if (RR.direct) atu[((size_t)p.off[RR.term] + fx.id) * K + k] = a;
        else RR.run_sum[(size_t)fx.id * K + k] = a;
        return;
    }
    const int i = (int)((blockIdx.x - fix_blocks) * (CS_FIN_THREADS / 32) + (threadIdx.x >> 5));
    if (i >= K + rw.n_buckets * K || (i < K && !NORM)) return;   // whole warps
    const int lane = threadIdx.x & 31;
    double a = 0.0;
    for (unsigned b = lane; b < nblk; b += 32) a += __ldcg(&rw.part[(size_t)i * nblk + b]);
    a = warp_sum(a);
    if (lane != 0) return;
    if (i < K) {
        if (MODE == 1 && !cur[i].done) cur[i].beta = sqrt(a);
        if (MODE == 3) sq_out[(size_t)i * sq_stride] = a;
        return;
    }
    const int bk = (i - K) / K, k = (i - K) % K;
#pragma unroll
    for (int t = 0; t < CS_MAXQ; ++t)
        if (t < ct.nq && ct.cls[t] == 2 && bk >= ct.slot[t] && bk < ct.slot[t] + (int)p.L[t])
            atu[((size_t)p.off[t] + (uint32_t)(bk - ct.slot[t])) * K + k] = a;
}

}  // namespace wgpu
