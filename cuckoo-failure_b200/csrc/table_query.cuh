// Queries served from resident tables (cf_tables_query): N_bad(n, M) mod p for primes whose whole
// V (packed triangle) and tables fact, ifact, inv were kept by a serving build (KParams::keep).  The
// arithmetic is that of the build's own query and finish phases (query_row and finish in
// prime_fp.cuh): the per-row sums of fast/cuckoo_fast.cu:306-323, 595-622 and the Horner finish of
// :877-890, read from the resident triangle instead of from the row the build is about to consume.
//
// The rows' factors F(q) = inv[q] ifact[n-q] ifact[M-q] Q^(n-q) go in front of the inner sums:
//   sum_q F(q) sum_w Vs[q][w] / (M-w)  =  sum_w 1/(M-w) sum_q F(q) Vs[q][w],
// so a warp takes TQ_ROWS rows of TQ_COLS columns, each lane its own columns down the rows: an entry
// costs one product by a factor all lanes share, the inverses enter once per column, and nothing is
// summed across lanes but the tile's total.  A prime's tiles go to the warps of a cluster of CTAs.
//
// Bound by the triangle's bytes where few queries read it (8 queries, two of them as large as the
// table, n = 2048, 148 primes: 2.5 GB), by the products (seven double-precision operations each) where
// many do.  A warp reads 2 KB of a row at a time, a row ahead: with 256 bytes of four rows at a
// time, summing along the rows, HBM gave 2.2 TB/s (1320 us for that case); the form before that, one
// CTA of 64-bit integer products per (prime, query), took 3570 us; this one takes 600 to 700 (3.6 to 4.2 TB/s).
#pragma once
#include <cuda_runtime.h>

#include "suffix_engine.cuh"
#include "table_split.hpp"

namespace cfb {

// Queries per launch: their sizes travel in the kernel parameters (no staging buffer, so launches
// on several streams never share one).
constexpr int TQ_MAXJ = 256;  // (the host sorts by size << 8 | place)
struct TQParams {
    const u64* primes;  // [B]
    int B, n, F, d, d0, model, J;
    int S, G, W;        // the launch's split (tq_split)
    const u64* keep;    // [B][keep_words]
    size_t keep_words;
    u64* out;           // residue of prime b, query jq at out[b * out_stride + jq]
    size_t out_stride;
    int qn[TQ_MAXJ];    // each <= n, descending
    int qM[TQ_MAXJ];    // each <= F
    short qi[TQ_MAXJ];  // the query's place in out
};

// Shared memory: per query of a group Q and the warps' sums, and (read from the first CTA) the CTAs' sums.
inline size_t tq_smem_bytes(int Jg) { return 8 * (size_t)Jg * (1 + TQ_WARPS + TQ_CLUSTER); }

// a whole number below 2^52 as a double
__device__ __forceinline__ double tq_double(u64 v) { return __dadd_rn(__longlong_as_double((long long)(v | 0x4330000000000000ull)), -4503599627370496.0); }
__device__ __forceinline__ double tq_load(const u64* p) { return tq_double(__ldg(p)); }  // resident tables: another launch's writes

// One tile, rows q0 .. q0 + TQ_ROWS - 1 and columns w0 .. w0 + TQ_COLS - 1, for the group's queries
// j0 .. j0 + NJ - 1 (query j of the group is g0 + j of the launch): its part of their sums is added to sums[].
template <int NJ>
__device__ __forceinline__ void tq_tile(const TQParams& tp, const KeepLayout& kl, const u64* base, const FpMod& m, int q0, int w0,
                                        int g0, int j0, const double* Qs, double* sums) {
    auto at = [&](int j) { return g0 + j; };
    const int lane = threadIdx.x & 31, d0 = tp.d0;
    const u64* inv = base + kl.inv;
    const u64* tri = base + kl.tri + w0 + lane;
    const int qe = min(q0 + TQ_ROWS - 1, tp.qn[at(j0)]);  // the last row a query needs (sizes descend)
    u64 next[TQ_K];
    auto get = [&](int q) {
        const u64* row = tri + tri_off((size_t)q);
#pragma unroll
        for (int k = 0; k < TQ_K; ++k) {
            const int w = w0 + lane + 32 * k;
            next[k] = w < q && w >= d0 && q <= qe ? __ldg(row + 32 * k) : 0;  // resident tables: another launch's writes
        }
    };
    get(q0);
    // lane r + TQ_ROWS j computes F of row q0 + r for query j0 + j (zero past the query's size)
    double F = 0;
    {
        const int j = NJ > 1 ? j0 + lane / TQ_ROWS : j0, q = q0 + lane % TQ_ROWS, nj = tp.qn[at(j)], Mj = tp.qM[at(j)];
        if (q <= nj) {
            F = fp_mulmod(tq_load(inv + 2 * (size_t)q), tq_load(base + kl.ifact + 2 * (size_t)(nj - q)), m);
            F = fp_mulmod(F, tq_load(base + kl.ifact + 2 * (size_t)(Mj - q)), m);
            F = fp_mulmod(F, fp_pow(Qs[j], (u64)(nj - q), m), m);
        }
    }
    double acc[NJ][TQ_K];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int k = 0; k < TQ_K; ++k) acc[j][k] = 0;
#pragma unroll 1
    for (int r = 0; r < TQ_ROWS && q0 + r <= qe; ++r) {
        double x[TQ_K];
#pragma unroll
        for (int k = 0; k < TQ_K; ++k) x[k] = tq_double(next[k]);
        get(q0 + r + 1);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const double f = __shfl_sync(0xffffffffu, F, r + TQ_ROWS * j);
#pragma unroll
            for (int k = 0; k < TQ_K; ++k) acc[j][k] = fp_add(acc[j][k], fp_mulmod(x[k], f, m));
        }
        if ((r & 7) == 7)  // at most eight terms below 0.67p and the sum below 0.51p
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int k = 0; k < TQ_K; ++k) acc[j][k] = fp_red(acc[j][k], m);
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int Mj = tp.qM[at(j0 + j)];
        double y = 0;
#pragma unroll
        for (int k = 0; k < TQ_K; ++k) {
            const int w = w0 + lane + 32 * k;  // columns at or past the query's size hold zero
            const double c = w < qe && w < Mj ? tq_load(inv + 2 * (size_t)(Mj - w)) : 0.0;
            y = fp_add(y, fp_mulmod(fp_red(acc[j][k], m), c, m));  // eight below 0.65p
        }
        y = fp_red(y, m);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            y = fp_add(y, __shfl_xor_sync(0xffffffffu, y, o));
            if (o == 4) y = fp_red(y, m);
        }
        if (lane == 0) sums[j0 + j] = fp_red(fp_add(sums[j0 + j], y), m);
    }
    __syncwarp();
}

// A cluster of S CTAs per prime and group: CTA (b G + g) S + s is CTA s of prime b and group g.  ALL: a
// warp takes all the group's queries of a tile (W >= J; one kernel for both ways of dealing ran 1.4 % slower).
template <bool ALL>
__global__ void __launch_bounds__(TQ_THREADS, TQ_PER_SM) k_table_query(const __grid_constant__ TQParams tp) {
    extern __shared__ __align__(16) double tq_sm[];
    const int S = tp.S, G = tp.G, s = blockIdx.x % S, g = blockIdx.x / S % G, b = blockIdx.x / S / G;
    const int J = tp.J / G + (g < tp.J % G), g0 = tp.J / G * g + min(g, tp.J % G);  // the group's queries
    auto at = [&](int j) { return g0 + j; };
    const int t = threadIdx.x, warp = t >> 5;
    if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // waited for before the first remote store
    double* Qs = tq_sm;                    // [J] candidate sets per item
    double* sums = tq_sm + J;              // [TQ_WARPS][J]
    double* all = sums + TQ_WARPS * J;     // [S][J], in the cluster's first CTA
    const u64 P = tp.primes[b];
    FpMod m;
    m.p = tq_double(P), m.pinv = 1.0 / m.p;
    const KeepLayout kl = make_keep_layout(tp.n, tp.F);
    const u64* base = tp.keep + (size_t)b * tp.keep_words;
    const u64 *fact = base + kl.fact, *ifact = base + kl.ifact;
    for (int j = t; j < J; j += TQ_THREADS) {
        const int Mj = tp.qM[at(j)];
        Qs[j] = tp.model == MODEL_REPLACEMENT
                    ? fp_pow((double)Mj, (u64)tp.d, m)
                    : fp_mulmod(fp_mulmod(tq_load(fact + 2 * (size_t)Mj), tq_load(ifact + 2 * (size_t)tp.d), m), tq_load(ifact + 2 * (size_t)(Mj - tp.d)), m);
    }
    for (int k = t; k < TQ_WARPS * J; k += TQ_THREADS) sums[k] = 0;
    __syncthreads();
    // (tile, W queries) units, the last rows first, dealt to the cluster's warps in turn
    const int nw = S * TQ_WARPS, me = warp * S + s;
    int dealt = 0, jn = 0;  // jn: queries that have row q0
    for (int blk = (tp.qn[g0] - 1) / TQ_ROWS; blk >= 0; --blk) {
        const int q0 = 1 + TQ_ROWS * blk, tiles = (min(q0 + TQ_ROWS - 1, tp.qn[g0]) + TQ_COLS - 1) / TQ_COLS;  // columns 0 .. q0 + TQ_ROWS - 2
        if (q0 + TQ_ROWS - 1 <= tp.d0) break;
        if constexpr (ALL) {
            for (int c = (me - dealt % nw + nw) % nw; c < tiles; c += nw)
                for (int j = 0; j < J && tp.qn[g0 + j] >= q0;) {
                    if (j + 1 < J && tp.qn[g0 + j + 1] >= q0) tq_tile<2>(tp, kl, base, m, q0, c * TQ_COLS, g0, j, Qs, sums + warp * J), j += 2;
                    else tq_tile<1>(tp, kl, base, m, q0, c * TQ_COLS, g0, j, Qs, sums + warp * J), j += 1;
                }
            dealt += tiles;
        } else {
            while (jn < J && tp.qn[g0 + jn] >= q0) ++jn;
            const int parts = (jn + tp.W - 1) / tp.W, units = tiles * parts;
            for (int u = (me - dealt % nw + nw) % nw; u < units; u += nw) {
                const int c = u / parts, j = (u - c * parts) * tp.W;
                if (tp.W > 1 && j + 1 < jn) tq_tile<2>(tp, kl, base, m, q0, c * TQ_COLS, g0, j, Qs, sums + warp * J);
                else tq_tile<1>(tp, kl, base, m, q0, c * TQ_COLS, g0, j, Qs, sums + warp * J);
            }
            dealt += units;
        }
    }
    __syncthreads();
    if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA of the cluster has started
    for (int j = t; j < J; j += TQ_THREADS) {
        double a = 0;
        for (int w = 0; w < TQ_WARPS; ++w) a = fp_add(a, sums[w * J + j]);  // eight below 0.51p
        a = fp_red(a, m);
        if (S == 1) all[j] = a;
        else {
            u32 ra;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((u32)__cvta_generic_to_shared(all + s * J + j)), "r"(0));
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(a) : "memory");
        }
    }
    if (S == 1) __syncthreads();
    else {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (s) return;
    for (int j = t; j < J; j += TQ_THREADS) {  // N_bad = M! n! sum of the terms
        double a = 0;
        for (int c = 0; c < S; ++c) a = fp_add(a, all[c * J + j]);
        a = fp_mulmod(fp_red(a, m), tq_load(fact + 2 * (size_t)tp.qn[at(j)]), m);
        a = fp_mulmod(a, tq_load(fact + 2 * (size_t)tp.qM[at(j)]), m);
        tp.out[(size_t)b * tp.out_stride + tp.qi[at(j)]] = fp_canon(a, m);
    }
}

}  // namespace cfb
