// One-table suffix-table engine: the per-prime build of V[p][v] and the nbad(n, M) queries,
// written as a sequence of block-wide phases so one CTA owns one prime from setup to residues.
//
// Reference semantics (zcy05331/Cuckoo-Failure):
//   include/cuckoo/single_table.hpp:80-119,178-229  the algorithm (two 1/t convolutions per step)
//   fast/cuckoo_fast.cu:145-243                      stage bodies (Stage1Pre/Post, Stage2Pre/Post)
//   fast/cuckoo_fast.cu:306-323,877-890              query sums and the Horner finish
//
// Design (B200, one CTA per prime, persistent over all steps v = 1 .. n-1):
//   * the length-L transform lives in shared memory between radix-2^R register passes;
//   * primes below 2^50 compute in double precision (prime_fp.cuh, fparith.cuh), primes below 2^62
//     with 64-bit integers (prime_wide.cuh); this file holds what both share;
//   * the stage factors are folded into what is stored, so stage 1 needs no multiply on input:
//       Vs[p][w] = V[p][w] / (w! (p-1-w)! (p-1)!)        (stored V)
//       Ss[v][q] = S[v][q] / (q! (v-q)! v!)              (stored S)
//     which turns the reference's stage relations into
//       stage 1:  Ss[v'][v] = D[v'-v] inv[v] conv(Vs[v][.])[v'],            D[k] = 1/k!^2
//       stage 2:  Vs[p][v]  = g^p D[p-v-1] (D[v] - p conv(Ss[v][q] g^-q)[p])
//       query:    out(q)    = (q-1)! sum_w Vs[q][w] / (M - w)
//   * the powers g^p and g^-q of a step come from a small per-step table of powers in shared memory
//     (each thread holds the entries t + k T);
//   * the queries are evaluated on the fly from the stage-1 input rows (the same U[w] the
//     reference's k_query builds), over the row's live entries only; each warp leaves its partial
//     sum in shared memory and, after a barrier of the transform, a thread per query folds the
//     row's partials into one word, so a batch needs no separate pass over V and no barrier of its
//     own per row.
//
// The kernel code runs through an Exec policy: on the GPU `each` is the calling thread and
// `sync` is __syncthreads; a CPU harness (tests) runs the same phases thread by thread.
#pragma once
#include "fparith.cuh"
#include "modarith.cuh"

namespace cfb {

enum { MODEL_SUBSET = 0, MODEL_REPLACEMENT = 1 };

// Scheduling controls for the hot loops.  Constant tables are interleaved (value, companion)
// pairs fetched with one 16-byte load.  `ld_pair` is a volatile load and `pin` an empty volatile
// statement that consumes a result: a load placed after a pin cannot be hoisted above the work
// that produced the pinned value, which bounds how many constants are in flight (registers).
//
// L2 policy: the per-prime constant tables are re-read every step and are loaded with an
// evict-last hint; the rows and column tiles of V and S stream through once per step and use
// evict-first, so they do not push the tables out of L2.  Tables, V, S and the tiles are all written
// by the kernel itself, so they are read with plain coherent loads, never through the read-only path
// (ld.global.nc, __ldg): a read-only load is not ordered after the barrier that follows the write.
// With read-only loads the 2^11 kernel at two CTAs per SM read table words of setup before they were
// written (wrong residues on the first launch over a workspace).
#if defined(__CUDA_ARCH__)
CF_HD void pin(u64& v) { asm volatile("" : "+l"(v)); }
CF_HD void pin_int(int& v) { asm volatile("" : "+r"(v)); }
CF_HD void pin_word(u32& v) { asm volatile("" : "+r"(v)); }
CF_HD u64 policy_keep() {
    u64 pol;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
CF_HD u64 policy_stream() {
    u64 pol;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
CF_HD void ld_pair(const u64* p, u64& a, u64& b) {
    asm volatile("ld.global.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;" : "=l"(a), "=l"(b) : "l"(p), "l"(policy_keep()));
}
CF_HD u64 ld_stream(const u64* p) {
    u64 v;
    asm volatile("ld.global.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(policy_stream()));
    return v;
}
CF_HD void st_stream(u64* p, u64 v) { asm volatile("st.global.L2::cache_hint.u64 [%0], %1, %2;" ::"l"(p), "l"(v), "l"(policy_stream())); }
// one full 32-byte sector (p 32-byte aligned)
CF_HD void st_stream4(u64* p, u64 a, u64 b, u64 c, u64 d) {
    asm volatile("st.global.L2::cache_hint.v4.u64 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d),
                 "l"(policy_stream()));
}
CF_HD void ld_pair_shared(const u64* p, u64& a, u64& b) {
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"((u32)__cvta_generic_to_shared(p)));
}
#else
CF_HD u64 ld_stream(const u64* p) { return *p; }
CF_HD void st_stream(u64* p, u64 v) { *p = v; }
CF_HD void st_stream4(u64* p, u64 a, u64 b, u64 c, u64 d) { p[0] = a, p[1] = b, p[2] = c, p[3] = d; }
CF_HD void ld_pair_shared(const u64* p, u64& a, u64& b) { a = p[0], b = p[1]; }
CF_HD void pin(u64&) {}
CF_HD void pin_int(int&) {}
CF_HD void pin_word(u32&) {}
CF_HD void ld_pair(const u64* p, u64& a, u64& b) { a = p[0], b = p[1]; }
#endif
// Loads of data a kernel writes itself.  A CTA alone reads its own writes through L1.  In a cluster
// (CG), data another CTA wrote in this launch is read from L2 (.cg), where the writer's release at
// the cluster barrier has made it visible; L1 lines of an earlier read (block cells and tiles are
// reused) would not hold the new values.
template <bool CG>
CF_HD void ldp(const u64* p, u64& a, u64& b) {
#if defined(__CUDA_ARCH__)
    if constexpr (CG)
        asm volatile("ld.global.cg.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;" : "=l"(a), "=l"(b) : "l"(p), "l"(policy_keep()));
    else ld_pair(p, a, b);
#else
    a = p[0], b = p[1];
#endif
}
template <bool CG>
CF_HD u64 lds(const u64* p) {
#if defined(__CUDA_ARCH__)
    if constexpr (CG) {
        u64 v;
        asm volatile("ld.global.cg.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(policy_stream()));
        return v;
    } else return ld_stream(p);
#else
    return *p;
#endif
}
template <bool CG>
CF_HD u64 ldc(const u64* p) {
#if defined(__CUDA_ARCH__)
    if constexpr (CG) {
        u64 v;
        asm volatile("ld.global.cg.u64 %0, [%1];" : "=l"(v) : "l"(p));
        return v;
    } else return *p;
#else
    return *p;
#endif
}
// Lambdas that index the register array must be inlined, or the array goes to local memory.
#define CF_INL __attribute__((always_inline))
// Compile-time slot index handed to the bodies below (so register-array indices are constants).
template <int V>
struct IC {
    static constexpr int value = V;
    CF_HD constexpr operator int() const { return V; }
};
// Unrolled loop over N units with a bounded window: body(IC<J>) pins its inputs and computes unit
// J; done(IC<J>) pins unit J's outputs and is issued right after body(IC<J + K>).  Since volatile
// statements keep their order, unit J + K + 1 cannot start before unit J has finished: at most
// K + 1 units are in flight, which bounds the registers the compiler's interleaving may use.
template <int N, int K, int J, class B, class Dn>
CF_HD void window_step(B& body, Dn& done) {
    if constexpr (J < N + K) {
        if constexpr (J < N) body(IC<J>{});
        if constexpr (J >= K && J - K < N) done(IC<J - K>{});
        window_step<N, K, J + 1>(body, done);
    }
}
template <int N, int K, class B, class Dn>
CF_HD void window(B&& body, Dn&& done) {
    window_step<N, K, 0>(body, done);
}
// Per-slot constant pairs over a window: slot J's pair addr(IC<J>) is loaded D slots ahead.
template <int N, int D, int K, bool CG = false, class A, class F, class Dn>
CF_HD void pipe_pairs(A&& addr, F&& apply, Dn&& done) {
    u64 ra[D + 1], rb[D + 1];
    window<D, 0>([&](auto jc) CF_INL {
        constexpr int j = decltype(jc)::value;
        if constexpr (j < N) ldp<CG>(addr(jc), ra[j], rb[j]);
    }, [&](auto) CF_INL {});
    window<N, K>(
        [&](auto jc) CF_INL {
            constexpr int j = decltype(jc)::value;
            if constexpr (j + D < N) ldp<CG>(addr(IC<j + D>{}), ra[(j + D) % (D + 1)], rb[(j + D) % (D + 1)]);
            apply(jc, ra[j % (D + 1)], rb[j % (D + 1)]);
        },
        done);
}
// The same over the slots for which live(IC<J>) holds (a warp-uniform test): the others issue
// neither their constant load nor their unit.
template <int N, int D, int K, bool CG = false, class Lv, class A, class F, class Dn>
CF_HD void pipe_pairs_live(Lv&& live, A&& addr, F&& apply, Dn&& done) {
    u64 ra[D + 1] = {}, rb[D + 1] = {};
    window<D, 0>([&](auto jc) CF_INL {
        constexpr int j = decltype(jc)::value;
        if constexpr (j < N)
            if (live(jc)) ldp<CG>(addr(jc), ra[j], rb[j]);
    }, [&](auto) CF_INL {});
    window<N, K>(
        [&](auto jc) CF_INL {
            constexpr int j = decltype(jc)::value;
            if constexpr (j + D < N)
                if (live(IC<j + D>{})) ldp<CG>(addr(IC<j + D>{}), ra[(j + D) % (D + 1)], rb[(j + D) % (D + 1)]);
            if (live(jc)) apply(jc, ra[j % (D + 1)], rb[j % (D + 1)]);
        },
        done);
}
#ifndef CF_PIPE_D
#define CF_PIPE_D 4
#endif
#ifndef CF_WIN_K
#define CF_WIN_K 3
#endif
constexpr int PIPE_D = CF_PIPE_D;  // constants loaded ahead
constexpr int WIN_K = CF_WIN_K;    // units in flight beyond the current one

// Transform geometry: L = 2^LG entries, T threads holding E = 2^R entries each.  The LG levels
// are done in passes of R levels (the last pass may have fewer); between passes the entries go
// through shared memory.
//
// Clusters (LC > 0): the T threads are spread over C = 2^LC CTAs of CT = T / C threads, thread t
// being thread t % CT of the cluster's CTA t / CT.  Pass 0 holds index t + jT in slot j (a
// column of every one of the E blocks of L / E entries); after it every later pass works inside one
// block, and CTA c holds blocks c E / C .. (c + 1) E / C - 1 (E >= C), i.e. the indices
// [c L / C, (c + 1) L / C).  So the entries cross between CTAs only after the first forward pass
// and before the last inverse pass, through distributed shared memory.
template <int LG_, int R_, int LC_ = 0>
struct Geo {
    static constexpr int LG = LG_, R = R_, LC = LC_;
    static constexpr int L = 1 << LG, E = 1 << R, T = 1 << (LG - R);
    static constexpr int C = 1 << LC, CT = T >> LC, LCN = L >> LC;  // CTAs, threads and entries per CTA
    static constexpr int NP = (LG + R - 1) / R;  // number of passes
    static constexpr int SWZ = R > 4 ? R : 4;    // shared-memory swizzle shift
    static constexpr int NW = (CT + 31) / 32;    // warps per CTA
    static_assert(C == 1 || (E >= C && CT % 128 == 0 && NP >= 3), "a cluster needs E >= C, whole warp quarters and 3 passes");
    CF_HD static constexpr int pass_b(int p) { return LG - (p + 1) * R > 0 ? LG - (p + 1) * R : 0; }
    CF_HD static constexpr int pass_r(int p) { return LG - p * R - pass_b(p); }
    // index of the entry held in slot j by thread t during pass p
    CF_HD static int idx(int p, int t, int j) {
        if (p == NP - 1) return t * E + j;
        const int b = pass_b(p);
        return ((t >> b) << (b + R)) + (t & ((1 << b) - 1)) + (j << b);
    }
    CF_HD static int swz(int i) { return i ^ ((i >> SWZ) & 15); }
    static constexpr int R_LAST = LG - (NP - 1) * R;  // levels of the last pass
};

CF_HD u64 red2(u64 x, u64 m) { return x >= m ? x - m : x; }  // [0, 2m) -> [0, m)

// V and S are read by rows (a step reads row v) but produced by columns (step v writes column v).
// The columns of the current TILE steps are staged column-major in VS / SS (contiguous writes) and
// moved into row storage every TILE steps, the scheme of fast/cuckoo_fast.cu:133-144, 227-243.
//
// Row storage is made of TILE x TILE blocks: block (P, W) holds rows 1 + 16P .. 16 + 16P and
// columns 1 + 16W .. 16 + 16W, row-major (a row's 16 entries are one 128-byte line).  Only blocks
// below the diagonal (W < P) are stored; a row's own group of columns is read from the staging
// tile.  Block (P, W) is written when tile W is flushed and dead once the steps of tile P have read
// its rows (row n of V stays until the finish), so at most (k + 1)(G - 1 - k) blocks are live
// after flush k, G = number of row groups.  The blocks map onto an (G - h) x h array of cells,
// h = ceil(G / 2), that is exactly that peak:
//   W < h <= P : cell (P - h, W)          the rectangle, live through the middle of the run
//   P < h      : cell (W, P)              rows read before step 16h; their cell's rectangle block
//                                        is written at flush P, after its last read
//   h <= W     : cell (W - h, P - h - 1)  written from flush h on, into cells whose rectangle
//                                        block was read in tile W, before that flush
// so a prime's V and S take about n^2 / 4 words each instead of n^2 / 2 for packed triangles.
constexpr int TILE = 16;
CF_HD int grp(int x) { return (x - 1) >> 4; }  // row / column group of index x >= 1
CF_HD int block_h(int n) { return (((n - 1) >> 4) + 2) >> 1; }  // h = ceil(G / 2), G = grp(n) + 1
CF_HD size_t block_count(int n) {
    if (n < 1) return 0;
    const size_t G = (size_t)grp(n) + 1, h = (size_t)block_h(n);
    return (G - h) * h;
}
CF_HD size_t block_cell(int P, int W, int h) {  // W < P
    if (P < h) return (size_t)W * h + P;
    if (W < h) return (size_t)(P - h) * h + W;
    return (size_t)(W - h) * h + (P - h - 1);
}
// word offset of entry (row r, column c), grp(c) < grp(r), inside a block pool
CF_HD size_t blk_off(int r, int c, int h) {
    return (block_cell(grp(r), grp(c), h) << 8) + ((size_t)((r - 1) & 15) << 4) + (size_t)((c - 1) & 15);
}

// Per-prime global workspace, in 64-bit words (every table 256-byte aligned).
// Tables marked "pairs" hold (value, Shoup companion) interleaved: entry k at [2k], [2k+1].
struct Layout {
    size_t V, S, VS, SS, fact, ifact, inv, D, Gm, hat, ps, total;
    size_t WL[8];  // pass-0 twiddles by level: WL[s] holds pairs w^(u 2^s), u = 0 .. L/2^(s+1)
};
CF_HD size_t lay_take(size_t& at, size_t cnt) {
    const size_t r = at;
    at += (cnt + 31) & ~(size_t)31;
    return r;
}
// nw = warps per CTA: query partial sums are kept per warp.  C: CTAs per prime (each keeps its own
// row sums of the queries).
CF_HD Layout make_layout(int n, int F, int L, int J, int nw, int R, int C = 1) {
    Layout o;
    size_t at = 0;
    o.V = lay_take(at, block_count(n) << 8);         // rows p = 1..n, entries w = 1..p-1 (blocks)
    o.S = lay_take(at, block_count(n) << 8);         // rows v = 1..n-1, entries q = 1..v (blocks)
    o.VS = lay_take(at, (size_t)TILE * (n + 1));      // column tiles, [column - v0][row]
    o.SS = lay_take(at, (size_t)TILE * (n + 1));
    o.fact = lay_take(at, 2 * ((size_t)F + 1));   // pairs: k!
    o.ifact = lay_take(at, 2 * ((size_t)F + 1));  // pairs: 1/k!
    o.inv = lay_take(at, 2 * ((size_t)F + 1));    // pairs: 1/k
    o.D = lay_take(at, 2 * ((size_t)n + 1));      // pairs: 1/k!^2
    o.Gm = lay_take(at, 2 * ((size_t)n + 1));     // (g(v), 1/g(v)) in Montgomery form, v = 0 .. n
    for (int l = 0; l < 8; ++l) o.WL[l] = l < R ? lay_take(at, 2 * (((size_t)L >> (l + 1)) + 1)) : 0;  // pairs
    o.hat = lay_take(at, 2 * (size_t)L);          // pairs: spectrum of the kernel 1/t, times 1/L
    o.ps = lay_take(at, (size_t)C * J * (n + 1));  // [C][J][n+1] row sums per query (per CTA of the prime)
    (void)nw;
    o.total = at;
    return o;
}
CF_HD int tile_v0(int v) { return 1 + TILE * ((v - 1) / TILE); }  // first column of v's tile

// Resident tables (serving): per prime, the whole V as a packed triangle (row p at p(p-1)/2,
// entries w = 0..p-1, entries w < d0 unused) and the pair tables fact, ifact, inv up to F, so that
// later queries (n' <= n, M' <= F) need no rebuild.
struct KeepLayout {
    size_t tri, fact, ifact, inv, total;
};
CF_HD KeepLayout make_keep_layout(int n, int F) {
    KeepLayout k;
    size_t at = 0;
    k.tri = lay_take(at, (size_t)n * (n + 1) / 2);
    k.fact = lay_take(at, 2 * ((size_t)F + 1));
    k.ifact = lay_take(at, 2 * ((size_t)F + 1));
    k.inv = lay_take(at, 2 * ((size_t)F + 1));
    k.total = at;
    return k;
}
CF_HD size_t tri_off(size_t p) { return p * (p - 1) / 2; }  // V[p][w] at tri + tri_off(p) + w

// Launch parameters shared by all CTAs of a batch (one CTA per prime).
struct KParams {
    const u64* primes;  // [B]
    int B, n, F, d, d0, model, J;
    const int* qn;      // [J] query sizes n_j <= n
    const int* qM;      // [J] query table sizes M_j <= F
    u64* ws;            // workspace base
    size_t ws_words;    // words per prime
    Layout lay;         // offsets inside a prime's workspace
    u64* out;           // [B][J] residues, or out[qout[j]] when qout is set
    int* err;           // device error word (0 = ok)
    const long long* qout = nullptr;  // [J] output index of each query (work-queue items), or null
    u64* keep = nullptr;  // resident tables [B][keep_words] (serving builds), or null
    size_t keep_words = 0;
    int JC = 0;  // queries whose partial sums shared memory holds at a time (0: all J)
    u64 p_lo = 0;  // an integer-kernel launch leaves primes below it alone (another launch's)
};

// Error codes recorded in *err by the kernel.
enum { KERR_NONE = 0, KERR_NO_ROOT = 1 };

// Shared memory per CTA, in 64-bit words.  K: the kernel for primes below 2^50 (0), below 2^62 (1), or
// room for either (2).
template <class G, int K = 2>
struct Smem {
    // [L] transform exchange by index (swizzled); a CTA of a cluster holds the LCN indices of its
    // blocks there (by index - c LCN) and, at X0, pass 0's column layout: slot j of thread t at
    // X0 + t % CT + j CT, written by the CTAs that finish the inverse transform's upper levels
    static constexpr int X = 0;
    static constexpr int X0 = G::C > 1 ? G::LCN : 0;
    // [2 CT + 64] reduction and scan scratch of setup and finish, when no transform is under way
    static constexpr int RED = 0, RED_N = 2 * G::CT + 64;
    static constexpr int XN = G::C > 1 ? 2 * G::LCN : (G::L > RED_N ? G::L : RED_N);
    static_assert(XN >= RED_N, "the scratch shares the exchange area");
    static constexpr int MISC = XN;                   // [16] modulus constants and scalars
    // twiddles of the passes that do not read theirs from global or tensor memory:
    // wide: pairs w^(k 2^R), k = 0 .. L/2^(R+1); 2^50: FTN forward ones, then T - 1 inverse ones
    static constexpr int TWS = MISC + 16;
    static constexpr int TWS_N = (G::L >> (G::R + 1)) + 1;
    static constexpr int FTN = G::C == 1 ? 1 << (G::LG - G::R_LAST - 1) : G::E - 1 + ((1 << (G::LG - G::R_LAST)) - G::E) / G::C;
    static constexpr int TW_WIDE = 2 * TWS_N, TW_FP = FTN + G::T;
    static constexpr int TW_N = K == 0 ? TW_FP : K == 1 ? TW_WIDE : (TW_FP > TW_WIDE ? TW_FP : TW_WIDE);
    // [2][PW_STRIDE] powers of 1/g(v) and g(v) for stage 2, rebuilt every step (power_tables)
    static constexpr int PW = TWS + ((TW_N + 1) & ~1);
    static constexpr int PW_STRIDE = 104;
    static constexpr int WORDS = PW + 2 * PW_STRIDE;
    // A cluster's CTAs take more than half an SM's shared memory, so no two share an SM (a CTA
    // waiting for tensor memory held by another CTA of its own cluster would never get it).
    static constexpr size_t BYTES = G::C > 1 && WORDS * 8 < 120 * 1024 ? 120 * 1024 : (size_t)WORDS * 8;
    // [JC][NW] per-warp query partial sums of the current row, after the fixed part (the launch's
    // dynamic shared memory is BYTES + 8 JC NW)
    static constexpr int QS = WORDS;
    static constexpr size_t bytes_for(int J) { return BYTES + (size_t)8 * J * G::NW; }
};
enum { MI_P = 0, MI_PINV = 1, MI_R1 = 2, MI_R2 = 3, MI_ONEQ = 4, MI_ROOT = 5, MI_LINV = 6, MI_TMEM = 7, MI_R1Q = 8, MI_PD = 9, MI_PINVD = 10, MI_NEXT = 11 };
// Slots of a power table (power_tables): h^k at PW_A + k (k < TA), h^(TA k) at PW_B + k (k < TB),
// h^(T j) at PW_J + j (j < E), and h^L at PW_L; for the integer kernels the running products' step
// h^(NCH T) as a plain residue and its Shoup companion at PW_STEP, PW_STEPQ.
enum { PW_A = 0, PW_B = 32, PW_J = 64, PW_STEP = 96, PW_STEPQ = 97, PW_L = 98 };

template <class G>
struct Regs {
    u64 x[G::E];     // the integer kernels' entries
    double f[G::E];  // the double-precision kernels' entries
};
// What the per-prime kernels of both arithmetics share: the prime's workspace and shared memory, row
// loads, the fold of the query partial sums, the tile flush.  K: 0 (double precision), 1 (integers).
template <class G, class X, int K>
struct PrimeBase {
    static constexpr int L = G::L, T = G::T, E = G::E, NP = G::NP, NW = G::NW;
    static constexpr int C = G::C, CT = G::CT, LCN = G::LCN;  // a cluster of C CTAs of CT threads per prime
    static constexpr bool CG = C > 1;  // loads of what other CTAs wrote go to L2 (ldp / lds / ldc)
    typedef Smem<G, K> SM;
    static_assert(NP > 1, "layout 0 must hold index t + jT in slot j of thread t");
    X& ex;
    const KParams& kp;
    int b;      // prime index within the batch
    u64* base;  // this prime's workspace
    u64* sm;    // shared memory
    u64 P;
    int rank_;  // this CTA's rank in its cluster

    // bi: the prime's index in kp.primes (and its output row); slot: its workspace slot (bi if < 0)
    CF_HD PrimeBase(X& e, const KParams& k, int bi, u64* smem, int slot) : ex(e), kp(k), b(bi), sm(smem) {
        P = kp.primes[b];
        base = kp.ws + (size_t)(slot < 0 ? bi : slot) * kp.ws_words;
        rank_ = ex.rank();
    }
    CF_HD int rank() const {
        if constexpr (C == 1) return 0;
        else return rank_;
    }
    CF_HD static int lt(int t) {  // thread index within the CTA
        if constexpr (C == 1) return t;
        else return t & (CT - 1);
    }
    CF_HD void csync() {  // barrier of the whole cluster (of the CTA alone when C = 1)
        if constexpr (C == 1) ex.sync();
        else ex.cluster_sync();
    }
    // workspace tables (offsets live in the kernel parameters, so these hold no registers)
    CF_HD u64* V() const { return base + kp.lay.V; }
    CF_HD u64* S() const { return base + kp.lay.S; }
    CF_HD u64* VS() const { return base + kp.lay.VS; }
    CF_HD u64* SS() const { return base + kp.lay.SS; }
    CF_HD u64* fact() const { return base + kp.lay.fact; }
    CF_HD u64* ifact() const { return base + kp.lay.ifact; }
    CF_HD u64* inv() const { return base + kp.lay.inv; }
    CF_HD u64* D() const { return base + kp.lay.D; }
    CF_HD u64* Gm() const { return base + kp.lay.Gm; }
    CF_HD u64* WL(int l) const { return base + kp.lay.WL[l]; }
    CF_HD u64* hat() const { return base + kp.lay.hat; }
    CF_HD u64* ps() const { return ps_of(rank()); }
    CF_HD u64* ps_of(int c) const { return base + kp.lay.ps + (size_t)c * kp.J * (kp.n + 1); }  // CTA c's row sums
    CF_HD u64* misc() const { return sm + Smem<G>::MISC; }
    CF_HD Mod md() const {  // modulus constants, kept in shared memory
        const u64* m = misc();
        Mod r;
        r.p = m[MI_P], r.pinv = m[MI_PINV], r.r1 = m[MI_R1], r.r2 = m[MI_R2];
        return r;
    }

    // Block sum mod p of the values the CTA's threads left in RED[t] (returned to every thread).
    CF_HD u64 sum_red() {
        u64* red = sm + SM::RED;
        ex.sync();
        ex.reduce_mod(red, CT, P);
        ex.sync();
        return red[CT];
    }

    // Index range [lo, hi] of slot j (layout 0: index t + jT) over the calling thread's warp: the
    // stage loops skip a slot, warp-uniformly, when no lane of the warp needs it.
    CF_HD static void warp_slot_range(int t, int j, int& lo, int& hi) {
        const int tw = t & ~31;
        lo = tw + j * T;
        hi = (T < 32 ? T - 1 : tw + 31) + j * T;
    }

    // Addresses of row r of V or S by slot (layout 0: slot j of thread t holds index i = t + jT).
    // Columns of earlier groups lie in the blocks, those of r's own group in the staging tile.
    //
    // When T is a multiple of 16 the column group of slot j is W0 + j T/16 and the entry's place in
    // its block is the same for every slot.  The block cell of (P, W) is then linear in W on either
    // side of h (block_cell's three cases): W < h: W a_lo + b_lo; W >= h: W h + b_hi.  Word offsets
    // from the pool fit 32 bits (block_count(65536) 256 = 2^30 words).
    struct Row {
        const u64 *pool, *tl;  // the pool; the tile at the thread's column 0 (slot 0) and row r
        int n, t, v0, h, a_lo, b_lo, b_hi, W0;
        u32 at;
        // first: the first column read from the staging tile
        CF_HD Row(int n_, int t_, const u64* pool_, const u64* tile, int r, int first) : pool(pool_), n(n_), t(t_), v0(first) {
            h = block_h(n);
            const int Pr = grp(r);
            W0 = (t - 1) >> 4;  // -1 for t = 0, whose slot 0 is never in range
            a_lo = Pr < h ? h : 1, b_lo = Pr < h ? Pr : (Pr - h) * h, b_hi = Pr - h - 1 - h * h;
            at = ((u32)((r - 1) & 15) << 4) + (u32)((t - 1) & 15);
            tl = tile + r + (ptrdiff_t)(t - v0) * (n + 1);
            if (T % TILE) at = (u32)r;
        }
        CF_HD const u64* operator()(int j) const {
            const int i = t + j * T;
            if (i >= v0) return tl + (ptrdiff_t)(j * T) * (n + 1);
            if constexpr (T % TILE) return pool + blk_off((int)at, i, h);
            else {
                const int wg = W0 + j * (T / TILE);
                return pool + (((u32)(wg < h ? wg * a_lo + b_lo : wg * h + b_hi) << 8) + at);
            }
        }
    };
    // Row r into the registers: the slot of index i gets entry i for lo <= i < hi, zero elsewhere.
    CF_HD void load_row(int t, u64 (&x)[E], const u64* pool, const u64* tile, int r, int lo, int hi) const {
        const Row row(kp.n, t, pool, tile, r, tile_v0(r));
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int i = t + j * T;
            x[j] = (i >= lo && i < hi) ? lds<CG>(row(j)) : 0;
        }
    }

    // Row q's per-warp partials of queries ja .. jb - 1 (written before a barrier) into ps[j][q], a thread
    // per query.  A query with n_j < q has none: its word of row q is never read.
    // Clusters of the integer kernels: a warp per query, with shuffles.  Their fold stands in every CTA's
    // way to the next cluster barrier (ms a thread per query, a warp; n = 20000, 24 primes: one query 1861,
    // 1844, nine 1991, 1971; 16 primes, 40 queries 2512, 2484; n = 40000, 4 primes: 3800, 3804).  On one CTA
    // a warp per query is the slower form (n = 3000, 128 primes: 129.7, 131.7; n = 16384, 148: 3602, 3648).
    CF_HD void fold_queries(int q, int ja, int jb) {
        const u64* qs = sm + SM::QS;
        ex.each([&](int t, Regs<G>&) CF_INL {
            if constexpr (K == 1 && C > 1) {
                for (int jq = ja + (lt(t) >> 5), lane = t & 31; jq < jb; jq += NW) {
                    const u64 v = lane < NW ? qs[(size_t)(jq - ja) * NW + lane] : 0;
                    ex.warp_sum_store(lt(t), v, P, ps() + (size_t)jq * (kp.n + 1) + q, 0);
                }
                return;
            }
            for (int jq = ja + lt(t); jq < jb; jq += CT) {
                u64 s = 0;
#pragma unroll 4
                for (int w = 0; w < NW; ++w) s = madd(s, qs[(size_t)(jq - ja) * NW + w], P);
                ps()[(size_t)jq * (kp.n + 1) + q] = s;
            }
        });
    }
    // some(ja, jb, where the warps' partials of query ja go) for ranges of the queries, JC at a time: all
    // but the last batch are folded here, the last by fold_last after the caller's next barrier.
    CF_HD int query_batch() const { return kp.JC > 0 && kp.JC < kp.J ? kp.JC : kp.J; }
    template <class F>
    CF_HD void query_batches(int q, F&& some) {
        const int jc = query_batch();
        for (int ja = 0; ja < kp.J; ja += jc) {
            const int jb = ja + jc < kp.J ? ja + jc : kp.J;
            some(ja, jb, sm + SM::QS);
            if (jb < kp.J) {
                ex.sync();
                fold_queries(q, ja, jb);
                ex.sync();
            }
        }
    }
    CF_HD void fold_last(int q) {
        const int jc = query_batch();
        if (kp.J > 0) fold_queries(q, jc == kp.J ? 0 : (kp.J - 1) / jc * jc, kp.J);  // no division where one batch holds all
    }

    // The full tile's columns v0 .. v0 + 15 into row storage, the rows r = t + jT of the warp's threads (rows of
    // later groups only: a row of this tile's group reads these columns from the tile).  The warp wrote
    // the staged columns of these rows itself, so only its own threads need to meet before it.  Other warps
    // may have read the cells written: a block that the flush replaces holds rows of this tile's group, of
    // which row v = v0 + 15 of V was read in step v - 1, and row v of S in stage 1 of this step.  So
    // the flush must stay behind the barriers of step v's second convolution, which every thread
    // passes after that read of S.  Four lanes take a row, four columns each, so a
    // store instruction fills eight whole 128-byte lines (one row per lane wrote a sector of 32 lines:
    // the flush was bound by those).
    CF_HD void flush_rows(int t, int v0) const {
        constexpr int LPR = CT < 32 ? 1 : 4, RW = CT < 32 ? 1 : 8;  // lanes per row, rows of a warp at a time
        const int n = kp.n, d0 = kp.d0, h = block_h(n), lane = t & 31;
        const size_t cs = (size_t)n + 1;  // tile column stride
        const int cS = d0 + 1 > v0 ? d0 + 1 - v0 : 0, cV = d0 > v0 ? d0 - v0 : 0;
        const int r0 = CT < 32 ? t : (t & ~31) + lane / LPR, c0 = CT < 32 ? 0 : (lane % LPR) * (TILE / LPR);
        for (int rb = (v0 + TILE - (CT < 32 ? t : (t & ~31) + 31) + T - 1) / T * T; r0 + rb <= n; rb += T) {
#pragma unroll
            for (int g = 0; g < (CT < 32 ? 1 : 32 / RW); ++g) {
                const int r = r0 + rb + g * RW;
                if (r < v0 + TILE || r > n) continue;
                const size_t off = blk_off(r, v0, h);  // columns v0 + c at off + c
                if (cS == 0) {
                    const u64 *sS = SS() + (r < n ? r : n - 1) + c0 * cs, *sV = VS() + r + c0 * cs;
                    u64 a[TILE / LPR], b[TILE / LPR];
#pragma unroll
                    for (int c = 0; c < TILE / LPR; ++c) a[c] = lds<CG>(sS + c * cs), b[c] = lds<CG>(sV + c * cs);
#pragma unroll
                    for (int c = 0; c < TILE / LPR; c += 4) {
                        if (r < n) st_stream4(S() + off + c0 + c, a[c], a[c + 1], a[c + 2], a[c + 3]);
                        st_stream4(V() + off + c0 + c, b[c], b[c + 1], b[c + 2], b[c + 3]);
                    }
                } else {  // rows r < n of S: entries q = v0 .. v, written for q > d0; of V: w = v0 .. v, written for w >= d0
                    const int ce = c0 + TILE / LPR;
                    for (int c = c0 > cS ? c0 : cS; c < ce && r < n; ++c) st_stream(S() + off + c, lds<CG>(SS() + r + c * cs));
                    for (int c = c0 > cV ? c0 : cV; c < ce; ++c) st_stream(V() + off + c, lds<CG>(VS() + r + c * cs));
                }
            }
        }
    }
    // The end of step v: the tile's columns go to the rows when it is full (or the last), and row v + 1
    // is complete after the barrier.  keep(v0, v): copies the tile's columns of a serving build.
    template <class F>
    CF_HD void end_step(int v, F&& keep) {
        // columns of S and of V in flight per thread: fewer where registers bound the threads (1024 of them,
        // or a warp or less to a CTA, where 16 columns took 160 registers and four CTAs fewer fit an SM)
        constexpr int FL = CT >= 1024 ? 8 : CT <= 32 ? 4 : TILE;
        const int n = kp.n, d0 = kp.d0;
        const int v0 = tile_v0(v);
        if (v - v0 == TILE - 1 || v == n - 1) {  // move the tile's columns v0 .. v into the rows
            csync();
            // Rows of later groups only: a row of this tile's group reads these columns from the tile.
            // A full tile's 2 FL loads of a row go out before its first store (the stores wait for
            // them in order; four at a time left the flush waiting on memory latency).
            ex.each([&](int t, Regs<G>&) CF_INL {
                const int cnt = v - v0 + 1, h = block_h(n);
                const size_t cs = (size_t)n + 1;  // tile column stride
                const int cS = d0 + 1 > v0 ? d0 + 1 - v0 : 0, cV = d0 > v0 ? d0 - v0 : 0;
                // rows r < n of S: entries q = v0 .. v, written for q > d0; rows of V: entries w = v0 .. v,
                // written for w >= d0
                if (cnt == TILE && cS == 0) {
                    for (int r = v0 + TILE + t; r <= n; r += T) {
                        const size_t off = blk_off(r, v0, h);  // columns v0 + c at off + c
                        const u64 *sS = SS() + (r < n ? r : n - 1), *sV = VS() + r;
                        u64 a[FL], b[FL];
#pragma unroll
                        for (int c0 = 0; c0 < TILE; c0 += FL) {
#pragma unroll
                            for (int c = 0; c < FL; ++c) a[c] = lds<CG>(sS + (c0 + c) * cs), b[c] = lds<CG>(sV + (c0 + c) * cs);
#pragma unroll
                            for (int c = 0; c < FL; c += 4) {
                                if (r < n) st_stream4(S() + off + c0 + c, a[c], a[c + 1], a[c + 2], a[c + 3]);
                                st_stream4(V() + off + c0 + c, b[c], b[c + 1], b[c + 2], b[c + 3]);
                            }
                        }
                    }
                } else {
                    for (int r = v0 + TILE + t; r <= n; r += T) {
                        const size_t off = blk_off(r, v0, h);
                        for (int c = cS; c < cnt && r < n; ++c) st_stream(S() + off + c, lds<CG>(SS() + r + c * cs));
                        for (int c = cV; c < cnt; ++c) st_stream(V() + off + c, lds<CG>(VS() + r + c * cs));
                    }
                }
            });
            if (kp.keep) keep(v0, v);
        }
        csync();  // row v + 1 is read by the next step
    }
    // Serving builds: the tile's columns v0 .. v of V, for every row below them, into the resident
    // packed triangle; word(w) is the canonical residue of a stored word.
    template <class F>
    CF_HD void keep_tile(int v0, int v, F&& word) {
        const int n = kp.n, d0 = kp.d0, cnt = v - v0 + 1;
        u64* tri = kp.keep + (size_t)b * kp.keep_words;  // the triangle sits at offset 0
        ex.each([&](int t, Regs<G>&) CF_INL {
            for (int r = v0 + 1 + t; r <= n; r += T) {
                u64* dst = tri + tri_off(r);
                const u64* src = VS() + r;
                for (int c = 0; c < cnt; ++c) {
                    const int w = v0 + c;
                    if (w >= d0 && w < r) dst[w] = word(lds<CG>(src + (size_t)c * (n + 1)));
                }
            }
        });
    }
};

// The engine of one prime.  W = false: primes below 2^50 (the fixed list of fast/cuckoo_fast.cu with
// FP_RB = 52), in double precision.  W = true: primes below 2^62 (the list of the FP_RB = 64 build),
// with 64-bit integers.
template <class G, class X, bool W = false>
struct PrimeRun;

}  // namespace cfb

#include "prime_fp.cuh"
#include "prime_wide.cuh"
