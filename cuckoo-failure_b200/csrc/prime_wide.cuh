// The per-prime kernel for primes below 2^62 (the list of the FP_RB = 64 build), in 64-bit integers.
// Every multiplication by a stored constant is a Shoup product with a precomputed companion, products
// of two varying values are Montgomery products.  With 8p beyond 2^64 every transform value stays in
// [0, 2p), and the few products whose lazy factor could reach 2^62 take a canonical one.  The
// powers g^p and g^-q of a step are running Montgomery products per thread, started from the step's
// table of powers.
#pragma once
#include "suffix_engine.cuh"

namespace cfb {

template <class G, class X>
struct PrimeRun<G, X, true> : PrimeBase<G, X, 1> {
    typedef PrimeBase<G, X, 1> Base;
    static constexpr int L = G::L, T = G::T, E = G::E, NP = G::NP, NW = G::NW, C = G::C, CT = G::CT, LCN = G::LCN;
    static constexpr bool CG = C > 1;
    typedef typename Base::SM SM;
    using Base::ex;
    using Base::kp;
    using Base::b;
    using Base::base;
    using Base::sm;
    using Base::P;
    using Base::rank;
    using Base::lt;
    using Base::csync;
    using Base::V;
    using Base::S;
    using Base::VS;
    using Base::SS;
    using Base::fact;
    using Base::ifact;
    using Base::inv;
    using Base::D;
    using Base::Gm;
    using Base::WL;
    using Base::hat;
    using Base::ps;
    using Base::ps_of;
    using Base::misc;
    using Base::md;
    using Base::sum_red;
    using Base::warp_slot_range;
    using Base::load_row;
    using Base::fold_last;
    // L = 2^14 (1024 threads x 16 entries): the kernel spectrum lives in tensor memory, each
    // thread's 16 (value, companion) pairs in its own 64 columns (all 512 columns of the SM's 128
    // lanes); smaller transforms, several CTAs to an SM, read it from global.  A cluster's CTAs
    // (one per SM) keep their blocks' part of it in 4 E CT / 128 columns.
    static constexpr bool TM = (T == 1024 && E == 16) || (T == 512 && E == 32) || (C > 1 && 4 * E * (CT / 128) <= 512);
    // Constants in flight and units in flight of the hot loops.  At 1024 threads (64 registers each)
    // the shallowest schedule spills least and measured fastest (49.7 vs 48.9 prime-residues/s).
    static constexpr int PD = CT >= 1024 ? 1 : PIPE_D, WK = CT >= 1024 ? 1 : WIN_K;
    CF_HD PrimeRun(X& e, const KParams& k, int bi, u64* smem, int slot = -1) : Base(e, k, bi, smem, slot) {}
    CF_HD u64* tws() const { return sm + SM::TWS; }

    CF_HD u64 sh(u64 a, const u64* pairs, int k) const {  // a * pairs[k], result in [0, 4p)
        return shoup_mul_lazy(a, ldc<CG>(pairs + 2 * k), ldc<CG>(pairs + 2 * k + 1), P);
    }
    // Shoup companion of w < p, from the per-prime constants setup keeps in shared memory
    CF_HD u64 companion(u64 w) const { return shoup_companion_fast(w, P, misc()[MI_ONEQ], misc()[MI_R1], misc()[MI_R1Q]); }
    CF_HD void put_pair(u64* pairs, int k, u64 v) const {
        pairs[2 * k] = v;
        pairs[2 * k + 1] = companion(v);
    }
    CF_HD u64 canon(u64 x) const { return red2(red2(x, 2 * P), P); }  // [0, 4p) -> [0, p)

    // ---------------------------------------------------------------------------------------
    // Transform passes.  Forward: Gentleman-Sande (natural in, bit-reversed out); inverse:
    // Cooley-Tukey with inverse roots (bit-reversed in, natural out, unscaled), the same pair of
    // transforms as fast/cuckoo_fast.cu:258-305 and include/cuckoo/ntt.hpp:97-123.  W[k] = w^k
    // for k <= L/2 (W[L/2] = -1), so w_{2h}^{-j} = -W[L/2 - j L/2h] for every j, including 0.
    // Every value stays in [0, 2p).
    // ---------------------------------------------------------------------------------------
    // Butterfly schedule of one register pass.  Unit q runs in order of level (forward: m = r-1
    // down to 0; inverse: 0 up), then twiddle group (ul), then register pair; grp(q) numbers the
    // twiddle groups in that order.
    template <int PASS, bool FWD>
    struct Plan {
        static constexpr int bb = G::pass_b(PASS), r = G::pass_r(PASS);
        static constexpr int BPL = E / 2, NB = BPL * r, NG = (1 << r) - 1;
        // levels done before this pass, in processing order (forward: passes 0 ..; inverse: NP-1 ..)
        static constexpr int s0 = FWD ? PASS * G::R : (PASS == NP - 1 ? 0 : G::R_LAST + (NP - 2 - PASS) * G::R);
        CF_HD static constexpr int lvl(int q) { return s0 + q / BPL; }
        CF_HD static constexpr int m(int q) { return FWD ? r - 1 - q / BPL : q / BPL; }
        CF_HD static constexpr int per(int q) { return E >> (m(q) + 1); }  // butterflies per group
        CF_HD static constexpr int ul(int q) { return (q % BPL) / per(q); }
        CF_HD static constexpr int kk(int q) { return (q % BPL) % per(q); }
        CF_HD static constexpr int grp(int q) { return FWD ? (1 << r) - (1 << (m(q) + 1)) + ul(q) : (1 << m(q)) - 1 + ul(q); }
        CF_HD static constexpr int j0(int q) {
            return ((kk(q) >> (r - 1 - m(q))) << r) + ((kk(q) & ((1 << (r - 1 - m(q))) - 1)) << (m(q) + 1)) + ul(q);
        }
        CF_HD static constexpr int j1(int q) { return j0(q) + (1 << m(q)); }
        // level and group-within-level of twiddle group f
        CF_HD static constexpr int gm(int f) {
            int mm = FWD ? r - 1 : 0;
            while (f >= (1 << mm)) f -= (1 << mm), mm += FWD ? -1 : 1;
            return mm;
        }
        CF_HD static constexpr int gul(int f) {
            int mm = FWD ? r - 1 : 0;
            while (f >= (1 << mm)) f -= (1 << mm), mm += FWD ? -1 : 1;
            return f;
        }
        CF_HD static constexpr bool trivial_grp(int f) { return bb == 0 && gul(f) == 0; }
    };
    // pair address of the twiddle of group F (forward: w_{2h}^j; inverse: W[L/2 - j L/2h], whose
    // negation is w_{2h}^{-j})
    // Pass 0 reads its level's table in global memory (a warp's lanes take consecutive pairs);
    // later passes only need multiples of 2^R, kept in shared memory.
    template <int PASS, bool FWD, int F>
    CF_HD const u64* tw_addr(int off) const {
        typedef Plan<PASS, FWD> PL;
        constexpr int mm = PL::gm(F), ul = PL::gul(F), sh = G::LG - 1 - PL::bb - mm;
        const int u = off + (ul << PL::bb);  // twiddle w^(u 2^sh)
        if constexpr (PASS == 0) return WL(sh) + 2 * (FWD ? u : (L >> (sh + 1)) - u);
        else return tws() + 2 * ((FWD ? u << sh : L / 2 - (u << sh)) >> G::R);
    }
    template <int PASS>
    CF_HD static void ld_tw(const u64* p, u64& a, u64& b) {
        if constexpr (PASS == 0) ldp<CG>(p, a, b);
        else ld_pair_shared(p, a, b);
    }
    template <int PASS, bool FWD>
    CF_HD void pass(int t, u64 (&x)[E]) const {
        typedef Plan<PASS, FWD> PL;
        // pass 0 reads its twiddles from L2 (the others from shared memory): at 1024 threads it
        // prefetches them two groups ahead (72.1 against 70.3 prime-residues/s at n = 16384)
        constexpr int D = (PASS == 0 && T >= 1024) ? 2 : PD;
        const int off = PL::bb ? (t & ((1 << PL::bb) - 1)) : 0;
        const u64 P = this->P, P2 = 2 * P;
        u64 rw[D + 1], rq[D + 1];
        window<D, 0>([&](auto fc) CF_INL {
            constexpr int f = decltype(fc)::value;
            if constexpr (f < PL::NG && !PL::trivial_grp(f)) ld_tw<PASS>(tw_addr<PASS, FWD, f>(off), rw[f], rq[f]);
        }, [&](auto) CF_INL {});
        window<PL::NB, WK>(
            [&](auto qc) CF_INL {
                constexpr int q = decltype(qc)::value, f = PL::grp(q), fn = f + D;
                if constexpr (PL::kk(q) == 0 && fn < PL::NG && !PL::trivial_grp(fn))
                    ld_tw<PASS>(tw_addr<PASS, FWD, fn>(off), rw[fn % (D + 1)], rq[fn % (D + 1)]);
                constexpr int j0 = PL::j0(q), j1 = PL::j1(q);
                constexpr bool trivial = PL::trivial_grp(f);
                pin(x[j0]);
                pin(x[j1]);
                const u64 w = rw[f % (D + 1)], wq = rq[f % (D + 1)];
                if constexpr (FWD) {  // inputs and outputs in [0, 2p)
                    const u64 a = x[j0], c = x[j1];
                    x[j0] = red2(a + c, P2);
                    const u64 dd = a - c + P2;
                    x[j1] = red2(trivial ? dd : shoup_mul_lazy(dd, w, wq, P), P2);
                } else {
                    const u64 a = x[j0];
                    if constexpr (trivial) {
                        const u64 c = x[j1];
                        x[j0] = red2(a + c, P2);
                        x[j1] = red2(a - c + P2, P2);
                    } else {
                        const u64 c = red2(shoup_mul_lazy(x[j1], w, wq, P), P2);  // -w_{2h}^{-j} y
                        x[j0] = red2(a - c + P2, P2);
                        x[j1] = red2(a + c, P2);
                    }
                }
            },
            [&](auto qc) CF_INL {
                constexpr int q = decltype(qc)::value;
                pin(x[PL::j0(q)]);
                pin(x[PL::j1(q)]);
            });
    }
    template <int PASS>
    CF_HD void fwd_pass(int t, u64 (&x)[E]) const { pass<PASS, true>(t, x); }
    template <int PASS>
    CF_HD void inv_pass(int t, u64 (&x)[E]) const { pass<PASS, false>(t, x); }
    // Entries to shared memory by index.  In a cluster, pass 0's outputs (forward) go to the CTA
    // whose block holds them, and with TO_L0 the inverse transform's pass-1 outputs go to the CTA that holds them in pass 0.
    template <int PASS, bool TO_L0 = false>
    CF_HD void to_smem(int t, u64 (&x)[E]) const {
        pin_int(t);  // recompute the addresses rather than keep the loads' 32 addresses live across the pass
        if constexpr (C > 1 && PASS == 0) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(0, t, j);
                ex.st_remote(sm + G::swz(i & (LCN - 1)), i / LCN, x[j]);
            }
        } else if constexpr (C > 1 && TO_L0) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(PASS, t, j);
                ex.st_remote(sm + SM::X0 + (i & (CT - 1)) + (i / T) * CT, (i & (T - 1)) / CT, x[j]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(PASS, t, j);
                sm[G::swz(C > 1 ? i & (LCN - 1) : i)] = x[j];
            }
        }
    }
    template <int PASS>
    CF_HD void from_smem(int t, u64 (&x)[E]) const {
        if constexpr (C > 1 && PASS == 0) {
#pragma unroll
            for (int j = 0; j < E; ++j) x[j] = sm[SM::X0 + lt(t) + j * CT];
        } else {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(PASS, t, j);
                x[j] = sm[G::swz(C > 1 ? i & (LCN - 1) : i)];
            }
        }
    }
    // the barrier before pass PASS reads shared memory: the cluster's at the exchanges
    template <int PASS, bool FWD>
    CF_HD void pass_sync() {
        if constexpr (C > 1 && ((FWD && PASS == 1) || (!FWD && PASS == 0))) ex.cluster_sync();
        else ex.sync();
    }

    template <int PASS>
    CF_HD void fwd_chain() {  // forward passes PASS .. NP-1, pointwise, last inverse pass (PASS >= 1)
        pass_sync<PASS, true>();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            from_smem<PASS>(t, rg.x);
            fwd_pass<PASS>(t, rg.x);
            if (PASS == NP - 1) {
                pointwise(t, rg.x);
                inv_pass<PASS>(t, rg.x);
            }
            to_smem<PASS, PASS == 1 && NP == 2>(t, rg.x);  // the inverse's pass 1 only when it is the last
        });
        if constexpr (PASS + 1 < NP) fwd_chain<PASS + 1>();
    }
    template <int PASS>
    CF_HD void inv_chain() {  // inverse passes PASS .. 0 (entry: data in smem in layout PASS + 1)
        pass_sync<PASS, false>();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            from_smem<PASS>(t, rg.x);
            inv_pass<PASS>(t, rg.x);
            if (PASS > 0) to_smem<PASS, PASS == 1>(t, rg.x);
        });
        if constexpr (PASS > 0) inv_chain<PASS - 1>();
    }
    // spectrum pairs of chunk C (entries 4C .. 4C+3) from tensor memory, then the next chunk
    template <int CH>
    CF_HD void tm_pointwise(int t, u32 ta, u64 (&x)[E], u32 (&b0)[16], u32 (&b1)[16]) const {
        if constexpr (CH < E / 4) {
            u32(&cur)[16] = (CH & 1) ? b1 : b0;
            u32(&nxt)[16] = (CH & 1) ? b0 : b1;
            if constexpr (CH + 1 < E / 4) ex.tmem_ld16(t, ta + 16 * (CH + 1), nxt);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const u64 w = (u64)cur[4 * k] | ((u64)cur[4 * k + 1] << 32), wq = (u64)cur[4 * k + 2] | ((u64)cur[4 * k + 3] << 32);
                x[4 * CH + k] = shoup_mul_lazy(x[4 * CH + k], w, wq, P);
                x[4 * CH + k] = red2(x[4 * CH + k], 2 * P);
            }
            ex.tmem_wait_ld();
            tm_pointwise<CH + 1>(t, ta, x, b0, b1);
        }
    }
    CF_HD void pointwise(int t, u64 (&x)[E]) const {
        if constexpr (TM) {
            const u32 ta = X::tmem_addr((u32)misc()[MI_TMEM], lt(t));
            u32 b0[16], b1[16];
            ex.tmem_ld16(t, ta, b0);
            ex.tmem_wait_ld();
            tm_pointwise<0>(t, ta, x, b0, b1);
            return;
        }
        const u64* h = hat();
        pipe_pairs<E, PD, WK, CG>(
            [&](auto jc) CF_INL { return h + 2 * G::idx(NP - 1, t, decltype(jc)::value); },
            [&](auto jc, u64 w, u64 wq) CF_INL {
                constexpr int j = decltype(jc)::value;
                pin(x[j]);
                x[j] = shoup_mul_lazy(x[j], w, wq, P);
                x[j] = red2(x[j], 2 * P);
            },
            [&](auto jc) CF_INL { pin(x[decltype(jc)::value]); });
    }
    // Cyclic convolution of the registers (layout of pass 0, values < 4p) with the kernel 1/t;
    // the result comes back in the same layout, below 2p.
    CF_HD void convolve() {
        if constexpr (NP == 1) {
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                fwd_pass<0>(t, rg.x);
                pointwise(t, rg.x);
                inv_pass<0>(t, rg.x);
            });
        } else {
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                fwd_pass<0>(t, rg.x);
                to_smem<0>(t, rg.x);
            });
            fwd_chain<1>();
            inv_chain<NP - 2>();
        }
    }
    // forward transform only (registers in layout 0 -> registers in layout NP-1), used for the
    // kernel spectrum
    template <int PASS>
    CF_HD void fwd_only_chain() {
        pass_sync<PASS, true>();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            from_smem<PASS>(t, rg.x);
            fwd_pass<PASS>(t, rg.x);
            if (PASS < NP - 1) to_smem<PASS>(t, rg.x);
        });
        if constexpr (PASS + 1 < NP) fwd_only_chain<PASS + 1>();
    }
    CF_HD void fwd_only() {
        if constexpr (NP == 1) {
            ex.each([&](int t, Regs<G>& rg) CF_INL { fwd_pass<0>(t, rg.x); });
        } else {
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                fwd_pass<0>(t, rg.x);
                to_smem<0>(t, rg.x);
            });
            fwd_only_chain<1>();
        }
    }

    // value of a pair table, canonical
    CF_HD static u64 val(const u64* pairs, int k) { return ldc<CG>(pairs + 2 * k); }

    // The slots' powers h^(t + jT), j = 0 .. E-1, as NCH independent running products: chain c
    // holds h^(t + jT) for j = c (mod NCH) and steps by h^(NCH T), so the products that depend on
    // one another are NCH times fewer than with one chain.
    static constexpr int NCH = E >= 4 ? 4 : E;

    // Stage-2 powers of h = 1/g(v) (base 0: the row products) and h = g(v) (base 1: the stage-2
    // products), Montgomery form, rebuilt at the start of each step in shared memory (the PW_*
    // slots): A[k] = h^k (k < TA = min(T, 32)), B[k] = h^(TA k) (k < TB = T / TA), J[j] = h^(T j)
    // (j < E), the chains' step h^(NCH T) as a plain residue with its Shoup companion (a Shoup product
    // by it keeps a Montgomery-form power in Montgomery form), and h^L.  Slot j of thread t holds
    // index t + jT, whose power is A[t % TA] B[t / TA] J[j].  The six groups (A, B, J for two bases)
    // go to six warps, fewer warps looping over them; a group's lanes raise a common base (h, h^TA
    // or h^T, which every lane squares up itself) to their own small exponent, so the deepest chain
    // is about 20 products, and h comes from the table of g(v) built at setup.  The other warps go
    // straight on with stage 1: the tables are read only after its barriers.  In a cluster, t is the
    // thread's index in its CTA and J[j] = h^(c CT + T j) carries the CTA's offset c CT.
    static constexpr int TA = CT < 32 ? CT : 32, TB = CT / TA;
    static constexpr int LW = CT < 32 ? CT : 32;  // lanes of a warp
    CF_HD static constexpr int log2c(int x) { return x <= 1 ? 0 : 1 + log2c(x / 2); }
    CF_HD void power_tables(int v) {
        u64* pw = sm + SM::PW;
        const u64* gm = Gm();
        ex.each([&](int t, Regs<G>&) CF_INL {
            const int lane = t & 31;
            for (int gi = lt(t) >> 5; gi < 6; gi += NW) {
                const int base = gi & 1, kind = gi >> 1;
                const int size = kind == 0 ? TA : kind == 1 ? TB : E + 2;
                if (lane >= size) continue;
                const Mod m = md();
                u64* tab = pw + base * SM::PW_STRIDE;
                u64 b = ldc<CG>(gm + 2 * v + 1 - base);  // 1/g(v) or g(v)
                u64 off = m.r1;                          // h^(c CT): the CTA's offset (clusters)
                if constexpr (C > 1)
                    if (kind == 2 && rank() > 0) off = mont_pow(b, (u64)rank() * CT, m);
                const int sq = kind == 0 ? 0 : kind == 1 ? log2c(TA) : log2c(T);
                for (int i = 0; i < sq; ++i) b = mont_mul(b, b, m);
                for (int k = lane; k < size; k += LW) {
                    if (kind == 0) tab[PW_A + k] = mont_pow(b, (u64)k, m);
                    else if (kind == 1) tab[PW_B + k] = mont_pow(b, (u64)k, m);
                    else if (k < E) tab[PW_J + k] = C > 1 ? mont_mul(mont_pow(b, (u64)k, m), off, m) : mont_pow(b, (u64)k, m);
                    else if (k == E) {
                        const u64 y = from_mont(mont_pow(b, (u64)NCH, m), m);
                        tab[PW_STEP] = y;
                        tab[PW_STEPQ] = shoup_companion_fast(y, P, misc()[MI_ONEQ], m.r1, misc()[MI_R1Q]);
                    } else tab[PW_L] = mont_pow(b, (u64)E, m);
                }
            }
        });
    }
    // chain c of thread t holds h^(t + jT) for j = c (mod NCH) in Montgomery form and steps by a
    // Shoup product with (step, stepq) = h^(NCH T) and its companion: canonical: mont_mul's full
    // product is exact only below 2^62
    CF_HD u64 chain_step(u64 f, u64 step, u64 stepq) const {
        const u64 y = shoup_mul_lazy(f, step, stepq, P);
        return canon(y);
    }
    // Chains started at slot j0 (the first slot a warp needs): chain c starts at the first slot
    // j >= j0 with j = c (mod NCH), from A[t % TA] B[t / TA] J[j].
    CF_HD void power_chains(int base, int t, const Mod& m, u64 (&f)[NCH], u64& step, u64& stepq, int j0 = 0) const {
        const u64* pw = sm + SM::PW + base * SM::PW_STRIDE;
        const int tl = lt(t);
        const u64 ab = TB > 1 ? mont_mul(pw[PW_A + tl % TA], pw[PW_B + tl / TA], m) : pw[PW_A + tl];
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const int jc = j0 + ((c - j0) & (NCH - 1));
            // J[0] = 1 on a CTA alone; in a cluster it carries the CTA's offset h^(c CT)
            f[c] = (jc == 0 && C == 1) ? ab : (jc < E ? mont_mul(ab, pw[PW_J + jc], m) : 0);
        }
        step = pw[PW_STEP], stepq = pw[PW_STEPQ];
    }
    // g(v) and 1/g(v) in Montgomery form, from the table built at setup (0 for v < d0, subset model)
    CF_HD u64 g_mont(int v) const { return ldc<CG>(Gm() + 2 * v); }
    CF_HD u64 ginv_mont(int v) const { return ldc<CG>(Gm() + 2 * v + 1); }

    // ---------------------------------------------------------------------------------------
    // Setup: factorials, inverses, D, twiddles and the kernel spectrum of 1/t (the per-batch host
    // work of fast/cuckoo_fast.cu:797-839, done on the device).
    // ---------------------------------------------------------------------------------------
    CF_HD void setup() {
        u64* red = sm + SM::RED;  // red[t]: prefix before chunk t; red[CT + t]: chunk product / suffix
        u64* mi = misc();
        const int F = kp.F, n = kp.n, J = kp.J;
        ex.single([&]() CF_INL {
            const Mod m = make_mod(P);
            mi[MI_P] = m.p, mi[MI_PINV] = m.pinv, mi[MI_R1] = m.r1, mi[MI_R2] = m.r2;
            mi[MI_ONEQ] = shoup_companion(1, P);
            mi[MI_R1Q] = shoup_companion(m.r1, P);
        });
        ex.sync();
        // The prime's tables in global memory: one CTA builds them (the cluster's first, which its
        // other CTAs wait for at the cluster barrier below).
        if (rank() == 0) {
            const int CH = (F + 1 + CT - 1) / CT;  // factorial entries k = 0..F, chunk of CH per thread
            // product of the integers in each chunk (Montgomery form)
            ex.each([&](int t, Regs<G>&) CF_INL {
                const Mod m = md();
                const int k0 = t * CH > 1 ? t * CH : 1, k1 = (t + 1) * CH < F + 1 ? (t + 1) * CH : F + 1;
                u64 pr = m.r1;
                u64 km = to_mont((u64)k0, m);
                for (int k = k0; k < k1; ++k) {
                    pr = mont_mul(pr, km, m);
                    km = madd(km, m.r1, P);
                }
                red[CT + t] = pr;
            });
            ex.sync();
            ex.single([&]() CF_INL {  // exclusive prefix products, F!, 1/F!, exclusive suffix products / F!
                const Mod m = md();
                u64 run = m.r1;
                for (int t = 0; t < CT; ++t) {
                    red[t] = run;
                    run = mont_mul(run, red[CT + t], m);
                }
                u64 suf = mont_pow(run, P - 2, m);  // 1/F!
                for (int t = CT - 1; t >= 0; --t) {
                    const u64 c = red[CT + t];
                    red[CT + t] = suf;  // 1/F! times the product of the chunks after t = 1/(last k of chunk t)!
                    suf = mont_mul(suf, c, m);
                }
            });
            ex.sync();
            ex.each([&](int t, Regs<G>&) CF_INL {
                const Mod m = md();
                const int k0 = t * CH, k1 = (t + 1) * CH < F + 1 ? (t + 1) * CH : F + 1;
                u64 run = red[t];  // (k0 - 1)! (Montgomery), 1 for the first chunk
                u64 km = to_mont((u64)(k0 > 0 ? k0 : 1), m);
                for (int k = k0; k < k1; ++k) {  // k! = (k-1)! k
                    if (k > 0) {
                        run = mont_mul(run, km, m);
                        km = madd(km, m.r1, P);
                    }
                    put_pair(fact(), k, from_mont(run, m));
                }
                run = red[CT + t];  // 1/(k1 - 1)!
                for (int k = k1 - 1; k >= k0; --k) {  // 1/(k-1)! = k / k!
                    put_pair(ifact(), k, from_mont(run, m));
                    if (k > 0) run = mont_mul(run, to_mont((u64)k, m), m);
                }
            });
            ex.sync();
            // inv[k] = (k-1)!/k!, D[k] = 1/k!^2, Kq[k] = companion of k
            ex.each([&](int t, Regs<G>&) CF_INL {
                for (int k = t; k <= F; k += CT) put_pair(inv(), k, k ? canon(sh(val(ifact(), k), fact(), k - 1)) : 0);
                for (int k = t; k <= n; k += CT) put_pair(D(), k, canon(sh(val(ifact(), k), ifact(), k)));
                // g(k) and 1/g(k), Montgomery form: C(k, d) and its inverse, or k^d and (1/k)^d
                const Mod m = md();
                for (int k = t; k <= n; k += CT) {
                    u64 g = 0, gi = 0;
                    if (kp.model == MODEL_REPLACEMENT) {
                        if (k > 0) {
                            g = mont_pow(to_mont((u64)k, m), (u64)kp.d, m);
                            gi = mont_pow(to_mont(inv()[2 * k], m), (u64)kp.d, m);  // this thread wrote inv[k]
                        }
                    } else if (k >= kp.d) {
                        g = to_mont(canon(sh(sh(val(fact(), k), ifact(), kp.d), ifact(), k - kp.d)), m);
                        gi = to_mont(canon(sh(sh(val(ifact(), k), fact(), kp.d), fact(), k - kp.d)), m);
                    }
                    Gm()[2 * k] = g;
                    Gm()[2 * k + 1] = gi;
                }
            });
        }
        // query partial sums zeroed (each CTA's own)
        ex.each([&](int t, Regs<G>&) CF_INL {
            const size_t nps = (size_t)J * (n + 1);
            for (size_t k = lt(t); k < nps; k += CT) ps()[k] = 0;
        });
        // a root of unity of order L: x^((p-1)/L) whose (L/2)-th power is -1 (fast/cuckoo_fast.cu:815-820)
        ex.single([&]() CF_INL {
            const Mod m = md();
            const u64 minus1 = P - m.r1;
            u64 w = 0;
            int found = 0;
            for (u64 x = 2; x < 1000; ++x) {
                w = mont_pow(to_mont(x, m), (P - 1) / L, m);
                if (mont_pow(w, L / 2, m) == minus1) {
                    found = 1;
                    break;
                }
            }
            if (!found && rank() == 0) ex.set_error(kp.err, KERR_NO_ROOT);
            mi[MI_ROOT] = w;
            mi[MI_LINV] = from_mont(mont_pow(to_mont((u64)L, m), P - 2, m), m);  // 1/L, canonical
        });
        ex.sync();
        // w^k into every table that holds it: the pass-0 tables by level (global, the first CTA)
        // and the multiples of 2^R of the later passes (every CTA's shared memory)
        ex.each([&](int t, Regs<G>&) CF_INL {
            const Mod m = md();
            const u64 w = mi[MI_ROOT];
            const int tl = lt(t);
            u64 cur = mont_pow(w, (u64)tl, m);
            const u64 step = mont_pow(w, (u64)CT, m);
            for (int k = tl; k <= L / 2; k += CT) {
                const bool tw = (k & ((1 << G::R) - 1)) == 0;
                if (rank() == 0 || tw) {
                    const u64 c = from_mont(cur, m), cq = companion(c);
                    if (rank() == 0)
                        for (int l = 0; l < G::R && (k & ((1 << l) - 1)) == 0; ++l) {
                            u64* d = WL(l) + 2 * (k >> l);
                            d[0] = c, d[1] = cq;
                        }
                    if (tw) {
                        u64* d = tws() + 2 * (k >> G::R);
                        d[0] = c, d[1] = cq;
                    }
                }
                cur = mont_mul(cur, step, m);
            }
        });
        csync();  // the first CTA's tables are read below and by every later step
        // kernel spectrum: hat = DIF(ker) / L with ker[t] = 1/t for 1 <= t <= n-1 (fast/cuckoo_fast.cu:829,838-839)
        ex.each([&](int t, Regs<G>& rg) CF_INL {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(0, t, j);
                rg.x[j] = (i >= 1 && i < n) ? val(inv(), i) : 0;
            }
        });
        fwd_only();
        if (kp.keep) {  // the pair tables, for queries served later from this prime's resident V
            const KeepLayout kl = make_keep_layout(n, F);
            u64* kb = kp.keep + (size_t)b * kp.keep_words;
            ex.each([&](int t, Regs<G>&) CF_INL {
                for (size_t k = t; k < 2 * ((size_t)F + 1); k += T) {
                    kb[kl.fact + k] = fact()[k];
                    kb[kl.ifact + k] = ifact()[k];
                    kb[kl.inv + k] = inv()[k];
                }
            });
        }
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            const u64 linv = mi[MI_LINV];
            const u64 linvq = companion(linv);
            if constexpr (TM) {
                const u32 ta = X::tmem_addr((u32)mi[MI_TMEM], lt(t));
#pragma unroll
                for (int c = 0; c < E / 4; ++c) {
                    u32 v[16];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const u64 h = canon(shoup_mul_lazy(rg.x[4 * c + k], linv, linvq, P)), hq = companion(h);
                        v[4 * k] = lo32(h), v[4 * k + 1] = hi32(h), v[4 * k + 2] = lo32(hq), v[4 * k + 3] = hi32(hq);
                    }
                    ex.tmem_st16(t, ta + 16 * c, v);
                }
                ex.tmem_wait_st();
            } else {
#pragma unroll
                for (int j = 0; j < E; ++j) put_pair(hat(), G::idx(NP - 1, t, j), canon(shoup_mul_lazy(rg.x[j], linv, linvq, P)));
            }
        });
        csync();  // no CTA's transform exchange may start while another still reads its spectrum pass
    }

    // ---------------------------------------------------------------------------------------
    // Query partial sums for row q: sum_{w<q} Vs[q][w] / (M_j - w) for every query with n_j >= q
    // (the U[w] / (M - w) sums of fast/cuckoo_fast.cu:306-323, 595-622).  The row is in the
    // registers (layout 0, entries outside the row zero).  Only the slots below q are visited: the
    // warp leaves the unrolled slot loop at its first slot wholly at or above q (slot indices grow
    // with j, so the exit is warp-uniform), which makes a query cost about n_j^2 / 2 products
    // instead of n_j L.  Each warp leaves its sum at QS[j][warp] in shared memory; fold_last
    // combines them after the next barrier.
    // ---------------------------------------------------------------------------------------
    CF_HD void query_row(int q) {
        this->query_batches(q, [&](int ja, int jb, u64* qs0) CF_INL {
          for (int jq = ja; jq < jb; ++jq) {
            const int nj = kp.qn[jq], Mj = kp.qM[jq];
            u64* qs = qs0 + (size_t)(jq - ja) * NW;
            if (nj < q) continue;
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                const u64* iv = inv() + 2 * (size_t)Mj;  // the pair of 1/(M_j - w) sits at iv - 2w
                const int tw = t & ~31;                  // the warp's first thread
                u64 acc = 0;
                if constexpr (C == 1) {  // the next slot's inverse loaded one slot ahead
                    u64 c0 = 0, q0 = 0;
                    if (G::idx(0, t, 0) < q) ldp<CG>(iv - 2 * G::idx(0, t, 0), c0, q0);
#pragma unroll
                    for (int j = 0; j < E; ++j) {
                        const bool more = j + 1 < E && G::idx(0, tw, j + 1) < q;
                        u64 c1 = 0, q1 = 0;  // slots at or above q multiply by zero
                        if (more && G::idx(0, t, j + 1) < q) ldp<CG>(iv - 2 * G::idx(0, t, j + 1), c1, q1);
                        acc = madd(acc, canon(shoup_mul_lazy(rg.x[j], c0, q0, P)), P);
                        if (!more) break;
                        c0 = c1, q0 = q1;
                    }
                } else {
                    // A cluster's CTAs have half the warps of the 2^14 kernel to hide the inverses'
                    // L2 latency: they load QD slots ahead (a ring of QD + 1 pairs).  Measured at
                    // n = 65536 with 126 queries: 8.29 against 8.86 s per launch; with one query the
                    // deeper ring cost the 2^14 kernel 1.5 %, so that kernel keeps one slot.
                    constexpr int QD = 4;
                    u64 rc[QD + 1], rq[QD + 1];
#pragma unroll
                    for (int j = 0; j < QD + 1; ++j) rc[j] = rq[j] = 0;
#pragma unroll
                    for (int j = 0; j < QD && j < E; ++j)
                        if (G::idx(0, t, j) < q) ldp<CG>(iv - 2 * G::idx(0, t, j), rc[j], rq[j]);
#pragma unroll
                    for (int j = 0; j < E; ++j) {
                        if (G::idx(0, tw, j) >= q) break;  // warp-uniform: this slot and the later ones lie past the row
                        const int jn = j + QD;
                        if (jn < E && G::idx(0, t, jn) < q) ldp<CG>(iv - 2 * G::idx(0, t, jn), rc[jn % (QD + 1)], rq[jn % (QD + 1)]);
                        const u64 c0 = G::idx(0, t, j) < q ? rc[j % (QD + 1)] : 0;  // slots at or above q multiply by zero
                        const u64 q0 = G::idx(0, t, j) < q ? rq[j % (QD + 1)] : 0;
                        acc = madd(acc, canon(shoup_mul_lazy(rg.x[j], c0, q0, P)), P);
                    }
                }
                const u64 part = canon(shoup_mul_lazy(acc, 1, misc()[MI_ONEQ], P));
                ex.warp_sum_store(lt(t), part, P, qs, 1);
            });
          }
        });
    }
    // One step of the suffix recurrence (fast/cuckoo_fast.cu:841-855).
    CF_HD void step(int v) {
        const int n = kp.n, d0 = kp.d0;
        if (v >= d0) power_tables(v);  // read after the barriers of stage 1 / the stage-2 barrier
        if (v > d0) {  // stage 1: column v of S from row v of V
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                load_row(t, rg.x, V(), VS(), v, d0, v);  // columns w < d0 of V are zero (g(w) = 0), never written
            });
            query_row(v);
            convolve();
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                const u64 iv = val(inv(), v), ivq = ldc<CG>(inv() + 2 * v + 1);
                u64* col = SS() + (size_t)(v - tile_v0(v)) * (n + 1);  // S[.][v], by row
                const u64* Dt = D();
                pipe_pairs_live<E, PD, WK, CG>(
                    [&](auto jc) CF_INL {  // rows v .. n-1 of column v: slots where the warp holds one
                        int lo, hi;
                        warp_slot_range(t, decltype(jc)::value, lo, hi);
                        return hi >= v && lo < n;
                    },
                    [&](auto jc) CF_INL {
                        const int i = G::idx(0, t, decltype(jc)::value);
                        return Dt + 2 * (i >= v && i < n ? i - v : 0);
                    },
                    [&](auto jc, u64 c, u64 cq) CF_INL {
                        constexpr int j = decltype(jc)::value;
                        const int i = G::idx(0, t, j);
                        pin(rg.x[j]);
                        rg.x[j] = shoup_mul_lazy(shoup_mul_lazy(rg.x[j], c, cq, P), iv, ivq, P);
                        rg.x[j] = canon(rg.x[j]);
                        if (i >= v && i < n) st_stream(col + i, rg.x[j]);
                    },
                    [&](auto jc) CF_INL { pin(rg.x[decltype(jc)::value]); });
            });
            fold_last(v);  // after the transform's barriers: every warp's partial of row v is in
        }
        if (v >= d0) {  // stage 2: column v of V from row v of S
            csync();  // column v of S is read below
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                const Mod m = md();
                u64 f[NCH], step, stepq;  // g^-(t + jT)
                power_chains(0, t, m, f, step, stepq);
                // columns q <= d0 of S are zero (stage 1 skipped: row q of V is zero), never written
                load_row(t, rg.x, S(), SS(), v, d0 + 1, v + 1);
                window<E, WK>(
                    [&](auto jc) CF_INL {
                        constexpr int j = decltype(jc)::value;
                        int lo, hi;
                        warp_slot_range(t, j, lo, hi);
                        if (lo > v) return;  // entries q <= v only: this slot and the later ones stay zero
                        pin(rg.x[j]);
                        rg.x[j] = mont_mul(rg.x[j], f[j % NCH], m);  // x, f < 4p: exact, canonical
                        f[j % NCH] = chain_step(f[j % NCH], step, stepq);
                    },
                    [&](auto jc) CF_INL { pin(rg.x[decltype(jc)::value]); });
            });
            convolve();
            ex.each([&](int t, Regs<G>& rg) CF_INL {
                const Mod m = md();
                // Entries p = v+1 .. n: the warp's first slot holding one is j0, and its chains start
                // there.  When L = n, e[n] sits at index 0 (thread 0, slot 0): a slot of its own, done
                // below by thread 0 alone when warp 0 skips slot 0, so no warp does more than the rest.
                int j0 = 0;
#pragma unroll
                for (int j = 0; j < E; ++j) {
                    int lo, hi;
                    warp_slot_range(t, j, lo, hi);
                    j0 += hi <= v;
                }
                u64 f[NCH], step, stepq;  // g^(t + jT)
                power_chains(1, t, m, f, step, stepq, j0);
                const u64 dv = val(D(), v);
                u64* col = VS() + (size_t)(v - tile_v0(v)) * (n + 1);  // V[.][v], by row
                const u64* Dt = D();
                const u64 fwrap = sm[SM::PW + SM::PW_STRIDE + PW_L];  // g^L, for e[n] at index 0 when L = n
                // the multipliers p of the slots as a running Montgomery form (p = t + j T)
                u64 pm = to_mont((u64)(t + j0 * T), m);
                const u64 pmT = to_mont((u64)T, m), pmL = (t == 0 && n == L) ? to_mont((u64)L, m) : 0;
                // V[p][v] = g^p D[p-v-1] (D[v] - p e[p]) for a conv output x = e[p], (c, cq) = D[p-v-1],
                // gp = g^p and pmv = p in Montgomery form
                auto entry = [&](u64 x, int p, u64 c, u64 cq, u64 gp, u64 pmv) CF_INL {
                    const u64 pe = mont_mul(x, pmv, m);  // p e[p]: x < 2P, pmv < P keep the product exact below 2^126
                    const u64 y = canon(shoup_mul_lazy(dv + P - pe, c, cq, P));
                    return mont_mul(y, gp, m);
                };
                const bool wrap0 = n == L && t == 0;  // this thread holds e[n] at index 0
                if (wrap0 && j0 > 0 && L > v) {
                    u64 c, cq;
                    ldp<CG>(Dt + 2 * (L - v - 1), c, cq);
                    st_stream(col + L, entry(rg.x[0], L, c, cq, fwrap, pmL));
                }
                pipe_pairs_live<E, PD, WK, CG>(
                    [&](auto jc) CF_INL {
                        int lo, hi;
                        warp_slot_range(t, decltype(jc)::value, lo, hi);
                        return decltype(jc)::value >= j0 && lo <= n;
                    },
                    [&](auto jc) CF_INL {
                        const int i = G::idx(0, t, decltype(jc)::value), p = i == 0 ? L : i;
                        return Dt + 2 * (p > v && p <= n ? p - v - 1 : 0);
                    },
                    [&](auto jc, u64 c, u64 cq) CF_INL {
                        constexpr int j = decltype(jc)::value;
                        const int i = G::idx(0, t, j);
                        const bool wrap = (i == 0);  // e[n] sits at index 0 when L = n
                        const int p = wrap ? L : i;
                        pin(rg.x[j]);
                        if (p > v && p <= n) {
                            rg.x[j] = entry(rg.x[j], p, c, cq, wrap ? fwrap : f[j % NCH], wrap ? pmL : pm);
                            st_stream(col + p, rg.x[j]);
                        }
                        f[j % NCH] = chain_step(f[j % NCH], step, stepq);
                        pm = madd(pm, pmT, P);
                    },
                    [&](auto jc) CF_INL { pin(rg.x[decltype(jc)::value]); });
            });
        }
        this->end_step(v, [&](int v0, int v1) CF_INL { this->keep_tile(v0, v1, [](u64 x) CF_INL { return x; }); });
    }

    // Horner finish (fast/cuckoo_fast.cu:877-890):
    //   N_bad = M! n! sum_k inv[k] ifact[n-k] ifact[M-k] Q^{n-k} ps[k],  ps[k] = sum of the warp partials.
    CF_HD void finish() {
        const int n = kp.n, d0 = kp.d0;
        u64* red = sm + SM::RED;
        if (n > d0) {  // the last row n for queries with n_j = n
            ex.each([&](int t, Regs<G>& rg) CF_INL { load_row(t, rg.x, V(), VS(), n, d0, n); });
            query_row(n);
            ex.sync();
            fold_last(n);
        }
        csync();  // every CTA's row sums are in
        if (rank() == 0) {  // in a cluster, the first CTA adds up the CTAs' row sums
            for (int jq = 0; jq < kp.J; ++jq) {
                const int nj = kp.qn[jq], Mj = kp.qM[jq];
                ex.each([&](int t, Regs<G>&) CF_INL {
                    const Mod m = md();
                    u64 Qm;
                    if (kp.model == MODEL_REPLACEMENT) Qm = mont_pow(to_mont((u64)Mj, m), (u64)kp.d, m);
                    else Qm = to_mont(canon(sh(sh(val(fact(), Mj), ifact(), kp.d), ifact(), Mj - kp.d)), m);
                    const size_t pj = (size_t)jq * (n + 1);
                    u64 acc = 0;
                    for (int k = t + 1; k <= nj; k += CT) {
                        u64 y = ldc<CG>(ps_of(0) + pj + k);
                        for (int c = 1; c < C; ++c) y = madd(y, ldc<CG>(ps_of(c) + pj + k), P);
                        y = sh(y, inv(), k);
                        y = sh(y, ifact(), nj - k);
                        y = sh(y, ifact(), Mj - k);
                        y = canon(y);  // a factor below 2^62 keeps mont_mul exact
                        y = mont_mul(y, mont_pow(Qm, (u64)(nj - k), m), m);
                        acc = madd(acc, y, P);
                    }
                    red[t] = acc;
                });
                const u64 s = sum_red();
                ex.single([&]() CF_INL {
                    kp.out[kp.qout ? (size_t)kp.qout[jq] : (size_t)b * kp.J + jq] = canon(sh(canon(sh(s, fact(), nj)), fact(), Mj));
                });
            }
        }
    }

    // Tensor memory for the kernel spectrum is taken once per CTA, around all the primes it runs.
    CF_HD void acquire() {
        if constexpr (TM) ex.tmem_alloc((u32*)(misc() + MI_TMEM));
    }
    CF_HD void release() {
        if constexpr (TM) ex.tmem_free((u32)misc()[MI_TMEM]);
    }
    CF_HD void run_prime() {
        setup();
        for (int v = 1; v < kp.n; ++v) step(v);
        finish();
    }
    CF_HD void run() {
        acquire();
        run_prime();
        release();
    }
};

}  // namespace cfb
