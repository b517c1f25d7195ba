// The per-prime kernel for primes below 2^50 (the fixed list of fast/cuckoo_fast.cu with FP_RB = 52,
// and the library CLI's 32-bit primes), in double precision (fparith.cuh).
//
// Transforms.  Forward: butterflies (a, b) -> (a + w b, a - w b) from the natural order to the
// bit-reversed one, in the ring of polynomials split level by level: block k of a level is taken modulo
// x^2h - w^2 and splits into x^h - w and x^h + w with w = tau(k) = w_L^(L sum_i k_i 2^(-i-2)) over the
// bits k_i of k, the same table for every level.  The twiddles depend on the block alone, so the
// first pass reads constants that all threads share, the middle ones constants that most lanes share,
// and only the last pass has twiddles of its own per thread.  Inverse: the same butterflies from
// the bit-reversed order back, with the twiddle w_2h^-j of the place j in the block: shared constants
// in its first pass, a set per thread in its last.  The spectrum is the same as that of
// fast/cuckoo_fast.cu:258-305, so the pair computes the same convolution.
//
// Bounds.  A level adds a product below (1/2 + a/8) p to an entry below a p, so the entries grow slowly
// and few need reducing: where the sum would pass 4p (a factor's limit, see fparith.cuh), the level
// reduces its first inputs (three operations a butterfly, on about one level in four).  Bounds
// tracks this at compile time, and host builds with CF_CHECK_BOUNDS check every butterfly.
//
// What a step spends: 4 (lg L - 1/2) L/2 butterflies of 8 operations, about 3.3e6 of the 4.3e6
// double-precision operations of a step at L = 2^14.
#pragma once
#include "suffix_engine.cuh"

namespace cfb {

// Compile-time loop: f(IC<0>) .. f(IC<N - 1>).
template <int N, int J = 0, class F>
CF_HD void static_for(F&& f) {
    if constexpr (J < N) {
        f(IC<J>{});
        static_for<N, J + 1>(f);
    }
}

// Bounds of the transforms' entries, in multiples of p, by level in processing order.
template <class G>
struct Bounds {
    static constexpr double IN = 0.70;   // inputs (stored entries and products lie below 0.65p)
    static constexpr double LIM = 4.0;   // a product's factor, with the other below p/2
    static constexpr double RED = 0.51;  // after fp_red
    CF_HD static constexpr double prod(double a) { return 0.501 + a / 8; }  // a product of a factor below a p
    // does a level with inputs below a p reduce its first inputs?
    CF_HD static constexpr bool reduces(double a) { return a + prod(a) > LIM; }
    CF_HD static constexpr double next(double a) { return (reduces(a) ? RED : a) + prod(a); }
    // inputs of level s of the forward transform (level 0's twiddle is 1: a plain sum)
    CF_HD static constexpr double fwd(int s) {
        double a = IN;
        for (int k = 0; k < s; ++k) a = k == 0 ? 2 * a : next(a);
        return a;
    }
    CF_HD static constexpr double inv(int s) {  // of the inverse transform (level 0 likewise)
        double a = prod(fwd(G::LG));
        for (int k = 0; k < s; ++k) a = k == 0 ? 2 * a : next(a);
        return a;
    }
    static_assert(fwd(G::LG) <= LIM && inv(G::LG) <= LIM, "the transforms' outputs are factors of products");
};

template <class G, class X>
struct PrimeRun<G, X, false> : PrimeBase<G, X, 0> {
    typedef PrimeBase<G, X, 0> Base;
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
    using Base::WL;
    using Base::hat;
    using Base::ps;
    using Base::ps_of;
    using Base::misc;
    using Base::md;
    using Base::sum_red;
    typedef typename Base::Row Row;
    using Base::fold_last;
    typedef Bounds<G> BD;
    static constexpr int R = G::R, LG = G::LG, RL = G::R_LAST;

    // Tensor memory holds each thread's spectrum entries (E) and forward twiddles of the last pass
    // (FTR rows), in 4E of its lane's 32-bit columns: L / 32 columns a CTA.  Where 2^11 entries or
    // fewer leave more CTAs on an SM than its 512 columns serve, both come from global memory.
    static constexpr int FTR = E - (E >> RL);
    static constexpr bool TM = CT % 128 == 0 && 4 * E * (CT / 128) <= 512 && L >= 4096 && E >= 8;
    // Rows of per-thread constants in global memory that are loaded ahead of their use.
    static constexpr int PD = CT >= 1024 ? 2 : 4;


    int fold_ = 0, pow_ = 0;  // work the next convolution carries along (chain_work)

    CF_HD PrimeRun(X& e, const KParams& k, int bi, u64* smem, int slot = -1) : Base(e, k, bi, smem, slot) {}

    // Tables of doubles (centred residues) in the prime's workspace.  The areas are laid out for the
    // integer kernel's pairs, so each holds at least these.
    CF_HD double* invd() const { return (double*)(base + kp.lay.inv); }  // 1/k, k = 0 .. F
    CF_HD double* Dd() const { return (double*)(base + kp.lay.D); }      // 1/k!^2, k = 0 .. n
    CF_HD double* Gd() const { return (double*)(base + kp.lay.Gm); }     // (g(v), 1/g(v)), v = 0 .. n
    CF_HD double* hatd() const { return (double*)(base + kp.lay.hat); }  // [E][T] spectrum; in setup w^k, k < L
    CF_HD double* IW() const { return (double*)WL(0); }                  // [E - 1][T] inverse twiddles of pass 0
    CF_HD double* FT() const { return IW() + (size_t)(E - 1) * T; }      // [FTR][T] forward twiddles of the last pass
    CF_HD const double* fts() const { return (const double*)(sm + SM::TWS); }
    CF_HD const double* its() const { return fts() + SM::FTN; }
    CF_HD FpMod fm() const {
        FpMod m;
        m.p = fp_bits(misc()[MI_PD]), m.pinv = fp_bits(misc()[MI_PINVD]);
        return m;
    }
    CF_HD static double ldd(const double* p) { return fp_bits(ldc<CG>((const u64*)p)); }
    // a table entry, with the tables' L2 policy and in program order
    CF_HD static double ldt(const double* p) {
#if defined(__CUDA_ARCH__)
        double v;
        if constexpr (CG) asm volatile("ld.global.cg.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(policy_keep()));
        else asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(policy_keep()));
        return v;
#else
        return *p;
#endif
    }
    CF_HD double ud(u64 v) const { return (double)(long long)v; }  // a canonical residue

    CF_HD void check(double x, double mult) const {
#if defined(CF_CHECK_BOUNDS) && !defined(__CUDA_ARCH__)
        if (!(x < mult * (double)P && -x < mult * (double)P) || x != std::nearbyint(x))
            throw std::runtime_error("transform value above its bound");
#else
        (void)x, (void)mult;
#endif
    }

    // ---------------------------------------------------------------------------------------
    // Transform passes
    // ---------------------------------------------------------------------------------------
    // One butterfly of the level with inputs below A p.  KIND 0: the twiddle is 1 and the sums stay
    // plain; 1: the twiddle is 1 and the second input is reduced; 2: a product.
    template <int KIND, bool RED>
    CF_HD void butterfly(double& xa, double& xb, double w, const FpMod& m, double A) const {
        check(xa, A), check(xb, A);
        const double c = KIND == 0 ? xb : KIND == 1 ? fp_red(xb, m) : fp_mulmod(xb, w, m);
        const double a = RED && KIND != 0 ? fp_red(xa, m) : xa;
        xa = fp_add(a, c), xb = fp_add(a, -c);
    }
    // twiddle groups of a pass, numbered in processing order: forward from the widest level down
    template <int PASS>
    struct FwdPlan {
        static constexpr int bb = G::pass_b(PASS), r = G::pass_r(PASS), NG = E - (E >> r);
        CF_HD static constexpr int m(int f) {  // level (slot bit) of group f
            int mm = r - 1;
            while (f >= (1 << (R - 1 - mm))) f -= 1 << (R - 1 - mm), --mm;
            return mm;
        }
        CF_HD static constexpr int u(int f) {  // group within the level: the slots j >> (m + 1) = u
            int mm = r - 1;
            while (f >= (1 << (R - 1 - mm))) f -= 1 << (R - 1 - mm), --mm;
            return f;
        }
        CF_HD static constexpr int s(int f) { return PASS * R + r - 1 - m(f); }  // level in processing order
    };
    // shared-memory index of tau(k) for level s; in a cluster, past pass 0, k counts from the CTA's
    // first block of the level
    CF_HD static constexpr int fts_at(int s, int k) {
        if (C == 1) return k;
        return s < R ? (1 << s) - 1 + k : E - 1 + ((1 << s) - E) / C + k;
    }
    template <int PASS>
    CF_HD void fwd_pass(int t, double (&x)[E]) const {
        typedef FwdPlan<PASS> PL;
        const FpMod md = fm();
        auto group = [&](auto fc, double w) CF_INL {
            constexpr int f = decltype(fc)::value, m = PL::m(f), u = PL::u(f), s = PL::s(f);
            constexpr int kind = PASS > 0 || u > 0 ? 2 : s == 0 ? 0 : 1;
            static_for<(1 << m)>([&](auto kc) CF_INL {
                constexpr int j = (u << (m + 1)) + decltype(kc)::value;
                this->template butterfly<kind, BD::reduces(BD::fwd(s))>(x[j], x[j + (1 << m)], w, md, BD::fwd(s));
            });
        };
        if constexpr (PASS < NP - 1) {
            const double* tw = fts();
            const int tb = lt(t) >> PL::bb;
            static_for<PL::NG>([&](auto fc) CF_INL {
                constexpr int f = decltype(fc)::value, m = PL::m(f), u = PL::u(f), s = PL::s(f);
                if constexpr (PASS == 0) group(fc, u ? tw[fts_at(s, u)] : 1.0);
                else group(fc, tw[fts_at(s, 0) + (tb << (R - 1 - m)) + u]);
            });
        } else if constexpr (TM) {
            const u32 ta = X::tmem_addr((u32)misc()[MI_TMEM], lt(t)) + 2 * E;
            u32 v[16];
            static_for<PL::NG>([&](auto fc) CF_INL {
                constexpr int f = decltype(fc)::value, k = f % 8;
                if constexpr (k == 0) tm_load(t, ta + 2 * f, v);
                group(fc, fp_bits((u64)v[2 * k] | ((u64)v[2 * k + 1] << 32)));
            });
        } else {
            const double* g = FT() + t;
            rows_ahead<PL::NG>(g, group);
        }
    }
    // body(IC<f>, row f's constant of this thread) for f < N; rows are T words apart
    template <int N, class F>
    CF_HD void rows_ahead(const double* g, F&& body) const {
        double w[PD + 1];
        static_for<(PD < N ? PD : N)>([&](auto fc) CF_INL {
            constexpr int f = decltype(fc)::value;
            w[f] = ldt(g + (size_t)f * T);
        });
        static_for<N>([&](auto fc) CF_INL {
            constexpr int f = decltype(fc)::value;
            if constexpr (f + PD < N) w[(f + PD) % (PD + 1)] = ldt(g + (size_t)(f + PD) * T);
            body(fc, w[f % (PD + 1)]);
        });
    }
    // eight doubles of the thread's tensor memory, complete on return
    CF_HD void tm_load(int t, u32 ta, u32 (&v)[16]) const {
        ex.tmem_ld16(t, ta, v);
        ex.tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 16; ++k) pin_word(v[k]);  // no use of v may move above the wait
    }
    template <int PASS>
    CF_HD void inv_pass(int t, double (&x)[E]) const {
        constexpr int bb = G::pass_b(PASS), r = G::pass_r(PASS);
        const FpMod md = fm();
        auto group = [&](auto fc, double w) CF_INL {  // group f = 2^m - 1 + ul: the slots j mod 2^m = ul
            constexpr int f = decltype(fc)::value, m = lg2(f + 1), ul = f + 1 - (1 << m);
            constexpr int s = bb + m, kind = PASS < NP - 1 || ul > 0 ? 2 : s == 0 ? 0 : 1;
            static_for<(1 << (R - 1 - m))>([&](auto hc) CF_INL {
                constexpr int j = (decltype(hc)::value << (m + 1)) + ul;
                this->template butterfly<kind, BD::reduces(BD::inv(s))>(x[j], x[j + (1 << m)], w, md, BD::inv(s));
            });
        };
        if constexpr (PASS > 0) {
            const double* tw = its();
            const int off = bb ? (t & ((1 << bb) - 1)) : 0;
            static_for<(1 << r) - 1>([&](auto fc) CF_INL {
                constexpr int f = decltype(fc)::value, m = lg2(f + 1), ul = f + 1 - (1 << m);
                if constexpr (PASS == NP - 1) group(fc, ul ? tw[(1 << m) - 1 + ul] : 1.0);
                else group(fc, tw[(1 << (bb + m)) - 1 + (ul << bb) + off]);
            });
        } else {
            const double* g = IW() + t;
            rows_ahead<E - 1>(g, group);
        }
    }
    CF_HD static constexpr int lg2(int x) { return x <= 1 ? 0 : 1 + lg2(x / 2); }

    // Shared-memory word of the thread's own slot j in layout 0: nobody else touches it from the last
    // inverse pass of one convolution to the first forward pass of the next, so the stages' loops
    // hold the transform's entries there instead of in registers.
    CF_HD static int own(int t, int j) { return C > 1 ? SM::X0 + lt(t) + j * CT : G::swz(t + j * T); }

    // Entries to shared memory by index.  In a cluster, pass 0's outputs (forward) go to the CTA whose
    // block holds them, and with TO_L0 the inverse transform's pass-1 outputs go to the CTA that holds
    // them in pass 0.
    template <int PASS, bool TO_L0 = false>
    CF_HD void to_smem(int t, double (&x)[E]) const {
        pin_int(t);  // recompute the addresses rather than keep the loads' addresses live across the pass
        if constexpr (C > 1 && PASS == 0) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(0, t, j);
                ex.st_remote(sm + G::swz(i & (LCN - 1)), i / LCN, fp_word(x[j]));
            }
        } else if constexpr (C > 1 && TO_L0) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(PASS, t, j);
                ex.st_remote(sm + SM::X0 + (i & (CT - 1)) + (i / T) * CT, (i & (T - 1)) / CT, fp_word(x[j]));
            }
        } else {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(PASS, t, j);
                sm[G::swz(C > 1 ? i & (LCN - 1) : i)] = fp_word(x[j]);
            }
        }
    }
    template <int PASS>
    CF_HD void from_smem(int t, double (&x)[E]) const {
        if constexpr (C > 1 && PASS == 0) {
#pragma unroll
            for (int j = 0; j < E; ++j) x[j] = fp_bits(sm[SM::X0 + lt(t) + j * CT]);
        } else {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(PASS, t, j);
                x[j] = fp_bits(sm[G::swz(C > 1 ? i & (LCN - 1) : i)]);
            }
        }
    }
    // The barrier before pass PASS reads shared memory.  Every pass but 0 works inside one block of
    // L / E entries, held by GT threads, so only the exchanges with pass 0 need all threads (the
    // cluster's); the others meet in their group of GS threads.  A group then waits for no other
    // group between the two exchanges, and its shared-memory phases overlap the others' arithmetic.
    // GS: GT, at least a warp, and at most 15 groups of more than a warp (named barriers 1 .. 15).
    static constexpr int GT = T / E < 1 ? 1 : T / E;
    static constexpr int gs_from(int g) { return g <= 32 ? (CT < 32 ? CT : 32) : (CT / g > 15 ? gs_from(2 * g) : g); }
    static constexpr int GS = gs_from(GT);
    template <int PASS, bool FWD>
    CF_HD void pass_sync() {
        if constexpr ((FWD && PASS == 1) || (!FWD && PASS == 0)) csync();
        else {
#if defined(__CUDA_ARCH__)
            if constexpr (GS <= 32) __syncwarp();
            else asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / GS), "n"(GS) : "memory");
#else
            ex.sync();
#endif
        }
    }
    // Work done behind a convolution's first barrier, where the groups of threads go on alone, so the
    // few warps that do it delay nobody: row fold_'s query partials, the power tables of step pow_.
    CF_HD void chain_work() {
        if (fold_) fold_last(fold_);
        if (pow_) ex.each([&](int t, Regs<G>&) CF_INL { power_tables(t, pow_); });
    }
    template <int PASS>
    CF_HD void fwd_chain() {  // forward passes PASS .. NP-1, pointwise, last inverse pass (PASS >= 1)
        pass_sync<PASS, true>();
        if constexpr (PASS == 1) chain_work();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            from_smem<PASS>(t, rg.f);
            fwd_pass<PASS>(t, rg.f);
            if constexpr (PASS == NP - 1) {
                pointwise(t, rg.f);
                inv_pass<PASS>(t, rg.f);
            }
            to_smem<PASS, PASS == 1 && NP == 2>(t, rg.f);  // the inverse's pass 1 only when it is the last
        });
        if constexpr (PASS + 1 < NP) fwd_chain<PASS + 1>();
    }
    template <int PASS>
    CF_HD void inv_chain() {  // inverse passes PASS .. 0 (entry: data in smem in layout PASS + 1)
        pass_sync<PASS, false>();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            from_smem<PASS>(t, rg.f);
            inv_pass<PASS>(t, rg.f);
            if constexpr (PASS > 0) to_smem<PASS, PASS == 1>(t, rg.f);
        });
        if constexpr (PASS > 0) inv_chain<PASS - 1>();
    }
    CF_HD void pointwise(int t, double (&x)[E]) const {
        const FpMod md = fm();
        auto entry = [&](auto jc, double w) CF_INL {
            constexpr int j = decltype(jc)::value;
            check(x[j], BD::fwd(LG));
            x[j] = fp_mulmod(x[j], w, md);
        };
        if constexpr (TM) {
            const u32 ta = X::tmem_addr((u32)misc()[MI_TMEM], lt(t));
            u32 v[16];
            static_for<E>([&](auto jc) CF_INL {
                constexpr int j = decltype(jc)::value, k = j % 8;
                if constexpr (k == 0) tm_load(t, ta + 2 * j, v);
                entry(jc, fp_bits((u64)v[2 * k] | ((u64)v[2 * k + 1] << 32)));
            });
        } else rows_ahead<E>(hatd() + t, entry);
    }
    // Cyclic convolution of the entries in the own slots (those at index hi and above are zero and not
    // stored) with the kernel 1/t; the results below index hi_out and at lo_out or above, and
    // index 0 if zero_out, go back to the own slots, below BD::LIM p.
    CF_HD void convolve(int hi, int lo_out, int hi_out, bool zero_out) {
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            const int tw = t & ~31;
#pragma unroll
            for (int j = 0; j < E; ++j) rg.f[j] = tw + j * T < hi ? fp_bits(sm[own(t, j)]) : 0.0;  // warp-uniform
            fwd_pass<0>(t, rg.f);
            to_smem<0>(t, rg.f);
        });
        fwd_chain<1>();
        inv_chain<NP - 2>();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            const int tw = t & ~31, te = T < 32 ? T - 1 : tw + 31;
#pragma unroll
            for (int j = 0; j < E; ++j)
                if ((te + j * T >= lo_out && tw + j * T < hi_out) || (j == 0 && zero_out)) sm[own(t, j)] = fp_word(rg.f[j]);
        });
    }
    // forward transform only (registers in layout 0 -> registers in layout NP-1), for the kernel spectrum
    template <int PASS>
    CF_HD void fwd_only_chain() {
        pass_sync<PASS, true>();
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            from_smem<PASS>(t, rg.f);
            fwd_pass<PASS>(t, rg.f);
            if constexpr (PASS < NP - 1) to_smem<PASS>(t, rg.f);
        });
        if constexpr (PASS + 1 < NP) fwd_only_chain<PASS + 1>();
    }
    CF_HD void fwd_only() {
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            fwd_pass<0>(t, rg.f);
            to_smem<0>(t, rg.f);
        });
        fwd_only_chain<1>();
    }

    // Powers of h in shared memory (the PW_* slots): base 1: h = g(v) for step v's column of V; base 0:
    // h = 1/g(v + 1) for the next step's row of S, both built behind the first barrier of step v's
    // second convolution.  A[k] = h^k (k < TA = min(CT, 32)), B[k] = h^(TA k) (k < TB = CT / TA),
    // J[j] = h^(T j) (j < E) and h^L.  Slot j of thread t holds index t + jT, whose power is
    // A[t % TA] B[t / TA] J[j].  Every entry is a power by its own thread (the first 2 PWN threads, fewer
    // taking several), a chain as long as its exponent's bits.  In a cluster, t is the thread's index in
    // its CTA and J[j] = h^(c CT + T j) carries the CTA's offset c CT.
    static constexpr int TA = CT < 32 ? CT : 32, TB = CT / TA, PWN = TA + TB + E + 1;
    CF_HD void power_tables(int t, int v) {
        double* pw = (double*)(sm + SM::PW);
        const FpMod m = fm();
        for (int x = lt(t); x < 2 * PWN; x += CT) {
            const int bs = x >= PWN, y = x - bs * PWN;
            int slot, e;
            if (y < TA) slot = PW_A + y, e = y;
            else if (y < TA + TB) slot = PW_B + (y - TA), e = TA * (y - TA);
            else if (y < TA + TB + E) slot = PW_J + (y - TA - TB), e = T * (y - TA - TB) + rank() * CT;
            else slot = PW_L, e = L;
            const double h = ldd(Gd() + 2 * v + (bs ? 0 : 3));  // g(v) or 1/g(v + 1)
            pw[bs * SM::PW_STRIDE + slot] = fp_pow_fast(h, e, m);
        }
    }
    // the thread's part A[t % TA] B[t / TA] of its slots' powers, and the table J of the slots'
    CF_HD double power_of_thread(int bs, int t, const FpMod& m) const {
        const double* pw = (const double*)(sm + SM::PW) + bs * SM::PW_STRIDE;
        const int tl = lt(t);
        return TB > 1 ? fp_mulmod(pw[PW_A + tl % TA], pw[PW_B + tl / TA], m) : pw[PW_A + tl];
    }
    CF_HD const double* power_of_slot(int bs) const { return (const double*)(sm + SM::PW) + bs * SM::PW_STRIDE + PW_J; }

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
            mi[MI_PD] = fp_word(ud(P)), mi[MI_PINVD] = fp_word(1.0 / ud(P));
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
                    fact()[k] = from_mont(run, m);
                }
                run = red[CT + t];  // 1/(k1 - 1)!
                for (int k = k1 - 1; k >= k0; --k) {  // 1/(k-1)! = k / k!
                    ifact()[k] = from_mont(run, m);
                    if (k > 0) run = mont_mul(run, to_mont((u64)k, m), m);
                }
            });
            ex.sync();
            // inv[k] = (k-1)!/k!, D[k] = 1/k!^2, g(k) and 1/g(k): C(k, d) and its inverse, or k^d and (1/k)^d
            ex.each([&](int t, Regs<G>&) CF_INL {
                const FpMod m = fm();
                auto fa = [&](int k) CF_INL { return ud(ldc<CG>(fact() + k)); };
                auto ifa = [&](int k) CF_INL { return ud(ldc<CG>(ifact() + k)); };
                for (int k = t; k <= F; k += CT) invd()[k] = k ? fp_red(fp_mulmod(ifa(k), fa(k - 1), m), m) : 0;
                for (int k = t; k <= n; k += CT) Dd()[k] = fp_red(fp_mulmod(ifa(k), ifa(k), m), m);
                for (int k = t; k <= n; k += CT) {
                    double g = 0, gi = 0;
                    if (kp.model == MODEL_REPLACEMENT) {
                        if (k > 0) {
                            g = fp_pow(ud(k), (u64)kp.d, m);
                            gi = fp_pow(invd()[k], (u64)kp.d, m);  // this thread wrote inv[k]
                        }
                    } else if (k >= kp.d) {
                        g = fp_mulmod(fp_mulmod(fa(k), ifa(kp.d), m), ifa(k - kp.d), m);
                        gi = fp_mulmod(fp_mulmod(ifa(k), fa(kp.d), m), fa(k - kp.d), m);
                    }
                    Gd()[2 * k] = fp_red(g, m);
                    Gd()[2 * k + 1] = fp_red(gi, m);
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
            mi[MI_ROOT] = from_mont(w, m);
        });
        ex.sync();
        if (rank() == 0)  // w^k, k < L, for the twiddle tables gathered below
            ex.each([&](int t, Regs<G>&) CF_INL {
                const FpMod m = fm();
                const double w = fp_centre(mi[MI_ROOT], P);
                double cur = fp_pow(w, (u64)t, m);
                const double step = fp_pow(w, (u64)CT, m);
                for (int k = t; k < L; k += CT) {
                    hatd()[k] = fp_red(cur, m);
                    cur = fp_mulmod(cur, step, m);
                }
            });
        csync();  // the first CTA's tables are read below and by every later step
        ex.each([&](int t, Regs<G>&) CF_INL {
            const double* pw = hatd();
            auto tau = [&](int s, int k) CF_INL {  // of block k of level s: exponent brv_s(k) L / 2^(s+1)
                int e = 0;
                for (int i = 0; i < s; ++i) e |= ((k >> i) & 1) << (LG - 2 - i);
                return ldd(pw + e);
            };
            auto winv = [&](int be, int pos) CF_INL { return ldd(pw + ((L - (pos << (LG - 1 - be))) & (L - 1))); };  // w_2h^-pos, h = 2^be
            double* fs = (double*)(sm + SM::TWS);
            double* is = fs + SM::FTN;
            if constexpr (C == 1) {
                for (int k = lt(t); k < SM::FTN; k += CT) fs[k] = tau(LG - 1, k);
            } else {
                for (int s = 0; s < LG - RL; ++s) {
                    const int cnt = s < R ? 1 << s : (1 << s) / C, k0 = s < R ? 0 : rank() * cnt;
                    for (int k = lt(t); k < cnt; k += CT) fs[fts_at(s, k)] = tau(s, k0 + k);
                }
            }
            for (int be = 0; be < LG - R; ++be)
                for (int k = lt(t); k < (1 << be); k += CT) is[(1 << be) - 1 + k] = winv(be, k);
            // this thread's rows of the last forward and the last inverse pass
            for (int m = 0; m < R; ++m)
                for (int ul = 0; ul < (1 << m); ++ul)
                    IW()[(size_t)((1 << m) - 1 + ul) * T + t] = winv(LG - R + m, t + ul * T);
            auto ft = [&](int f) CF_INL {  // row f: level m, group u (FwdPlan<NP - 1>)
                int m = RL - 1, u = f;
                while (u >= (1 << (R - 1 - m))) u -= 1 << (R - 1 - m), --m;
                return tau(LG - 1 - m, (t << (R - 1 - m)) + u);
            };
            if constexpr (TM) {
                const u32 ta = X::tmem_addr((u32)mi[MI_TMEM], lt(t)) + 2 * E;
                for (int c = 0; c < (FTR + 7) / 8; ++c) {
                    u32 v[16];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const u64 w = 8 * c + k < FTR ? fp_word(ft(8 * c + k)) : 0;
                        v[2 * k] = lo32(w), v[2 * k + 1] = hi32(w);
                    }
                    ex.tmem_st16(t, ta + 16 * c, v);
                }
                ex.tmem_wait_st();
            } else {
                for (int f = 0; f < FTR; ++f) FT()[(size_t)f * T + t] = ft(f);
            }
        });
        csync();  // every CTA has read the powers: the spectrum takes their place
        // kernel spectrum: hat = DIF(ker) / L with ker[t] = 1/t for 1 <= t <= n-1 (fast/cuckoo_fast.cu:829,838-839)
        ex.each([&](int t, Regs<G>& rg) CF_INL {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int i = G::idx(0, t, j);
                rg.f[j] = (i >= 1 && i < n) ? ldd(invd() + i) : 0;
            }
        });
        fwd_only();
        if (kp.keep) {  // the pair tables, for queries served later from this prime's resident V
            const KeepLayout kl = make_keep_layout(n, F);
            u64* kb = kp.keep + (size_t)b * kp.keep_words;
            ex.each([&](int t, Regs<G>&) CF_INL {
                const FpMod m = fm();
                const u64 r1 = mi[MI_R1], oneq = shoup_companion(1, P), r1q = shoup_companion(r1, P);
                auto put = [&](u64* pairs, int k, u64 v) CF_INL {
                    pairs[2 * k] = v;
                    pairs[2 * k + 1] = shoup_companion_fast(v, P, oneq, r1, r1q);
                };
                for (int k = t; k <= F; k += T) {
                    put(kb + kl.fact, k, ldc<CG>(fact() + k));
                    put(kb + kl.ifact, k, ldc<CG>(ifact() + k));
                    put(kb + kl.inv, k, fp_canon(ldd(invd() + k), m));
                }
            });
        }
        ex.each([&](int t, Regs<G>& rg) CF_INL {
            const FpMod m = fm();
            const double linv = fp_centre(P - (P - 1) / L, P);  // 1/L: L (p - (p-1)/L) = 1 mod p
            if constexpr (TM) {
                const u32 ta = X::tmem_addr((u32)mi[MI_TMEM], lt(t));
#pragma unroll
                for (int c = 0; c < E / 8; ++c) {
                    u32 v[16];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const u64 w = fp_word(fp_red(fp_mulmod(rg.f[8 * c + k], linv, m), m));
                        v[2 * k] = lo32(w), v[2 * k + 1] = hi32(w);
                    }
                    ex.tmem_st16(t, ta + 16 * c, v);
                }
                ex.tmem_wait_st();
            } else {
#pragma unroll
                for (int j = 0; j < E; ++j) hatd()[(size_t)j * T + t] = fp_red(fp_mulmod(rg.f[j], linv, m), m);
            }
        });
        csync();  // no CTA's transform exchange may start while another still reads its spectrum pass
    }

    // A row of V or S for the own slots, in two parts: ask() sends the loads of the first PRE slots,
    // put() loads the others and stores f(j, entry) for the entries i with lo <= i < hi, zero for
    // the others of the warp's slots up to index top.  Between the two the thread works on the
    // column that the convolution before has left in the own slots.
    static constexpr int PRE = E < 8 ? E : 8;
    struct RowIn {
        Row row;
        int tw, lo, hi, top;
        u64 w[PRE];
        CF_HD RowIn(const Row& r, int t, int lo_, int hi_, int top_) : row(r), tw(t & ~31), lo(lo_), hi(hi_), top(top_) {}
        CF_HD u64 word(int t, int j) const {
            const int i = t + j * T;
            u64 x = 0;
            if (tw + j * T < hi && i >= lo && i < hi) x = lds<CG>(row(j));  // the first test is warp-uniform
            return x;
        }
        CF_HD void ask(int t) {
#pragma unroll
            for (int j = 0; j < PRE; ++j) w[j] = word(t, j);
        }
        template <class F>
        CF_HD void put(u64* sm, int t, F&& f) const {
#pragma unroll
            for (int j = 0; j < PRE; ++j)
                if (tw + j * T <= top) sm[own(t, j)] = fp_word(f(j, fp_bits(w[j])));
#pragma unroll 1
            for (int j0 = PRE; j0 < E && tw + j0 * T <= top; j0 += 8) {
                u64 x[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = word(t, j0 + k);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (tw + (j0 + k) * T <= top) sm[own(t, j0 + k)] = fp_word(f(j0 + k, fp_bits(x[k])));
            }
        }
    };
    // ---------------------------------------------------------------------------------------
    // Query partial sums for row q: sum_{w<q} Vs[q][w] / (M_j - w) for every query with n_j >= q
    // (the U[w] / (M - w) sums of fast/cuckoo_fast.cu:306-323, 595-622).  The row is in the own
    // slots; only the warp's slots below q are visited, which makes a query cost about n_j^2 / 2
    // products instead of n_j L.  Each warp leaves its sum at QS[j][warp] in shared memory;
    // fold_last combines them after the next barrier.
    // ---------------------------------------------------------------------------------------
    CF_HD void query_row(int q) {
        this->query_batches(q, [&](int ja, int jb, u64* qs) CF_INL {
            int at[4], cnt = 0;
            for (int jq = ja; jq < jb; ++jq) {
                if (kp.qn[jq] >= q) at[cnt++] = jq;
                if (cnt == 4 || (jq + 1 == jb && cnt > 2)) query_group<4>(q, at, cnt, qs - (ptrdiff_t)ja * NW), cnt = 0;
            }
            if (cnt == 2) query_group<2>(q, at, cnt, qs - (ptrdiff_t)ja * NW);
            else if (cnt == 1) query_group<1>(q, at, cnt, qs - (ptrdiff_t)ja * NW);
        });
    }
    // NJ queries at a time (at[0 .. cnt - 1]): an entry is read once for all of them, and their loads,
    // products and warp sums overlap.  qs: where query 0's partials would go.
    template <int NJ>
    CF_HD void query_group(int q, const int (&at)[4], int cnt, u64* qs) {
        constexpr int U = E < 4 ? E : NJ > 2 ? 2 : 4;  // slots a turn; the next turn's inverses load meanwhile
        int M[NJ];
#pragma unroll
        for (int k = 0; k < NJ; ++k) M[k] = k < cnt ? kp.qM[at[k]] : -1;
        ex.each([&](int t, Regs<G>&) CF_INL {
            const FpMod m = fm();
            const double* iv = invd() - t;  // 1/(M - w) of slot j's w = t + jT sits at iv + M - jT
            const int tw = t & ~31;
            auto get = [&](double (&c)[NJ][U], int j0) CF_INL {  // zero past the row and for queries left out
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int k = 0; k < NJ; ++k) {
                        c[k][u] = 0;
                        if (t + (j0 + u) * T < q && M[k] >= 0) c[k][u] = ldt(iv + M[k] - (j0 + u) * T);
                    }
            };
            double acc[NJ], c[NJ][U];
#pragma unroll
            for (int k = 0; k < NJ; ++k) acc[k] = 0;
            get(c, 0);
#pragma unroll 1
            for (int j0 = 0; j0 < E && tw + j0 * T < q; j0 += U) {
                double next[NJ][U];
                get(next, j0 + U);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double x = tw + (j0 + u) * T < q ? fp_bits(sm[own(t, j0 + u)]) : 0.0;
#pragma unroll
                    for (int k = 0; k < NJ; ++k) acc[k] = fp_add(acc[k], fp_mulmod(x, c[k][u], m)), c[k][u] = next[k][u];
                }
#pragma unroll
                for (int k = 0; k < NJ; ++k) acc[k] = fp_red(acc[k], m);  // at most four terms below 0.6p and the sum below 0.51p
            }
#if defined(__CUDA_ARCH__)
            // the warp's sums: while a lane holds several, each exchange halves them (lane bit 4, then 3, picks
            // the query); at most three additions of values below 0.51p between reductions
            const unsigned mask = CT >= 32 ? 0xffffffffu : (1u << CT) - 1u;
            constexpr int O0 = CT >= 32 ? 16 : CT / 2;
            if constexpr (NJ == 4 && CT >= 32) {
                const int lane = t & 31;
                const bool up = lane & 16, up2 = lane & 8;
                const double a0 = fp_add(up ? acc[2] : acc[0], __shfl_xor_sync(mask, up ? acc[0] : acc[2], 16));
                const double a1 = fp_add(up ? acc[3] : acc[1], __shfl_xor_sync(mask, up ? acc[1] : acc[3], 16));
                double a = fp_add(up2 ? a1 : a0, __shfl_xor_sync(mask, up2 ? a0 : a1, 8));
                a = fp_add(a, __shfl_xor_sync(mask, a, 4));
                a = fp_red(a, m);
                a = fp_add(a, __shfl_xor_sync(mask, a, 2));
                a = fp_add(a, __shfl_xor_sync(mask, a, 1));
                const int k = lane >> 3;  // 2 (bit 4) + (bit 3)
                const int j = k == 0 ? at[0] : k == 1 ? at[1] : k == 2 ? at[2] : at[3];
                if ((lane & 7) == 0 && k < cnt) qs[(ptrdiff_t)j * NW + (lt(t) >> 5)] = fp_canon(a, m);
            } else {
#pragma unroll
                for (int k = 0; k < NJ; ++k) {
                    double a = acc[k];
#pragma unroll
                    for (int o = O0; o >= 1; o >>= 1) {
                        a = fp_add(a, __shfl_xor_sync(mask, a, o));
                        if (o == 4) a = fp_red(a, m);
                    }
                    if ((t & 31) == 0 && k < cnt) qs[(ptrdiff_t)at[k] * NW + (lt(t) >> 5)] = fp_canon(a, m);
                }
            }
#else
            for (int k = 0; k < NJ && k < cnt; ++k) ex.warp_sum_store(lt(t), fp_canon(acc[k], m), P, qs + (ptrdiff_t)at[k] * NW, 1);
#endif
        });
    }

    // body(j, entry of own slot j, D[i - off], lo <= i < hi) over the slots j whose index i = t + jT lies in
    // [lo, hi) for some lane of the warp (a warp-uniform range; i >= off there, or a word before D
    // is read and not used).  The next turn's D entries load meanwhile.
    template <class F>
    CF_HD void out_slots(int t, int lo, int hi, int off, F&& body) const {
        constexpr int U = E < 4 ? E : 4;
        const int tw = t & ~31, te = T < 32 ? T - 1 : tw + 31;
        const int ja = lo > te ? (lo - te + T - 1) / T : 0, jb = hi > tw ? (hi - tw - 1) / T : -1, jl = jb < E - 1 ? jb : E - 1;
        const double* p = Dd() + (t - off);
        auto get = [&](double (&c)[U], int j0) CF_INL {
#pragma unroll
            for (int k = 0; k < U; ++k) c[k] = ldt(p + (j0 + k < jl ? j0 + k : jl) * T);
        };
        if (ja > jl) return;
        double c[U];
        get(c, ja);
#pragma unroll 1
        for (int j0 = ja; j0 <= jl; j0 += U) {
            double next[U];
            get(next, j0 + U);
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int j = j0 + k, i = t + j * T;
                if (j <= jl) body(j, fp_bits(sm[own(t, j)]), c[k], i >= lo && i < hi);
                c[k] = next[k];
            }
        }
    }
    // Stage 1 after the transform: column v of S from the convolution of row v of V, then row v of S
    // times the powers of 1/g(v) into the own slots.  Its entry S[v][v], the only one of this step, is
    // computed by the thread whose slot it goes to.  Columns q <= d0 of S are zero (stage 1 skipped:
    // row q of V is zero), never written.
    CF_HD void stage1_out(int v) {
        const int n = kp.n, d0 = kp.d0;
        ex.each([&](int t, Regs<G>&) CF_INL {
            const FpMod m = fm();
            const double iv = ldd(invd() + v);
            RowIn in(Row(n, t, S(), SS(), v, tile_v0(v)), t, d0 + 1, v, v);
            in.ask(t);
            u64* col = SS() + (size_t)(v - tile_v0(v)) * (n + 1) + t;  // S[.][v], by row, from row t
            double svv = 0;
            out_slots(t, v, n, v, [&](int j, double x, double c, bool mine) CF_INL {  // rows v .. n-1 of column v
                const double y = fp_mulmod(fp_mulmod(x, c, m), iv, m);
                if (mine) check(x, BD::inv(LG)), st_stream(col + j * T, fp_word(y));
                if (t + j * T == v) svv = y;
            });
            const double ab = power_of_thread(0, t, m);  // g^-(t + jT) = ab J[j]
            const double* Js = power_of_slot(0);
            in.put(sm, t, [&](int j, double x) CF_INL {
                return fp_mulmod(t + j * T == v ? svv : x, fp_mulmod(ab, Js[j], m), m);
            });
        });
    }
    // Stage 2 after the transform: column v of V, then row v + 1 of V into the own slots (columns w < d0
    // are zero (g(w) = 0), never written).  Its entry V[v+1][v] goes to the thread of index v through
    // MI_NEXT and is put in place behind the step's last barrier.
    CF_HD void stage2_out(int v) {
        const int n = kp.n, d0 = kp.d0;
        ex.each([&](int t, Regs<G>&) CF_INL {
            const FpMod m = fm();
            const double dv = ldd(Dd() + v);
            RowIn in(Row(n, t, V(), VS(), v + 1, tile_v0(v)), t, d0, v, v);
            in.ask(t);
            const double ab = power_of_thread(1, t, m);  // g^(t + jT) = ab J[j]
            const double* Js = power_of_slot(1);
            u64* col = VS() + (size_t)(v - tile_v0(v)) * (n + 1) + t;  // V[.][v], by row, from row t
            // V[p][v] = g^p D[p-v-1] (D[v] - p e[p]) for a conv output x = e[p], c = D[p-v-1], gp = g^p
            auto entry = [&](double x, double p, double c, double gp) CF_INL {
                const double y = fp_add(dv, -fp_mulmod(x, p, m));
                return fp_word(fp_mulmod(fp_mulmod(y, c, m), gp, m));
            };
            auto next = [&](u64 y) CF_INL {  // V[v+1][v] to the CTA of index v
                if constexpr (C == 1) misc()[MI_NEXT] = y;
                else ex.st_remote(misc() + MI_NEXT, (v & (T - 1)) / CT, y);
            };
            // Entries p = v+1 .. n.  When L = n, e[n] sits at index 0 (thread 0, slot 0): done by
            // thread 0 alone, so no warp visits slot 0 only for it.
            if (n == L && t == 0) {
                const double gL = ((const double*)(sm + SM::PW))[SM::PW_STRIDE + PW_L];
                const u64 y = entry(fp_bits(sm[own(0, 0)]), (double)L, ldt(Dd() + (L - v - 1)), gL);
                st_stream(col + L, y);
                if (v + 1 == L) next(y);
            }
            out_slots(t, v + 1, n + 1, v + 1, [&](int j, double x, double c, bool mine) CF_INL {
                const u64 y = entry(x, (double)(t + j * T), c, fp_mulmod(ab, Js[j], m));
                if (mine) check(x, BD::inv(LG)), st_stream(col + j * T, y);
                if (t + j * T == v + 1) next(y);
            });
            in.put(sm, t, [&](int, double x) CF_INL { return x; });
        });
    }
    // One step of the suffix recurrence (fast/cuckoo_fast.cu:841-855), v >= d0.  On entry the own slots
    // hold row v of V, on return row v + 1.  The loops over slots around the convolution are rolled:
    // with them unrolled and a copy of the convolution for each stage the step's code did not fit
    // the instruction cache, and the 2^14 kernel spent 15 % of its warps' time waiting for
    // instructions.
    CF_HD void step(int v) {
        const int n = kp.n, d0 = kp.d0;
#pragma unroll 1
        for (int stage = v > d0 ? 1 : 2; stage <= 2; ++stage) {
            if (stage == 1) query_row(v);
            fold_ = stage == 1 ? v : 0;
            pow_ = stage == 2 ? v : 0;
            // rows v of V (entries w < v) and of S (q <= v; none at v = d0)
            convolve(stage == 1 ? v : v > d0 ? v + 1 : 0, v + stage - 1, n + stage - 1, n == L);
            if (stage == 1) stage1_out(v);
            else stage2_out(v);
        }
        if (v - tile_v0(v) == TILE - 1 && v < n - 1) {
#if defined(__CUDA_ARCH__)
            __syncwarp();  // the warp's columns of the tile are in
#else
            ex.sync();
#endif
            ex.each([&](int t, Regs<G>&) CF_INL { this->flush_rows(t, tile_v0(v)); });
        }
        csync();
        ex.each([&](int t, Regs<G>&) CF_INL {
            if (t == (v & (T - 1))) sm[own(t, v / T)] = misc()[MI_NEXT];
        });
        if (kp.keep && (v - tile_v0(v) == TILE - 1 || v == n - 1)) {
            const FpMod m = fm();
            this->keep_tile(tile_v0(v), v, [&](u64 w) CF_INL { return fp_canon(fp_bits(w), m); });
        }
    }

    // Horner finish (fast/cuckoo_fast.cu:877-890):
    //   N_bad = M! n! sum_k inv[k] ifact[n-k] ifact[M-k] Q^{n-k} ps[k],  ps[k] = sum of the warp partials.
    CF_HD void finish() {
        const int n = kp.n, d0 = kp.d0;
        u64* red = sm + SM::RED;
        if (n > d0) {  // the last row n, left in the own slots, for queries with n_j = n
            query_row(n);
            ex.sync();
            fold_last(n);
        }
        csync();  // every CTA's row sums are in
        if (rank() == 0) {  // in a cluster, the first CTA adds up the CTAs' row sums
            const FpMod m = fm();
            auto fa = [&](int k) CF_INL { return ud(ldc<CG>(fact() + k)); };
            auto ifa = [&](int k) CF_INL { return ud(ldc<CG>(ifact() + k)); };
            for (int jq = 0; jq < kp.J; ++jq) {
                const int nj = kp.qn[jq], Mj = kp.qM[jq];
                ex.each([&](int t, Regs<G>&) CF_INL {
                    double Q;
                    if (kp.model == MODEL_REPLACEMENT) Q = fp_pow(ud(Mj), (u64)kp.d, m);
                    else Q = fp_mulmod(fp_mulmod(fa(Mj), ifa(kp.d), m), ifa(Mj - kp.d), m);
                    const size_t pj = (size_t)jq * (n + 1);
                    double acc = 0;
                    for (int k = t + 1; k <= nj; k += CT) {
                        u64 s = ldc<CG>(ps_of(0) + pj + k);
                        for (int c = 1; c < C; ++c) s = madd(s, ldc<CG>(ps_of(c) + pj + k), P);
                        double y = fp_mulmod(ud(s), ldd(invd() + k), m);
                        y = fp_mulmod(y, ifa(nj - k), m);
                        y = fp_mulmod(y, ifa(Mj - k), m);
                        y = fp_mulmod(y, fp_pow(Q, (u64)(nj - k), m), m);
                        acc = fp_red(fp_add(acc, y), m);
                    }
                    red[t] = fp_canon(acc, m);
                });
                const u64 s = sum_red();
                ex.single([&]() CF_INL {
                    kp.out[kp.qout ? (size_t)kp.qout[jq] : (size_t)b * kp.J + jq] = fp_canon(fp_mulmod(fp_mulmod(ud(s), fa(nj), m), fa(Mj), m), m);
                });
            }
        }
    }

    // Tensor memory is taken once per CTA, around all the primes it runs.
    CF_HD void acquire() {
        if constexpr (TM) ex.tmem_alloc((u32*)(misc() + MI_TMEM));
    }
    CF_HD void release() {
        if constexpr (TM) ex.tmem_free((u32)misc()[MI_TMEM]);
    }
    CF_HD void run_prime() {
        setup();
        for (int v = kp.d0; v < kp.n; ++v) step(v);
        finish();
    }
    CF_HD void run() {
        acquire();
        run_prime();
        release();
    }
};

}  // namespace cfb
