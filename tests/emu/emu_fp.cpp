// Test harness (not product code): the double-precision arithmetic (fparith.cuh) by itself, and the
// per-prime phase code in the kernels' default geometries, on the CPU.
#include "emu_exec.hpp"

using namespace cfb;

template <int LG, int R, bool W>
static void run_one(const KParams& kp) {
    typedef Geo<LG, R> G;
    std::vector<u64> smem(Smem<G, W>::bytes_for(kp.JC > 0 ? kp.JC : kp.J) / 8, 0xA5A5A5A5A5A5A5A5ull);
    HostExec<G> ex;
    PrimeRun<G, HostExec<G>, W> pr(ex, kp, 0, smem.data());
    pr.run();
}

extern "C" {
void fp_products(const double* x, const double* w, double p, long n, double* out) {
    const FpMod m{p, 1.0 / p};
    for (long i = 0; i < n; ++i) out[i] = fp_mulmod(x[i], w[i], m);
}
void fp_reductions(const double* x, double p, long n, double* out, uint64_t* canon) {
    const FpMod m{p, 1.0 / p};
    for (long i = 0; i < n; ++i) out[i] = fp_red(x[i], m), canon[i] = fp_canon(x[i], m);
}
double fp_power_fast(double x, int k, double p) { return fp_pow_fast(x, k, FpMod{p, 1.0 / p}); }

// one prime's residues with 2^R entries per thread and the transform length forced to 2^lg, the
// queries' partial sums held JC at a time (0: all)
int emu_fp_geo(uint64_t prime, int nmax, int d, int model, const int* qn, const int* qM, int J, uint64_t* out, int lg, int R, int JC) {
    int F = nmax;
    for (int j = 0; j < J; ++j) F = qM[j] > F ? qM[j] : F;
    if (model == MODEL_SUBSET && d > F) F = d;
    const int T = 1 << (lg - R);
    const Layout lo = make_layout(nmax, F, 1 << lg, J, T >= 32 ? T / 32 : 1, R);
    std::vector<u64> ws(lo.total, 0xA5A5A5A5A5A5A5A5ull);
    int err = 0;
    KParams kp;
    kp.primes = &prime, kp.B = 1, kp.n = nmax, kp.F = F, kp.d = d, kp.d0 = model == MODEL_SUBSET ? d : 1;
    kp.model = model, kp.J = J, kp.qn = qn, kp.qM = qM, kp.ws = ws.data(), kp.ws_words = lo.total, kp.lay = lo;
    kp.out = out, kp.err = &err, kp.JC = JC;
    const bool wide = prime >= (1ull << 50);
    const int key = (wide ? 1000 : 0) + 10 * lg + R;
    try {
        switch (key) {
            case 145: run_one<14, 5, false>(kp); break;
            case 124: run_one<12, 4, false>(kp); break;
            case 113: run_one<11, 3, false>(kp); break;
            case 103: run_one<10, 3, false>(kp); break;
            case 102: run_one<10, 2, false>(kp); break;
            case 93: run_one<9, 3, false>(kp); break;
            case 92: run_one<9, 2, false>(kp); break;
            case 82: run_one<8, 2, false>(kp); break;
            case 81: run_one<8, 1, false>(kp); break;
            case 71: run_one<7, 1, false>(kp); break;
            case 1133: run_one<13, 3, true>(kp); break;
            case 1123: run_one<12, 3, true>(kp); break;
            case 1112: run_one<11, 2, true>(kp); break;
            case 1102: run_one<10, 2, true>(kp); break;
            case 1092: run_one<9, 2, true>(kp); break;
            case 1082: run_one<8, 2, true>(kp); break;
            case 1071: run_one<7, 1, true>(kp); break;
            default: return -4;
        }
    } catch (const std::runtime_error&) {
        return -6;
    }
    return err ? -5 : 0;
}
}
