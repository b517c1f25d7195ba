// Test harness (not product code): the double-precision arithmetic (fparith.cuh) by itself, and the
// per-prime phase code in the default geometries of the kernels for primes below 2^50, on the CPU.
#include "emu_exec.hpp"

using namespace cfb;

extern "C" {
void fp_products(const double* x, const double* w, double p, long n, double* out) {
    const FpMod m{p, 1.0 / p};
    for (long i = 0; i < n; ++i) out[i] = fp_mulmod(x[i], w[i], m);
}
void fp_reductions(const double* x, double p, long n, double* out, uint64_t* canon) {
    const FpMod m{p, 1.0 / p};
    for (long i = 0; i < n; ++i) out[i] = fp_red(x[i], m), canon[i] = fp_canon(x[i], m);
}
double fp_power_small(double x, int k, double p) { return fp_pow_small(x, k, FpMod{p, 1.0 / p}); }

// one prime's residues with 2^R entries per thread and the transform length forced to 2^lg
int emu_fp_geo(uint64_t prime, int nmax, int d, int model, const int* qn, const int* qM, int J, uint64_t* out, int lg, int R) {
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
    kp.out = out, kp.err = &err;
    try {
        if (lg == 14 && R == 5) run_geo<14, 5>(kp);
        else if (lg == 11 && R == 3) run_geo<11, 3>(kp);
        else if (lg == 10 && R == 3) run_geo<10, 3>(kp);
        else if (lg == 10 && R == 2) run_geo<10, 2>(kp);
        else if (lg == 9 && R == 3) run_geo<9, 3>(kp);
        else if (lg == 9 && R == 2) run_geo<9, 2>(kp);
        else if (lg == 8 && R == 2) run_geo<8, 2>(kp);
        else if (lg == 8 && R == 1) run_geo<8, 1>(kp);
        else if (lg == 7 && R == 1) run_geo<7, 1>(kp);
        else return -4;
    } catch (const std::runtime_error&) {
        return -6;
    }
    return err ? -5 : 0;
}
}
