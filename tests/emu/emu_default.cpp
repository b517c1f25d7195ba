// Test harness (not product code): the per-prime phase code in a default geometry, with exactly the shared
// memory and the workspace that a launch of it gets, words behind both checked for writes.
#include "emu_exec.hpp"

using namespace cfb;

static constexpr u64 MARK = 0xA5A5A5A5A5A5A5A5ull;
static bool untouched(const std::vector<u64>& v, size_t from) {
    for (size_t i = from; i < v.size(); ++i)
        if (v[i] != MARK) return false;
    return true;
}
template <int LG, int R, bool W>
static int run_one(KParams& kp) {
    typedef Geo<LG, R> G;
    kp.lay = make_layout(kp.n, kp.F, G::L, kp.J, G::NW, R);
    kp.ws_words = kp.lay.total;
    const size_t words = Smem<G, W>::bytes_for(kp.J) / 8;
    std::vector<u64> ws(kp.ws_words + 256, MARK), smem(words + 256, MARK);
    kp.ws = ws.data();
    HostExec<G> ex;
    PrimeRun<G, HostExec<G>, W> pr(ex, kp, 0, smem.data());
    pr.run();
    return untouched(ws, kp.ws_words) && untouched(smem, words) ? 0 : -7;
}

extern "C" int emu_default(uint64_t prime, int nmax, int d, int model, const int* qn, const int* qM, int J, uint64_t* out, int lg, int R) {
    KParams kp;
    int err = 0, rc = -4;
    kp.primes = &prime, kp.B = 1, kp.n = nmax, kp.F = nmax, kp.d = d, kp.d0 = model == MODEL_SUBSET ? d : 1, kp.model = model;
    for (int j = 0; j < J; ++j) kp.F = qM[j] > kp.F ? qM[j] : kp.F;
    kp.J = J, kp.qn = qn, kp.qM = qM, kp.out = out, kp.err = &err;
    try {
        switch ((prime >> 50 ? 1000 : 0) + 10 * lg + R) {
            case 41: rc = run_one<4, 1, false>(kp); break;
            case 51: rc = run_one<5, 1, false>(kp); break;
            case 61: rc = run_one<6, 1, false>(kp); break;
            case 123: rc = run_one<12, 3, false>(kp); break;
            case 124: rc = run_one<12, 4, false>(kp); break;
            case 134: rc = run_one<13, 4, false>(kp); break;
            case 1041: rc = run_one<4, 1, true>(kp); break;
            case 1051: rc = run_one<5, 1, true>(kp); break;
            case 1061: rc = run_one<6, 1, true>(kp); break;
            case 1144: rc = run_one<14, 4, true>(kp); break;
        }
    } catch (const std::runtime_error&) {
        return -6;
    }
    return err ? -5 : rc;
}
