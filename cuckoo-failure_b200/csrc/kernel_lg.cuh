// The persistent per-prime kernel: one CTA owns one prime from setup to residues.  Each
// transform length is instantiated in its own translation unit (k_lgNN.cu) so they build in parallel.
#pragma once
#include <cuda_runtime.h>

#include "suffix_engine.cuh"

namespace cfb {

// ------------------------------------------------------------------------------------------
// Device execution policy: `each` runs on the calling thread, `sync` is a block barrier.
// ------------------------------------------------------------------------------------------
template <class G>
struct DevExec {
    Regs<G> r;
    // this CTA's rank in its cluster (0 without clusters)
    __device__ __forceinline__ int rank() const {
        if constexpr (G::C == 1) return 0;
        else {
            u32 v;
            asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
            return (int)v;
        }
    }
    // f(t) with t the thread's index in the cluster's T threads (its CTA's CT threads without clusters)
    template <class F>
    __device__ __forceinline__ void each(F&& f) {
        if constexpr (G::C == 1) f((int)threadIdx.x, r);
        else f(rank() * G::CT + (int)threadIdx.x, r);
    }
    template <class F>
    __device__ __forceinline__ void single(F&& f) {
        if (threadIdx.x == 0) f();
    }
    __device__ __forceinline__ void sync() { __syncthreads(); }
    // Barrier of all the cluster's threads; orders their shared (local and distributed) and global
    // memory accesses at cluster scope.
    __device__ __forceinline__ void cluster_sync() {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    // Store into CTA `rk`'s shared memory at the offset `p` has in this CTA's (distributed shared memory).
    __device__ __forceinline__ void st_remote(u64* p, int rk, u64 v) const {
        u32 ra;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((u32)__cvta_generic_to_shared(p)), "r"(rk));
        asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(ra), "l"(v) : "memory");
    }
    __device__ __forceinline__ void set_error(int* err, int code) { atomicCAS(err, 0, code); }
    // Tensor memory: one warp allocates the columns the CTA's threads use, 4 E CT / 128 of the SM's
    // 512 (a power of two, at least 32); thread t of warp w owns lane 32 (w % 4) + (t % 32), columns
    // 4E (w / 4) + [0, 4E).
    static constexpr u32 TM_COLS = 4 * G::E * (G::CT / 128) < 32 ? 32 : 4 * G::E * (G::CT / 128);
    static_assert((TM_COLS & (TM_COLS - 1)) == 0 && TM_COLS <= 512, "tensor memory columns: a power of two up to 512");
    __device__ __forceinline__ void tmem_alloc(u32* slot) {
        if ((threadIdx.x >> 5) == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             (u32)__cvta_generic_to_shared(slot)), "r"(TM_COLS));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        tmem_sync();
    }
    __device__ __forceinline__ void tmem_free(u32 base) {
        tmem_sync();
        if ((threadIdx.x >> 5) == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(TM_COLS));
    }
    __device__ __forceinline__ void tmem_sync() {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    __device__ __forceinline__ static u32 tmem_addr(u32 base, int t) {
        const int w = t >> 5;
        return base + ((u32)(32 * (w & 3)) << 16) + (u32)(4 * G::E * (w >> 2));
    }
    __device__ __forceinline__ void tmem_st16(int, u32 ta, const u32 (&v)[16]) {
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(ta),
            "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
            "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]));
    }
    __device__ __forceinline__ void tmem_ld16(int, u32 ta, u32 (&v)[16]) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(ta));
    }
    __device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
    __device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
    // Sum mod p of v over the calling thread's warp; lane 0 stores it at dst[warp * stride].
    __device__ __forceinline__ void warp_sum_store(int t, u64 v, u64 P, u64* dst, size_t stride) {
        const int T = (int)blockDim.x;
        const unsigned mask = T >= 32 ? 0xffffffffu : ((1u << T) - 1u);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1)
            if (o < T) v = madd(v, __shfl_xor_sync(mask, v, o), P);
        if ((t & 31) == 0) dst[(size_t)(t >> 5) * stride] = v;
    }
    // red[0..T) holds values in [0, p); leaves their sum mod p in red[T].  Called by all threads.
    __device__ __forceinline__ void reduce_mod(u64* red, int T, u64 P) {
        const int t = threadIdx.x, lane = t & 31, w = t >> 5;
        const unsigned mask = T >= 32 ? 0xffffffffu : ((1u << T) - 1u);
        u64 v = red[t];
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1)
            if (o < T) v = madd(v, __shfl_xor_sync(mask, v, o), P);
        if (lane == 0) red[T + 1 + w] = v;
        __syncthreads();
        if (t == 0) {
            u64 s = 0;
            for (int k = 0; k < (T + 31) / 32; ++k) s = madd(s, red[T + 1 + k], P);
            red[T] = s;
        }
    }
};

// Default geometries by transform length 2^LG: 2^R entries per thread and MB resident CTAs per SM
// (the register cap 65536 / (T MB)).
//
// Primes below 2^50 (double precision), measured on B200 (ms per launch, n = 2^LG or the stated n):
//   2^14: 32 entries x 512 threads 703, 16 x 1024 853 (64 registers spill; n = 12500, 148 primes)
//   2^13: 16 x 512, 128 registers 264; 32 x 256 371, 8 x 1024 297 (148 primes)
//   2^12: 16 x 256 at 2 CTAs 238, 8 x 512 at 2 263, 32 x 128 at 4 329 (592 primes)
//   2^11: 8 x 256 at 3 CTAs 125, at 2 134, at 4 (64 registers, spills) 131, 16 x 128 at 4 139 (1184 primes)
//   2^10: 8 x 128 at 4 CTAs 17.7, 4 x 256 at 2 21.1, at 4 19.6 (n = 1000, 592 primes)
//   2^9:  8 x 64 at 8 CTAs 18.5, uncapped 23.2, 16 x 32 22.9 (2368 primes)
//   2^8:  4 x 64 at 8 CTAs 5.6, uncapped 8.0, 8 x 32 6.7, 2 x 128 13.1 (2368 primes)
//   2^7:  2 x 64 at 8 CTAs 1.80, 4 x 32 1.85 (n = 100, 2368 primes); 0.71 against 0.86 for 148 primes
// FEW: for batches of few primes, which leave SMs with one or two CTAs, more threads per prime shorten
// a step; used up to few_per_sm(LG) primes per SM:
//   2^12: 8 x 512 at 148 primes 69.9 against 78.2, at 200 138.6 against 120.5 (n = 4096): 1 per SM
//   2^10: 4 x 256 at 296 primes 10.7 against 12.0, at 360 17.9 against 14.5 (n = 1000): 2 per SM
//   2^9:  4 x 128 at 296 primes 3.7 against 4.9, at 360 6.8 against 5.8 (n = 500): 2 per SM
//   2^8:  2 x 128 at 296 primes 1.33 against 1.42, at 360 2.26 against 1.47 (n = 200): 2 per SM
//
// Primes below 2^62 (64-bit integers), registers uncapped above 2^8 (ms per launch, n = 2^LG or the
// stated n; in front the geometries with half to an eighth of the threads that were the default):
//   2^13: 16 x 512 941, 8 x 1024 762 (148 primes)     2^12: 16 x 256 269, 8 x 512 179, 4 x 1024 200 (148)
//   2^11: 16 x 128 126, 8 x 256 72, 4 x 512 51 (148); 271, 288, 204 (592)
//   2^10: 32 x 32 126, 8 x 128 32, 4 x 256 14.4 (n = 1000, 148); 499, 270, 229 (2368)
//   2^9:  16 x 32 30, 4 x 128 6.2, 2 x 256 5.5 (148); 34, 17, 21 (592)   2^8: 8 x 32 7.2, 4 x 64 2.9 (148); 8.1, 3.8 (592)
// Up to 2^8 the registers are capped at 128 (no spills), for 16 CTAs of a warp or 8 of two on an SM;
// uncapped they took 151 to 190 and fewer fitted (ms, 2368 primes, one query; in front the form with
// half the threads at 2^7 and 2^8 and all 121 to 238, then uncapped, then capped): n = 40 1.02, 1.24, 1.01; n = 64 1.48, 1.91, 1.48;
// n = 128 (1184 primes) 2.42, 2.85, 2.17; n = 200 14.07 with nine queries, 14.87, 12.54.
template <int LG, bool W, bool FEW = false>
struct Geometry {
    static constexpr int R = W          ? (LG == 14 ? 4 : LG >= 12 ? 3 : LG >= 10 ? 2 : LG >= 8 ? 2 : 1)
                             : LG == 14 ? 5
                             : LG == 13 ? 4
                             : LG == 12 ? (FEW ? 3 : 4)
                             : LG == 11 ? 3
                             : LG == 10 ? (FEW ? 2 : 3)
                             : LG == 9  ? (FEW ? 2 : 3)
                             : LG == 8  ? (FEW ? 1 : 2)
                                        : 1;
    static constexpr int MB = W          ? (LG <= 6 ? 16 : LG <= 8 ? 8 : 1)
                              : LG >= 13 ? 1
                              : LG == 12 ? (FEW ? 1 : 2)
                              : LG == 11 ? 3
                              : LG == 10 ? (FEW ? 2 : 4)
                              : LG == 9  ? (FEW ? 1 : 8)
                              : LG == 8  ? (FEW ? 1 : 8)
                              : LG == 7  ? 8
                                         : 1;
};
constexpr int few_per_sm(int lg) { return lg == 12 ? 1 : lg >= 8 && lg <= 10 ? 2 : 0; }
// Does this launch leave prime P alone?  The double-precision kernels compute nothing for a prime of
// 2^50 or above; where the host has not read the primes (cf_residues_async, batch graphs), a launch of
// the integer kernels follows for those, which leaves the primes below kp.p_lo = 2^50 alone.  A second
// launch rather than a branch: with the integer path as a function of these kernels their registers
// shifted, and they ran up to 5 % slower (n = 1500, 148 primes: 17.4 -> 18.2 ms); launched, it adds
// 2.4 to 4 us to a call (n = 24, one prime: 114.7 -> 117.0 us).
template <bool W>
__device__ __forceinline__ bool not_ours(const KParams& kp, u64 P) {
    return W ? P < kp.p_lo : P >> 50 != 0;
}
// MB: resident CTAs per SM the variant is compiled for (its register cap).
template <int LG, int R, bool W, int MB>
__global__ void __launch_bounds__(Geo<LG, R>::T, MB) k_suffix(KParams kp) {
    typedef Geo<LG, R> G;
    extern __shared__ __align__(16) u64 smem[];
    if (not_ours<W>(kp, kp.primes[blockIdx.x])) return;
    DevExec<G> ex;
    PrimeRun<G, DevExec<G>, W> pr(ex, kp, (int)blockIdx.x, smem);
    pr.run();
}

// ------------------------------------------------------------------------------------------
// Work queue: one persistent launch over many (d, prime) tables of one transform length, each with
// its own n, F, d, model and query list.  A CTA takes the next item from a device counter with an
// atomic add (nothing waits on anything), runs it in its own workspace slot, and takes another
// until the list is exhausted; the host orders the list heaviest first.
// ------------------------------------------------------------------------------------------
struct QItem {
    u64 prime;
    int n, F, d, model, J, q0;  // table size, factorial range, degree, model, queries [q0, q0 + J)
};
struct QueueParams {
    const QItem* items;
    int count;
    int* next;                // next unclaimed item (zeroed before the launch)
    const int* qn;            // [sum J] query sizes, by item
    const int* qM;
    const long long* qout;    // [sum J] output index of each query
};
template <int LG, int R, bool W, int MB>
__global__ void __launch_bounds__(Geo<LG, R>::T, MB) k_suffix_queue(KParams kp, QueueParams qp) {
    typedef Geo<LG, R> G;
    typedef PrimeRun<G, DevExec<G>, W> PR;
    extern __shared__ __align__(16) u64 smem[];
    __shared__ __align__(16) unsigned char ikp_raw[sizeof(KParams)];  // the current item's parameters
    KParams& ikp = *reinterpret_cast<KParams*>(ikp_raw);
    __shared__ int item;
    DevExec<G> ex;
    u32* tm_slot = (u32*)(smem + Smem<G, W>::MISC + MI_TMEM);
    if constexpr (PR::TM) ex.tmem_alloc(tm_slot);  // once for all the CTA's items
    for (;;) {
        if (threadIdx.x == 0) {
            item = atomicAdd(qp.next, 1);
            if (item < qp.count) {
                const QItem& q = qp.items[item];
                ikp = kp;
                ikp.primes = &q.prime;
                ikp.B = 1;
                ikp.n = q.n, ikp.F = q.F, ikp.d = q.d, ikp.model = q.model, ikp.J = q.J;
                ikp.d0 = q.model == MODEL_SUBSET ? q.d : 1;
                ikp.qn = qp.qn + q.q0, ikp.qM = qp.qM + q.q0, ikp.qout = qp.qout + q.q0;
            }
        }
        __syncthreads();
        if (item >= qp.count) break;
        PR pr(ex, ikp, 0, smem, (int)blockIdx.x);
        pr.run_prime();
        __syncthreads();  // ikp and item are rewritten for the next item
    }
    if constexpr (PR::TM) ex.tmem_free(*tm_slot);
}
typedef void (*qfn_t)(KParams, QueueParams);

typedef void (*kfn_t)(KParams);
struct KInfo {
    kfn_t fn;
    int threads;  // per CTA
    size_t smem;  // fixed dynamic shared memory; JC queries at a time add 8 JC (threads / 32)
    int r;        // log2 of the entries per thread
    qfn_t qfn;    // the work-queue form (the default geometry only)
    int mb;       // resident CTAs per SM the kernel is compiled for
    int cluster = 1;  // CTAs per prime (a thread-block cluster when above 1)
    int warps() const { return threads >= 32 ? threads / 32 : 1; }
    size_t smem_for(int JC) const { return smem + (size_t)8 * JC * warps(); }
    // queries whose partial sums a block's shared memory (optin bytes) holds at a time, at most J
    int batch_for(int J, int optin) const {
        const long fit = (long)optin > (long)smem ? ((long)optin - (long)smem) / (8 * warps()) : 0;
        return (int)(fit < J ? (fit > 0 ? fit : 1) : J);
    }
};
// W selects the kernel for primes below 2^62 (otherwise below 2^50), FEW the geometry for few primes.
template <int LG, bool W = false, bool FEW = false>
inline KInfo kinfo() {
    constexpr int R = Geometry<LG, W, FEW>::R, MB = Geometry<LG, W, FEW>::MB;
    typedef Geo<LG, R> G;
    return KInfo{&k_suffix<LG, R, W, MB>, G::T, Smem<G, W>::BYTES, R, &k_suffix_queue<LG, R, W, MB>, MB};
}
// Transform lengths above 2^14 (tables above n = 16384, primes below 2^50): one prime per cluster of
// 2^LC CTAs, one CTA per SM, launched with that cluster size (CTA b 2^LC + c is CTA c of prime b).
template <int LG, int R, int LC, bool W>
__global__ void __launch_bounds__(Geo<LG, R, LC>::CT, 1) k_suffix_cl(KParams kp) {
    typedef Geo<LG, R, LC> G;
    extern __shared__ __align__(16) u64 smem[];
    if (not_ours<W>(kp, kp.primes[blockIdx.x >> LC])) return;  // all CTAs of the cluster
    DevExec<G> ex;
    PrimeRun<G, DevExec<G>, W> pr(ex, kp, (int)blockIdx.x >> LC, smem);
    pr.run();
}
// 2^R entries per thread (16, or 8 for twice the threads per CTA when E = 8 >= C); W: primes
// below 2^62 (otherwise below 2^50).
template <int LG, int LC, int R = 4, bool W = false>
inline KInfo kinfo_cluster() {
    typedef Geo<LG, R, LC> G;
    return KInfo{&k_suffix_cl<LG, R, LC, W>, G::CT, Smem<G, W>::BYTES, R, nullptr, 1, G::C};
}
// Another geometry of the 50-bit kernel (autotuning candidates): 2^R entries per thread, MB CTAs per SM.
template <int LG, int R, int MB>
inline KInfo kinfo_geo() {
    typedef Geo<LG, R> G;
    return KInfo{&k_suffix<LG, R, false, MB>, G::T, Smem<G, 0>::BYTES, R, nullptr, MB};
}

}  // namespace cfb
