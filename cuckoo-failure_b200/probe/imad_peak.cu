// Roofline denominator probe: the device's sustained rates of 32-bit integer multiply-adds (IMAD) and of
// double-precision FMAs, measured with independent chains.  Separate library
// (libcuckoo_b200_probe.so) used only by bench.py; the engine never calls it.
#include <cuda_runtime.h>
#include <stdint.h>

static __global__ void k_imad(uint32_t* out, int iters, uint32_t m) {
    uint32_t x[8];
    for (int i = 0; i < 8; ++i) x[i] = threadIdx.x * 7 + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int i = 0; i < 8; ++i) asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(x[i]) : "r"(m), "r"(it));
    }
    uint32_t s = 0;
    for (int i = 0; i < 8; ++i) s ^= x[i];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
static __global__ void k_dfma(uint32_t* out, int iters, uint32_t m) {
    double x[8];
    const double a = 1.0 + 1e-9 * m, b = 1e-3;
    for (int i = 0; i < 8; ++i) x[i] = threadIdx.x * 7 + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int i = 0; i < 8; ++i) asm volatile("fma.rn.f64 %0, %0, %1, %2;" : "+d"(x[i]) : "d"(a), "d"(b));
    }
    double s = 0;
    for (int i = 0; i < 8; ++i) s += x[i];
    out[blockIdx.x * blockDim.x + threadIdx.x] = (uint32_t)(s != 0.0);
}

// Operations per second of `kernel` (0 on error), best of `reps` timed launches on `device`.
static double ops_per_s(void (*kernel)(uint32_t*, int, uint32_t), int device, int reps) {
    if (cudaSetDevice(device) != cudaSuccess) return 0;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int blocks = sms * 4, threads = 256, iters = 16384;
    uint32_t* d = nullptr;
    if (cudaMalloc(&d, sizeof(uint32_t) * blocks * threads) != cudaSuccess) return 0;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    kernel<<<blocks, threads>>>(d, iters, 12345u);
    double best = 0;
    for (int r = 0; r < reps; ++r) {
        cudaEventRecord(a);
        kernel<<<blocks, threads>>>(d, iters, 12345u);
        cudaEventRecord(b);
        cudaEventSynchronize(b);
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        const double ops = (double)blocks * threads * 8.0 * iters;
        if (ms > 0 && ops / (ms * 1e-3) > best) best = ops / (ms * 1e-3);
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(d);
    return cudaGetLastError() == cudaSuccess ? best : 0;
}
extern "C" double cfp_imad_ops_per_s(int device, int reps) { return ops_per_s(k_imad, device, reps); }
extern "C" double cfp_dfma_ops_per_s(int device, int reps) { return ops_per_s(k_dfma, device, reps); }
