// Test harness (not product code): stands in for the CUDA runtime, so that the host code of the engine
// runs on the CPU.  Two devices with SM counts that a test sets; memory is addresses only, copies to
// the host give zeros, and a launch is recorded (device, grid, block, dynamic shared memory) and not run.
#include <cuda_runtime_api.h>

#include <cstring>
#include <vector>

namespace {
struct Launch {
    int device, grid, block;
    long smem;
};
int current = 0, sms[2] = {148, 148};
std::vector<Launch> launches;
char* next_address = (char*)(1ull << 40);
cudaError_t give(void** p, size_t bytes) {
    *p = next_address;
    next_address += (bytes + 511) & ~(size_t)255;
    return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_set_sms(int device, int n) { sms[device] = n; }
void fake_clear() { launches.clear(); }
int fake_launches() { return (int)launches.size(); }
void fake_launch(int i, int* out) {
    const Launch& l = launches[(size_t)i];
    out[0] = l.device, out[1] = l.grid, out[2] = l.block, out[3] = (int)l.smem;
}

cudaError_t cudaGetDevice(int* d) { return *d = current, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return current = d, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
    *v = a == cudaDevAttrMultiProcessorCount ? sms[d] : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = (size_t)100 << 30, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return give(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return give(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = new char[n](), cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return delete[] (char*)p, cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void*, size_t n, cudaMemcpyKind k) {
    if (k == cudaMemcpyDeviceToHost) std::memset(d, 0, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return give(p, 1 << 26); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { return *p = nullptr, cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { return *n = 1, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { return *n = 1, cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
    launches.push_back({current, (int)g.x, (int)b.x, (long)smem});
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
    launches.push_back({current, (int)c->gridDim.x, (int)c->blockDim.x, (long)c->dynamicSmemBytes});
    return cudaSuccess;
}

// what the compiler's host stubs call
static dim3 cfg_grid, cfg_block;
static size_t cfg_smem;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void*) { return cfg_grid = g, cfg_block = b, cfg_smem = smem, 0u; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = cfg_grid, *b = cfg_block, *smem = cfg_smem, *(void**)s = nullptr;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 1; }
}
