// A CUDA runtime without a device, preloaded before the engine library so that its host code runs on a machine that
// has no GPU: memory is host memory, kernels are counted and not run, and what the tests ask about is recorded.
//
//   * a host-to-device cudaMemcpyAsync copies at the next synchronisation, as a copy from pageable memory may, and
//     counts the sources that changed in between (fake_changed_sources);
//   * launches (fake_launches) and streams by priority (fake_streams_of).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

namespace {
std::recursive_mutex mu;
struct Pending {
    void* dst;
    const void* src;
    std::vector<char> then;
};
std::vector<Pending> pending;
std::map<void*, int> streams;   // priority
int changed = 0, launches = 0, made[64] = {};
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
void* cfg_stream;

cudaError_t flush() {
    std::lock_guard<std::recursive_mutex> lk(mu);
    for (auto& p : pending) {
        if (std::memcmp(p.src, p.then.data(), p.then.size()) != 0) ++changed;
        std::memcpy(p.dst, p.src, p.then.size());
    }
    pending.clear();
    return cudaSuccess;
}
cudaError_t make_stream(cudaStream_t* s, int priority) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    *s = reinterpret_cast<cudaStream_t>(std::calloc(1, 64));
    streams[*s] = priority;
    ++made[-priority];
    return cudaSuccess;
}
}  // namespace

extern "C" {
int fake_changed_sources() { return changed; }
int fake_launches() { return launches; }
int fake_streams_of(int priority) { return made[-priority]; }   // created so far with this priority
void* fake_stream(int priority) {
    cudaStream_t s;
    make_stream(&s, priority);
    return s;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return flush(); }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }

cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n + 256, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { flush(); std::free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t* fr, size_t* tot) { *fr = *tot = size_t(8) << 30; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (kind == cudaMemcpyHostToDevice) {
        pending.push_back({d, s, std::vector<char>((const char*)s, (const char*)s + n)});
        return cudaSuccess;
    }
    flush();
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { flush(); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { flush(); std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make_stream(s, 0); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int priority) { return make_stream(s, priority); }
cudaError_t cudaStreamGetPriority(cudaStream_t s, int* priority) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const auto it = streams.find(s);
    *priority = it == streams.end() ? 0 : it->second;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    streams.erase(s);
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return flush(); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = reinterpret_cast<cudaGraphExec_t>(1); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(std::calloc(1, 64)); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return flush(); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { ++launches; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { ++launches; return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { ++launches; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, struct CUstream_st* s) {
    cfg_grid = g; cfg_block = b; cfg_smem = m; cfg_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = cfg_grid; *b = cfg_block; *m = cfg_smem;
    *static_cast<void**>(s) = cfg_stream;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* h = nullptr; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
}
