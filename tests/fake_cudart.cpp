// fake_cudart.cpp -- a CUDA runtime of two B200-shaped devices without a GPU.
//
// Preloaded under the product library (LD_PRELOAD), it keeps device memory in
// host memory, runs no kernel, and checks what a device checks of a launch: the
// dynamic shared memory and the cluster size must be within what
// cudaFuncSetAttribute allowed ON THAT DEVICE.  Each launch is one line of
// $FAKE_CUDART_LOG: device, kernel (mangled), grid, threads, shared memory,
// cluster, cooperative, status.  So the host side (plans, routes, attributes)
// is tested on the CPU, with more devices than the machine has.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

namespace {

constexpr int kDevices = 2, kSms = 148, kOptin = 232448;

struct Attr {
    int smem = 48 * 1024;
    int big_clusters = 0;
};

std::mutex mu;
std::map<const void*, std::string>& names() {
    static std::map<const void*, std::string> m;
    return m;
}
std::map<std::pair<int, const void*>, Attr>& attrs() {
    static std::map<std::pair<int, const void*>, Attr> m;
    return m;
}
thread_local int t_device = 0;
thread_local cudaError_t t_last = cudaSuccess;
thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} t_call;

cudaError_t keep(cudaError_t e) {
    if (e != cudaSuccess) t_last = e;
    return e;
}

template <class T>
T dummy() {
    return static_cast<T>(std::calloc(1, 8));
}

cudaError_t launch(const void* fn, dim3 grid, dim3 block, size_t smem, int cluster, int coop) {
    std::lock_guard<std::mutex> lk(mu);
    const Attr a = attrs()[{t_device, fn}];
    cudaError_t e = cudaSuccess;
    if (smem > (size_t)a.smem) e = cudaErrorInvalidValue;
    if (cluster > 8 && !a.big_clusters) e = cudaErrorInvalidClusterSize;
    if (cluster > 1 && grid.x % (unsigned)cluster) e = cudaErrorInvalidConfiguration;
    if (const char* path = std::getenv("FAKE_CUDART_LOG")) {
        if (FILE* f = std::fopen(path, "a")) {
            std::fprintf(f, "%d %s %u %u %zu %d %d %d\n", t_device, names()[fn].c_str(),
                         grid.x * grid.y * grid.z, block.x, smem, cluster, coop, (int)e);
            std::fclose(f);
        }
    }
    return keep(e);
}

// cuTensorMapEncodeTiled
int encode(void*, ...) { return 0; }

}  // namespace

extern "C" {

void** __cudaRegisterFatBinary(void*) { return dummy<void**>(); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
    std::lock_guard<std::mutex> lk(mu);
    names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
    t_call = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = t_call.grid;
    *b = t_call.block;
    *smem = t_call.smem;
    *static_cast<cudaStream_t*>(s) = t_call.stream;
    return cudaSuccess;
}

cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d >= kDevices) return keep(cudaErrorInvalidDevice);
    t_device = d;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = t_device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount             ? kSms
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kOptin
         : a == cudaDevAttrCooperativeLaunch            ? 1
                                                        : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = t_last;
    t_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e ? "error of the fake runtime" : "ok"; }

cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute a, int v) {
    std::lock_guard<std::mutex> lk(mu);
    Attr& t = attrs()[{t_device, fn}];
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > kOptin) return keep(cudaErrorInvalidValue);
        t.smem = v;
    }
    if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) t.big_clusters = v;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* out, const void* fn) {
    std::lock_guard<std::mutex> lk(mu);
    std::memset(out, 0, sizeof *out);
    out->maxDynamicSharedSizeBytes = attrs()[{t_device, fn}].smem;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* fn,
                                                                   int threads, size_t smem,
                                                                   unsigned) {
    std::lock_guard<std::mutex> lk(mu);
    const int by_smem = (int)(233472 / (smem + 1024)), by_threads = 2048 / threads;
    *n = smem > (size_t)attrs()[{t_device, fn}].smem ? 0 : by_smem < by_threads ? by_smem : by_threads;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int threads,
                                                          size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, fn, threads, smem, 0);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* fn, const cudaLaunchConfig_t* c) {
    int cluster = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension)
            cluster = (int)c->attrs[i].val.clusterDim.x;
    std::lock_guard<std::mutex> lk(mu);
    const Attr a = attrs()[{t_device, fn}];
    *n = 0;
    if (c->dynamicSmemBytes > (size_t)a.smem) return keep(cudaErrorInvalidValue);
    if (cluster > 8 && !a.big_clusters) return keep(cudaErrorInvalidClusterSize);
    *n = 8 * (18 / cluster);  // 8 GPCs of 18 SMs
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
    return launch(fn, g, b, smem, 1, 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
    int cluster = 1, coop = 0;
    for (unsigned i = 0; i < c->numAttrs; ++i) {
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension)
            cluster = (int)c->attrs[i].val.clusterDim.x;
        if (c->attrs[i].id == cudaLaunchAttributeCooperative) coop = c->attrs[i].val.cooperative;
    }
    return launch(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes, cluster, coop);
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long,
                                    cudaDriverEntryPointQueryResult* q) {
    *p = reinterpret_cast<void*>(&encode);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char space[1 << 20];
    *p = space;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) {
    *p = std::calloc(n ? n : 1, 1);
    return *p ? cudaSuccess : keep(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t* fr, size_t* total) {
    *fr = *total = size_t(180) << 30;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = dummy<cudaStream_t>();
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaFree(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = dummy<cudaGraph_t>();
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = dummy<cudaEvent_t>();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaFree(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = dummy<cudaGraphExec_t>();
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return cudaFree(g); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return cudaFree(x); }

}  // extern "C"
