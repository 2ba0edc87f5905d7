// fake_cudart.cpp -- the part of the CUDA runtime's interface that the engine's
// host code calls, without a GPU: device memory is host memory, kernels are
// counted instead of run, a stream capture collects its launches and a graph
// launch counts them again.  Linked with the engine's own objects in place of
// the runtime (tests/host_engine.py), it lets CPU tests look at what the host
// code does: which launches it makes, what it does when an allocation fails, and
// whether a graph is launched after memory it was captured with has been freed.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {

struct Graph {
    std::vector<std::string> kernels;
    std::set<const void *> memory;    // allocations of the time of the capture
};

std::map<const void *, std::string> g_name;       // host stub -> kernel
std::map<const void *, int> g_smem_limit;         // MaxDynamicSharedMemorySize
std::map<const void *, size_t> g_alloc;
std::set<Graph *> g_execs;
Graph *g_capture = nullptr;
std::vector<std::string> g_direct, g_replayed;    // kernels launched by themselves / by graphs
int g_graph_launches = 0, g_stale_launches = 0, g_captures = 0;
long g_fail_after = -1;                           // allocations until one fails (-1: none does)
cudaError_t g_last = cudaSuccess;

struct Config {
    dim3 grid, block;
    size_t smem;
    void *stream;
};
std::vector<Config> g_config;

cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}

cudaError_t launch(const void *f, size_t smem) {
    const auto lim = g_smem_limit.find(f);
    if (smem > (lim == g_smem_limit.end() ? 48u * 1024u : (size_t)lim->second)) return set(cudaErrorInvalidValue);
    const auto it = g_name.find(f);
    const std::string name = it == g_name.end() ? "?" : it->second;
    if (g_capture) g_capture->kernels.push_back(name);
    else g_direct.push_back(name);
    return cudaSuccess;
}

void *handle() { return std::malloc(8); }

}  // namespace

// ---- what the tests read and set
extern "C" {
void fake_reset() {
    g_direct.clear();
    g_replayed.clear();
    g_graph_launches = g_stale_launches = g_captures = 0;
}
int fake_direct() { return (int)g_direct.size(); }
int fake_replayed() { return (int)g_replayed.size(); }
int fake_graph_launches() { return g_graph_launches; }
int fake_stale_launches() { return g_stale_launches; }
int fake_captures() { return g_captures; }
void fake_fail_malloc(long after) { g_fail_after = after; }   // the allocation after `after` more
int fake_count(const char *part) {                            // launches of kernels whose name has this part
    int n = 0;
    for (const auto *v : {&g_direct, &g_replayed})
        for (const std::string &s : *v) n += s.find(part) != std::string::npos;
    return n;
}
int fake_live(size_t bytes) {                                 // live allocations of this size
    int n = 0;
    for (const auto &a : g_alloc) n += a.second == bytes;
    return n;
}
}

extern "C" {
// ---- registration and <<< >>> launches
void **__cudaRegisterFatBinary(void *) { return reinterpret_cast<void **>(handle()); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    g_name[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *stream) {
    g_config.push_back({grid, block, smem, stream});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    const Config c = g_config.back();
    g_config.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *reinterpret_cast<void **>(stream) = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t smem, cudaStream_t) {
    return launch(k, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
    return launch(f, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > 227 * 1024) return set(cudaErrorInvalidValue);
        g_smem_limit[f] = v;
    }
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *f) {
    std::memset(a, 0, sizeof(*a));
    const auto it = g_smem_limit.find(f);
    a->maxDynamicSharedSizeBytes = it == g_smem_limit.end() ? 48 * 1024 : it->second;
    return cudaSuccess;
}

// ---- device
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "fake runtime"; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = nullptr; return set(cudaErrorInvalidValue); }

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = nullptr;
    if (g_fail_after == 0) {
        g_fail_after = -1;
        return set(cudaErrorMemoryAllocation);
    }
    if (g_fail_after > 0) g_fail_after--;
    *p = std::calloc(n ? n : 1, 1);
    g_alloc[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (!p) return cudaSuccess;
    g_alloc.erase(p);
    // the block itself is kept, so that its address is not given out again
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (!g_capture) std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    if (!g_capture) std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(handle()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    g_capture = new Graph();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    g_captures++;
    *g = reinterpret_cast<cudaGraph_t>(g_capture);
    g_capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
    Graph *e = new Graph(*reinterpret_cast<Graph *>(g));
    for (const auto &a : g_alloc) e->memory.insert(a.first);
    g_execs.insert(e);
    *x = reinterpret_cast<cudaGraphExec_t>(e);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph *>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    g_execs.erase(reinterpret_cast<Graph *>(x));
    delete reinterpret_cast<Graph *>(x);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    const Graph *e = reinterpret_cast<Graph *>(x);
    g_graph_launches++;
    if (!g_execs.count(const_cast<Graph *>(e))) {
        g_stale_launches++;
        return cudaSuccess;
    }
    for (const void *p : e->memory)
        if (!g_alloc.count(p)) {
            g_stale_launches++;
            break;
        }
    g_replayed.insert(g_replayed.end(), e->kernels.begin(), e->kernels.end());
    return cudaSuccess;
}
}
