// A stand-in for libcudart with two devices and no GPU, for tests of the host code.
//
// Memory is host memory, kernels do nothing, graphs hold their kernel nodes.
// It refuses what the real library refuses of a thread whose current device is not the
// stream's: kernel launches, and parameter updates of a graph's kernel
// nodes.  A copy from pageable memory takes fake_copy_ms of its stream's time, and
// fails where the test asks for it (fake_refuse: at the call; fake_fault: when
// its stream is waited for).
#include <cuda_runtime_api.h>

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

using Clock = std::chrono::steady_clock;

namespace {
struct Stream {
    int device;
    Clock::time_point busy;
    cudaError_t fault = cudaSuccess;
};
struct Graph {
    int device;
    std::vector<const void*> kernels;
};
thread_local int t_device = 0;
thread_local cudaError_t t_error = cudaSuccess;
thread_local Graph* t_capture = nullptr;
std::mutex g_mutex;
std::map<const char*, std::pair<size_t, cudaMemoryType>> g_memory;
std::atomic<int> g_launches{0}, g_updates{0}, g_refuse{0}, g_slow{0}, g_staged{0}, g_direct{0}, g_waits{0}, g_live_streams{0};

cudaError_t fail(cudaError_t e) { return t_error = e; }
Stream* stream_of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }

cudaError_t allocate(void** p, size_t n, cudaMemoryType type) {
    *p = calloc(1, n + 256);
    std::lock_guard<std::mutex> lock(g_mutex);
    g_memory[static_cast<char*>(*p)] = {n, type};
    return cudaSuccess;
}

cudaError_t release(void* p) {
    std::lock_guard<std::mutex> lock(g_mutex);
    g_memory.erase(static_cast<char*>(p));
    free(p);
    return cudaSuccess;
}

cudaMemoryType type_of(const void* p) {
    std::lock_guard<std::mutex> lock(g_mutex);
    auto it = g_memory.upper_bound(static_cast<const char*>(p));
    if (it == g_memory.begin()) return cudaMemoryTypeUnregistered;
    --it;
    return static_cast<const char*>(p) < it->first + it->second.first ? it->second.second : cudaMemoryTypeUnregistered;
}

cudaError_t copy(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t height, cudaStream_t s) {
    if (type_of(src) == cudaMemoryTypeUnregistered) {
        if (g_refuse) return fail(cudaErrorInvalidValue);
        ++g_direct;
        const int first = *static_cast<const unsigned char*>(src);
        std::lock_guard<std::mutex> lock(g_mutex);
        Stream* st = stream_of(s);
        const auto now = Clock::now();
        // A frame that starts with 200 is slow, one that starts with 100 fails.
        if (g_slow && first == 200) st->busy = std::max(st->busy, now) + std::chrono::milliseconds(g_slow);
        if (first == 100) st->fault = cudaErrorUnknown;
    } else {
        ++g_staged;
    }
    if (t_capture) return cudaSuccess;
    for (size_t y = 0; y < height; ++y) {
        memcpy(static_cast<char*>(dst) + y * dpitch, static_cast<const char*>(src) + y * spitch, width);
    }
    return cudaSuccess;
}

cudaError_t launch(const void* f, cudaStream_t s) {
    if (t_capture) {
        t_capture->kernels.push_back(f);
        return cudaSuccess;
    }
    if (s && stream_of(s)->device != t_device) return fail(cudaErrorInvalidResourceHandle);
    ++g_launches;
    return cudaSuccess;
}
}  // namespace

extern "C" {
int fake_launches() { return g_launches; }
int fake_updates() { return g_updates; }
int fake_copies_from_page_locked() { return g_staged; }
int fake_direct_copies() { return g_direct; }
int fake_waits() { return g_waits; }
int fake_streams() { return g_live_streams; }
void fake_refuse(int on) { g_refuse = on; }
void fake_slow(int ms) { g_slow = ms; }

cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 1) return fail(cudaErrorInvalidDevice);
    t_device = d;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = t_error; t_error = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n, cudaMemoryTypeDevice); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return allocate(p, n, cudaMemoryTypeHost); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeHost(void* p) { return release(p); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    memset(a, 0, sizeof(*a));
    a->type = type_of(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    return copy(d, n, s, n, n, 1, st);
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t st) {
    return copy(d, dp, s, sp, w, h, st);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    ++g_live_streams;
    *s = reinterpret_cast<cudaStream_t>(new Stream{t_device, Clock::now()});
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { --g_live_streams; delete stream_of(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (!s) return cudaSuccess;
    ++g_waits;
    for (;;) {
        Clock::time_point until;
        {
            std::lock_guard<std::mutex> lock(g_mutex);
            Stream* st = stream_of(s);
            until = st->busy;
            if (until <= Clock::now()) {
                const cudaError_t e = st->fault;
                st->fault = cudaSuccess;
                return e == cudaSuccess ? e : fail(e);
            }
        }
        std::this_thread::sleep_until(until);
    }
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    t_capture = new Graph{stream_of(s)->device, {}};
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = reinterpret_cast<cudaGraph_t>(t_capture);
    t_capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { delete reinterpret_cast<Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t* nodes, size_t* n) {
    Graph* graph = reinterpret_cast<Graph*>(g);
    *n = graph->kernels.size();
    for (size_t i = 0; nodes && i < *n; ++i) nodes[i] = reinterpret_cast<cudaGraphNode_t>(&graph->kernels[i]);
    return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType* t) {
    *t = cudaGraphNodeTypeKernel;
    return cudaSuccess;
}
cudaError_t cudaGraphKernelNodeGetParams(cudaGraphNode_t n, cudaKernelNodeParams* p) {
    memset(p, 0, sizeof(*p));
    p->func = const_cast<void*>(*reinterpret_cast<const void**>(n));
    return cudaSuccess;
}
cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t e, cudaGraphNode_t, const cudaKernelNodeParams*) {
    if (reinterpret_cast<Graph*>(e)->device != t_device) return fail(cudaErrorInvalidDeviceFunction);
    ++g_updates;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(new int); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<int*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) { return launch(f, s); }

// What nvcc's host code calls.
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t s) {
    return launch(reinterpret_cast<const void*>(k), s);
}
namespace {
thread_local struct { dim3 grid, block; size_t smem; void* stream; } t_config;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
    t_config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = t_config.grid;
    *block = t_config.block;
    *smem = t_config.smem;
    *static_cast<void**>(stream) = t_config.stream;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
