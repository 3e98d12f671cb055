// A stand-in for the CUDA runtime on the host, for tests of the library's host
// code without a GPU (tests/host_runtime.py links it with the library's
// objects).  Device memory is host memory, copies and clears happen at once,
// kernels do nothing.  Work on a stream counts as pending until something waits
// for it, so that a test can see who waits for what; a hook sees every call
// first and can make it fail.
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

namespace {

struct Stream {
    unsigned long long enqueued = 0, done = 0;
    bool capturing = false;
};
struct Event {
    Stream *stream = nullptr;  // null: never recorded
    unsigned long long at = 0;
    int life = 0;  // the device's when it was made
};
using Hook = int (*)(const char *name, void *ptr, size_t size, void *stream);

std::recursive_mutex g_mutex;
Hook g_hook = nullptr;
int g_life = 0, g_staleUses = 0;
Stream g_legacy;
std::map<Stream *, bool> g_streams;  // made by the library
std::map<void *, size_t> g_blocks;   // cudaMalloc'd
size_t g_bytes = 0, g_capacity = size_t(180) << 30;
cudaError_t g_last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t shared;
    void *stream;
};
std::vector<Config> g_configs;

// by host stub or handle; the objects register their kernels while the library loads
std::map<const void *, std::string> &kernels() {
    static std::map<const void *, std::string> names;
    return names;
}

using Lock = std::lock_guard<std::recursive_mutex>;

constexpr size_t kArrayBytes = size_t(16) << 20;  // more than any __device__ array of the library
void *scratchArray() {
    static void *p = std::calloc(1, kArrayBytes);
    return p;
}
Stream *of(cudaStream_t s) { return s ? reinterpret_cast<Stream *>(s) : &g_legacy; }
cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}
cudaError_t ask(const char *name, const void *ptr = nullptr, size_t size = 0, cudaStream_t s = nullptr) {
    Hook hook;
    {
        Lock lock(g_mutex);
        hook = g_hook;
    }
    return hook ? result((cudaError_t)hook(name, const_cast<void *>(ptr), size, (void *)s)) : cudaSuccess;
}
bool anyCapture() {
    for (auto &s : g_streams)
        if (s.first->capturing) return true;
    return false;
}
void enqueue(cudaStream_t s) {
    Lock lock(g_mutex);
    if (!of(s)->capturing) of(s)->enqueued++;
}
void finishAll() {
    g_legacy.done = g_legacy.enqueued;
    for (auto &s : g_streams) s.first->done = s.first->enqueued;
}
// the hook gets the grid's blocks as the size
cudaError_t launch(const void *kernel, dim3 grid, cudaStream_t s) {
    std::string name = "launch:";
    {
        Lock lock(g_mutex);
        const auto it = kernels().find(kernel);
        name += it != kernels().end() ? it->second : "?";
    }
    const cudaError_t e = ask(name.c_str(), kernel, (size_t)grid.x * grid.y * grid.z, s);
    if (grid.x == 0 || grid.y == 0 || grid.z == 0) return result(cudaErrorInvalidConfiguration);
    if (e == cudaSuccess) enqueue(s);
    return e;
}

// the event, noting the use of one that went with a device reset (undefined in the real runtime)
Event *eventOf(cudaEvent_t e) {
    Event *x = reinterpret_cast<Event *>(e);
    if (x->life != g_life) g_staleUses++;
    return x;
}

#define ASK(...)                                        \
    do {                                                \
        const cudaError_t e_ = ask(__VA_ARGS__);        \
        if (e_ != cudaSuccess) return e_;               \
    } while (0)

std::atomic<int> g_newFails{0};  // how many of the next allocations by `new` fail

}  // namespace

void *operator new(size_t n) {
    if (g_newFails > 0 && g_newFails-- > 0) throw std::bad_alloc();
    void *p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

extern "C" {

// ------------------------------------------------------------- for the tests
void fake_fail_new(int times) { g_newFails = times; }
void fake_set_hook(Hook hook) {
    Lock lock(g_mutex);
    g_hook = hook;
}
// clears the library's device arrays, as no kernel does
void fake_clear_arrays(void) { std::memset(scratchArray(), 0, kArrayBytes); }
// device memory there is, and how much of it is allocated
void fake_set_capacity(size_t bytes) { g_capacity = bytes; }
size_t fake_allocated(void) {
    Lock lock(g_mutex);
    return g_bytes;
}
// operations enqueued on a stream (null: the legacy one) that nothing has waited for
unsigned long long fake_pending(void *stream) {
    Lock lock(g_mutex);
    Stream *s = of((cudaStream_t)stream);
    return s->enqueued - s->done;
}
// as a device reset: events made before are gone; and how often one was used all the same
void fake_reset_device(void) { g_life++; }
int fake_stale_uses(void) { return g_staleUses; }
void fake_set_capturing(void *stream, int on) { of((cudaStream_t)stream)->capturing = on != 0; }

// ------------------------------------------------------------- registration
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    kernels()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, void *stream) {
    Lock lock(g_mutex);
    g_configs.push_back({grid, block, shared, stream});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *shared, void *stream) {
    Lock lock(g_mutex);
    const Config c = g_configs.back();
    g_configs.pop_back();
    *grid = c.grid;
    *block = c.block;
    *shared = c.shared;
    *(void **)stream = c.stream;
    return cudaSuccess;
}

// ------------------------------------------------------------- devices, errors
cudaError_t cudaGetDeviceCount(int *n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) {
    static thread_local char text[32];
    std::snprintf(text, sizeof(text), "CUDA error %d", (int)e);
    return text;
}
cudaError_t cudaDeviceSynchronize(void) {
    ASK("cudaDeviceSynchronize");
    Lock lock(g_mutex);
    if (anyCapture()) return result(cudaErrorStreamCaptureUnsupported);
    finishAll();
    return cudaSuccess;
}

// ------------------------------------------------------------- memory
cudaError_t cudaMalloc(void **p, size_t n) {
    ASK("cudaMalloc", nullptr, n);
    Lock lock(g_mutex);
    if (g_bytes + n > g_capacity) return result(cudaErrorMemoryAllocation);
    void *block = std::calloc(1, n ? n : 1);
    if (!block) return result(cudaErrorMemoryAllocation);
    *p = block;
    g_blocks[block] = n;
    g_bytes += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    ASK("cudaFree", p);
    Lock lock(g_mutex);
    finishAll();
    const auto it = g_blocks.find(p);
    if (it == g_blocks.end()) return result(cudaErrorInvalidValue);
    g_bytes -= it->second;
    g_blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
    ASK("cudaMallocHost", nullptr, n);
    *p = std::calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *free, size_t *total) {
    Lock lock(g_mutex);
    *free = g_capacity - g_bytes;
    *total = g_capacity;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    *p = scratchArray();
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    ASK("cudaMemset", p, n);
    enqueue(nullptr);
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    ASK("cudaMemsetAsync", p, n, s);
    enqueue(s);
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind) {
    ASK("cudaMemcpy", d, n);
    enqueue(nullptr);  // from pageable memory it may return before the last bytes have arrived
    std::memcpy(d, s, n);
    if (kind == cudaMemcpyDeviceToHost) g_legacy.done = g_legacy.enqueued;
    return cudaSuccess;
}
// the hook gets the source
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    ASK("cudaMemcpyAsync", s, n, st);
    enqueue(st);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    for (size_t k = 0; k < h; k++) std::memcpy((char *)d + k * dp, (const char *)s + k * sp, w);
    return cudaSuccess;
}

// ------------------------------------------------------------- streams, events
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    ASK("cudaStreamCreateWithFlags");
    Lock lock(g_mutex);
    Stream *x = new Stream;
    g_streams[x] = true;
    *s = (cudaStream_t)x;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    ASK("cudaStreamDestroy", nullptr, 0, s);
    Lock lock(g_mutex);
    g_streams.erase(of(s));  // the object stays: events may point at it
    of(s)->done = of(s)->enqueued;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    ASK("cudaStreamSynchronize", nullptr, 0, s);
    Lock lock(g_mutex);
    if (of(s)->capturing) return result(cudaErrorStreamCaptureUnsupported);
    of(s)->done = of(s)->enqueued;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    ASK("cudaEventCreate");
    Event *x = new Event;
    x->life = g_life;
    *e = (cudaEvent_t)x;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }  // the object stays
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    ASK("cudaEventRecord", e, 0, s);
    Lock lock(g_mutex);
    Event *x = eventOf(e);
    x->stream = of(s);
    x->at = of(s)->enqueued;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    ASK("cudaEventSynchronize", e);
    Lock lock(g_mutex);
    Event *x = eventOf(e);
    if (x->stream && x->stream->done < x->at) x->stream->done = x->at;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    ASK("cudaEventQuery", e);
    Lock lock(g_mutex);
    const Event *x = eventOf(e);
    return x->stream && x->stream->done < x->at ? result(cudaErrorNotReady) : cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}

// ------------------------------------------------------------- kernels, modules
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t s) { return launch(f, grid, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) { return launch(f, c->gridDim, c->stream); }
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t s) { return launch(f, grid, s); }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaLibraryLoadData(cudaLibrary_t *l, const void *, cudaJitOption *, void **, unsigned, cudaLibraryOption *, void **, unsigned) {
    ASK("cudaLibraryLoadData");
    *l = (cudaLibrary_t) new char;
    return cudaSuccess;
}
cudaError_t cudaLibraryUnload(cudaLibrary_t l) {
    ASK("cudaLibraryUnload", l);
    return cudaSuccess;
}
cudaError_t cudaLibraryGetKernel(cudaKernel_t *k, cudaLibrary_t, const char *name) {
    Lock lock(g_mutex);
    *k = (cudaKernel_t) new char;
    kernels()[*k] = name;
    return cudaSuccess;
}

// ------------------------------------------------------------- graphs
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) {
    *g = (cudaGraph_t) new char;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) {
    *h = 1;
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, size_t, cudaGraphNodeParams *p) {
    static cudaGraph_t body;
    *n = (cudaGraphNode_t) new char;
    cudaGraphCreate(&body, 0);
    if (p->type == cudaGraphNodeTypeConditional) p->conditional.phGraph_out = &body;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
    ASK("cudaGraphInstantiate");
    *x = (cudaGraphExec_t) new char;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
    ASK("cudaGraphLaunch", nullptr, 0, s);
    enqueue(s);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                                          cudaStreamCaptureMode) {
    ASK("cudaStreamBeginCaptureToGraph", nullptr, 0, s);
    of(s)->capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
    ASK("cudaStreamEndCapture", nullptr, 0, s);
    of(s)->capturing = false;
    *g = (cudaGraph_t) new char;
    return cudaSuccess;
}

}  // extern "C"
