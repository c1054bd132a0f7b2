// A CUDA runtime for tests of the library's host code on a machine without a GPU: linked with the library's objects in
// place of the real one. Device memory is host memory, copies and memsets are done at once, kernels do nothing but what a
// test's hook asks for. It keeps counts of every call, of live allocations, streams and events, and of the work that a
// stream has been given and nobody has waited for; a test may have the n-th call of a function fail.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <thread>

namespace {
struct Stream {
    long work = 0;               // launches and copies not waited for
    std::set<Stream*> after;     // streams whose work this one's waits cover
};
struct Event {
    Stream* of = nullptr;
};
std::map<std::string, long> calls;
std::map<std::string, std::pair<long, cudaError_t>> failing;  // function -> (calls still to go, error)
std::map<void*, size_t> device, pinned;
std::map<const void*, std::string> kernels;
std::map<const void*, std::pair<void*, size_t>> vars;
std::set<Stream*> streams;
std::set<Event*> events;
Stream legacy;
std::string hook_kernel;
int hook_arg = 0, hook_value = 0, sync_ms = 0, major_version = 10;
dim3 push_grid, push_block;
size_t push_shmem = 0;
cudaStream_t push_stream = nullptr;
cudaError_t last = cudaSuccess;

Stream* of(cudaStream_t s) {
    return reinterpret_cast<uintptr_t>(s) < 16 ? &legacy : reinterpret_cast<Stream*>(s);
}
cudaError_t enter(const char* name) {
    ++calls[name];
    auto f = failing.find(name);
    if (f != failing.end() && --f->second.first == 0) {
        last = f->second.second;
        failing.erase(f);
        return last;
    }
    return cudaSuccess;
}
void waited(Stream* s, std::set<Stream*>& seen) {
    if (!seen.insert(s).second) return;
    s->work = 0;
    for (Stream* d : s->after) waited(d, seen);
    s->after.clear();
}
}  // namespace

#define ENTER(name)                                        \
    do {                                                   \
        const cudaError_t e_ = enter(name);                \
        if (e_ != cudaSuccess) return e_;                  \
    } while (0)

extern "C" {
// ---- what a test asks for
void fake_reset() {
    calls.clear();
    failing.clear();
    hook_kernel.clear();
    sync_ms = 0;
    major_version = 10;
    last = cudaSuccess;
}
void fake_fail(const char* name, long nth, int error) { failing[name] = {nth, cudaError_t(error)}; }
// every launch of a kernel whose name contains `name` writes `value` through its pointer argument `arg`
void fake_hook(const char* name, int arg, int value) {
    hook_kernel = name;
    hook_arg = arg;
    hook_value = value;
}
void fake_sync_ms(int ms) { sync_ms = ms; }  // how long a wait for a stream takes
void fake_major(int v) { major_version = v; }
long fake_calls(const char* name) { return calls.count(name) ? calls[name] : 0; }
long fake_launches(const char* part) {
    long n = 0;
    for (auto& c : calls)
        if (c.first.rfind("launch ", 0) == 0 && c.first.find(part) != std::string::npos) n += c.second;
    return n;
}
long fake_device_bytes() {
    size_t n = 0;
    for (auto& p : device) n += p.second;
    return long(n);
}
long fake_pinned() { return long(pinned.size()); }
long fake_streams() { return long(streams.size()); }
long fake_events() { return long(events.size()); }
long fake_pending_own() {  // on the library's own streams
    long n = 0;
    for (Stream* s : streams) n += s->work;
    return n;
}
long fake_pending() { return fake_pending_own() + legacy.work; }

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) {
    static void* handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) {
    vars[host] = {calloc(1, size), size};
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shmem, struct CUstream_st* stream) {
    push_grid = grid;
    push_block = block;
    push_shmem = shmem;
    push_stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shmem, void* stream) {
    *grid = push_grid;
    *block = push_block;
    *shmem = push_shmem;
    *static_cast<cudaStream_t*>(stream) = push_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t, cudaStream_t s) {
    ENTER("cudaLaunchKernel");
    if (grid.x == 0 || block.x == 0) return last = cudaErrorInvalidConfiguration;
    const std::string& name = kernels[f];
    ++calls["launch " + name];
    ++of(s)->work;
    if (!hook_kernel.empty() && name.find(hook_kernel) != std::string::npos)
        **static_cast<int**>(args[hook_arg]) = hook_value;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
    ENTER("cudaFuncSetAttribute");
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}

// ---- the device
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) {
    ENTER("cudaSetDevice");
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    ENTER("cudaGetDeviceProperties");
    std::memset(p, 0, sizeof(*p));
    p->major = major_version;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    ENTER("cudaDeviceGetAttribute");
    *v = a == cudaDevAttrComputeCapabilityMajor ? major_version : a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
    *least = 0;
    *greatest = -5;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the test's making"; }
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
    *p = vars[symbol].first;
    return cudaSuccess;
}
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    ENTER("cudaGetDriverEntryPoint");
    *p = reinterpret_cast<void*>(encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
    ENTER("cudaMalloc");
    *p = n ? calloc(1, n) : nullptr;
    if (n) device[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    ++calls["cudaFree"];
    if (p && !device.erase(p)) return last = cudaErrorInvalidValue;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    ENTER("cudaHostAlloc");
    *p = calloc(1, n);
    pinned[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    ENTER("cudaMallocHost");
    *p = calloc(1, n);
    pinned[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    if (p && !pinned.erase(p)) return last = cudaErrorInvalidValue;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
    if (!h) return last = cudaErrorInvalidValue;
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    ENTER("cudaMemcpyAsync");
    std::memcpy(d, s, n);
    ++of(st)->work;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    ENTER("cudaMemcpy");
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    ENTER("cudaMemsetAsync");
    std::memset(d, v, n);
    ++of(st)->work;
    return cudaSuccess;
}

// ---- streams and events
static cudaError_t new_stream(cudaStream_t* s) {
    ENTER("cudaStreamCreate");
    Stream* q = new Stream;
    streams.insert(q);
    *s = reinterpret_cast<cudaStream_t>(q);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return new_stream(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return new_stream(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    Stream* q = of(s);
    for (Stream* o : streams) o->after.erase(q);
    legacy.after.erase(q);
    for (Event* e : events)
        if (e->of == q) e->of = nullptr;
    streams.erase(q);
    delete q;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::set<Stream*> seen;
    waited(of(s), seen);
    std::this_thread::sleep_for(std::chrono::milliseconds(sync_ms));
    ENTER("cudaStreamSynchronize");
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    ENTER("cudaStreamWaitEvent");
    Event* ev = reinterpret_cast<Event*>(e);
    if (ev->of && ev->of != of(s)) of(s)->after.insert(ev->of);
    return cudaSuccess;
}
static cudaError_t new_event(cudaEvent_t* e) {
    ENTER("cudaEventCreate");
    Event* ev = new Event;
    events.insert(ev);
    *e = reinterpret_cast<cudaEvent_t>(ev);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return new_event(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return new_event(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    events.erase(reinterpret_cast<Event*>(e));
    delete reinterpret_cast<Event*>(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    ENTER("cudaEventRecord");
    reinterpret_cast<Event*>(e)->of = of(s);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::set<Stream*> seen;
    if (reinterpret_cast<Event*>(e)->of) waited(reinterpret_cast<Event*>(e)->of, seen);
    ENTER("cudaEventSynchronize");
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}

// ---- graphs: what was captured has been done already; a launch is some work on its stream
static int graph_object;
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    std::set<Stream*> seen;
    waited(of(s), seen);
    *g = reinterpret_cast<cudaGraph_t>(&graph_object);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    ENTER("cudaGraphInstantiate");
    *x = reinterpret_cast<cudaGraphExec_t>(&graph_object);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
    ENTER("cudaGraphLaunch");
    ++of(s)->work;
    return cudaSuccess;
}
}  // extern "C"
