// A CUDA runtime without a device, loaded in place of libcudart for tests of the library's host
// path: memory is host memory, copies and clears happen at once, kernels do not run.  It has two
// devices, keeps each kernel's shared-memory attribute per device, refuses a launch beyond it as
// the runtime does, and logs launches, copies and host allocations.
#include <cuda_runtime_api.h>

#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {
std::mutex mu;
std::map<const void*, std::string> names;
std::map<std::pair<int, const void*>, size_t> smem;
std::map<const char*, size_t> pinned;
std::vector<std::string> log_;
std::string pause_at;  // cudaFuncSetAttribute of a kernel with this in its name waits for fake_resume
bool paused = false, resumed = false;
std::condition_variable cv;
thread_local int device = 0;

void note(const std::string& line) {
    std::lock_guard<std::mutex> g(mu);
    log_.push_back(line);
}
// early: with the attribute that lets a kernel start before its predecessor ends
cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t dyn, bool early) {
    std::string name;
    size_t lim;
    {
        std::lock_guard<std::mutex> g(mu);
        name = names[f];
        auto it = smem.find({device, f});
        lim = it == smem.end() ? 48 * 1024 : it->second;
    }
    if (dyn > 48 * 1024 && dyn > lim) return cudaErrorInvalidValue;
    char line[160];
    std::snprintf(line, sizeof line, "launch %u %u %u %zu ", grid.x * grid.y, block.x, (unsigned)device, dyn);
    note(line + name + (early ? " early" : ""));
    return cudaSuccess;
}
cudaError_t give(void** p, size_t n) {
    *p = std::calloc(n + 256, 1);
    return cudaSuccess;
}
struct Call { dim3 grid, block; size_t dyn; cudaStream_t st; };
thread_local std::vector<Call> calls;
}  // namespace

extern "C" {
// ---- for the test
int fake_log(char* out, int room) {  // takes the log: lines separated by newlines
    std::lock_guard<std::mutex> g(mu);
    std::string s;
    for (auto& l : log_) s += l + "\n";
    log_.clear();
    std::snprintf(out, room, "%s", s.c_str());
    return (int)s.size();
}
void fake_pause(const char* name) { std::lock_guard<std::mutex> g(mu); pause_at = name; paused = resumed = false; }
int fake_paused() { std::lock_guard<std::mutex> g(mu); return paused; }
void fake_resume() { { std::lock_guard<std::mutex> g(mu); resumed = true; pause_at.clear(); } cv.notify_all(); }

// ---- modules and launches
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    std::lock_guard<std::mutex> g(mu);
    names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t dyn, cudaStream_t st) {
    calls.push_back({grid, block, dyn, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* dyn, void* st) {
    const Call c = calls.back();
    calls.pop_back();
    *grid = c.grid; *block = c.block; *dyn = c.dyn; *static_cast<cudaStream_t*>(st) = c.st;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t dyn, cudaStream_t) {
    return launch((const void*)k, grid, block, dyn, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    bool early = false;
    for (unsigned q = 0; q < c->numAttrs; ++q)
        early = early || (c->attrs[q].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                          c->attrs[q].val.programmaticStreamSerializationAllowed);
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, early);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v > 227 * 1024) return cudaErrorInvalidValue;
    std::unique_lock<std::mutex> g(mu);
    smem[{device, f}] = v;
    if (!pause_at.empty() && names[f].find(pause_at) != std::string::npos) {
        pause_at.clear();
        paused = true;
        cv.wait_for(g, std::chrono::milliseconds(500), [] { return resumed; });
    }
    return cudaSuccess;
}

// ---- devices
cudaError_t cudaSetDevice(int d) { device = d; return d >= 0 && d < 2 ? cudaSuccess : cudaErrorInvalidDevice; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 3 : 1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : "error"; }

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { return give(p, n); }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
    give(p, n);
    note("host_alloc " + std::to_string(n));
    std::lock_guard<std::mutex> g(mu);
    pinned[(const char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
    note("host_free");
    { std::lock_guard<std::mutex> g(mu); pinned.erase((const char*)p); }
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::memset(a, 0, sizeof *a);
    std::lock_guard<std::mutex> g(mu);
    auto it = pinned.upper_bound((const char*)p);
    a->type = cudaMemoryTypeUnregistered;
    if (it != pinned.begin() && (const char*)p < (--it)->first + it->second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    char line[128];
    std::snprintf(line, sizeof line, "copy %d %zu %zu %zu", (int)k, n, (size_t)d, (size_t)s);
    note(line);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return give(p, 1 << 16); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return give(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }

// ---- streams, events and graphs (a captured sequence has run while it was captured)
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)8; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { note("capture"); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)8; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)8; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1.f; return cudaSuccess; }
}
