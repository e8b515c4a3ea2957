// A CUDA runtime for host-logic tests on machines without a GPU, preloaded in front of libcudart: device memory
// is host memory, kernels are counted and their pointer arguments looked at but never run, and copies from
// pinned memory happen only when their stream or an event behind them is waited for, as the real ones may.
// Allocations, the library's host ones too, fail where the test asks for it. fake_* are the test's controls.
#include <cuda_runtime.h>
#include <cxxabi.h>
#include <dlfcn.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <utility>
#include <vector>

namespace {
std::mutex mu;
std::map<char*, size_t> dev, pinned;  // live allocations
long mallocs = 0, fail_at = -1, launches = 0;
size_t bytes_now = 0;
thread_local cudaError_t last = cudaSuccess;
std::string nulls, names;  // "kernel#argument;" of every null pointer passed, "kernel;" of every launch
std::string watch;  // kernel whose parameter `watch_arg` is kept
int watch_arg = 0;
unsigned char watched[64];
size_t watch_bytes = 0;
std::string poke;  // kernel that "writes" `poke_data` to its pointer parameter `poke_arg`
int poke_arg = 0;
unsigned char poke_data[64];
size_t poke_bytes = 0;

struct Copy {
    void* dst;
    const void* src;
    size_t n;
};
typedef std::pair<cudaStream_t, size_t> Queue;  // the per-thread handle names another queue in every thread
std::map<Queue, std::vector<Copy>> pending;
struct Event {
    bool recorded = false;
    Queue q;
};
Queue queue_of(cudaStream_t s) {
    return Queue(s, s == cudaStreamPerThread ? std::hash<std::thread::id>()(std::this_thread::get_id()) : 0);
}
void drain(const Queue& q) {
    for (const Copy& c : pending[q]) memcpy(c.dst, c.src, c.n);
    pending.erase(q);
}
cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
bool in(const std::map<char*, size_t>& m, const void* p) {
    auto it = m.upper_bound((char*)p);
    if (it == m.begin()) return false;
    --it;
    return (char*)p < it->first + it->second;
}
// the kernel's parameter types from its host function's symbol
std::string demangled(const void* f) {
    Dl_info info;
    if (!dladdr(f, &info) || !info.dli_sname) return "?";
    int st = 0;
    char* d = abi::__cxa_demangle(info.dli_sname, nullptr, nullptr, &st);
    std::string s = st == 0 ? d : info.dli_sname;
    free(d);
    return s;
}
cudaError_t launch(const void* f, void** args) {
    std::lock_guard<std::mutex> l(mu);
    ++launches;
    const std::string sig = demangled(f);
    const size_t open = sig.rfind('('), at = sig.find("gpsb::");
    std::string name = sig.substr(at == std::string::npos ? 0 : at, open == std::string::npos ? open : open - (at == std::string::npos ? 0 : at));
    names += name + ";";
    const std::string base = name.substr(0, name.find('<'));  // any instance of a template
    if (poke_bytes && (name == poke || base == poke)) memcpy(*(void**)args[poke_arg], poke_data, poke_bytes);
    if (watch_bytes && (name == watch || base == watch)) memcpy(watched, args[watch_arg], watch_bytes);
    if (open == std::string::npos) return cudaSuccess;
    int arg = 0, depth = 0;
    std::string type;
    for (size_t k = open + 1; k < sig.size(); ++k) {
        const char c = sig[k];
        depth += c == '<' ? 1 : c == '>' ? -1 : 0;
        if ((c == ',' && depth == 0) || c == ')') {
            if (!type.empty() && type.back() == '*' && *(void**)args[arg] == nullptr) nulls += name + "#" + std::to_string(arg) + ";";
            type.clear();
            ++arg;
        } else {
            type += c;
        }
    }
    return cudaSuccess;
}
int encode_tensor_map() { return 0; }
std::atomic<long> fail_new{-1};  // operator new calls of the renderer library until one fails
}  // namespace

void* operator new(size_t n) {
    if (fail_new.load() >= 0) {
        Dl_info info;
        if (dladdr(__builtin_return_address(0), &info) && strstr(info.dli_fname, "libgpsb200") && fail_new.fetch_sub(1) == 0)
            throw std::bad_alloc();
    }
    void* p = malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

extern "C" {
// ---- controls
void fake_fail_new(long n) { fail_new = n; }  // the library's n-th `new` from now on throws, once; < 0: none
void fake_fail_malloc(long n) { fail_at = n < 0 ? -1 : mallocs + n; }  // the n-th allocation from now on fails, once
long fake_mallocs() { return mallocs; }
long fake_launches() { return launches; }
size_t fake_live_bytes() { return bytes_now; }
size_t fake_pending() {
    std::lock_guard<std::mutex> l(mu);
    size_t n = 0;
    for (auto& q : pending) n += q.second.size();
    return n;
}
const char* fake_nulls() { return nulls.c_str(); }
const char* fake_kernels() { return names.c_str(); }
void fake_watch(const char* kernel, int arg, size_t bytes) { watch = kernel, watch_arg = arg, watch_bytes = bytes; }
void fake_poke(const char* kernel, int arg, const void* data, size_t bytes) {
    poke = kernel, poke_arg = arg, poke_bytes = bytes;
    memcpy(poke_data, data, bytes);
}
const void* fake_watched() { return watched; }
void fake_clear() { nulls.clear(), names.clear(), launches = 0; }

// ---- the runtime
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    return *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 148, cudaSuccess;  // else: multiprocessors
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = (size_t)8 << 30, cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    if (q) *q = cudaDriverEntryPointSuccess;
    return *f = (void*)encode_tensor_map, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = (void*)1024, cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> l(mu);
    *p = nullptr;
    if (++mallocs == fail_at) return fail_at = -1, set(cudaErrorMemoryAllocation);
    *p = calloc(1, n ? n : 1);
    dev[(char*)*p] = n;
    bytes_now += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> l(mu);
    if (!p) return cudaSuccess;
    bytes_now -= dev[(char*)p];
    dev.erase((char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    std::lock_guard<std::mutex> l(mu);
    *p = calloc(1, n);
    pinned[(char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> l(mu);
    pinned.erase((char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> l(mu);
    memset(a, 0, sizeof *a);
    a->type = in(dev, p) ? cudaMemoryTypeDevice : in(pinned, p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    const Queue q = queue_of(st);
    if (in(pinned, s)) {
        pending[q].push_back({d, s, n});
    } else {
        drain(q);
        memcpy(d, s, n);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (!p && n) return set(cudaErrorInvalidValue);
    if (!in(dev, p)) return cudaSuccess;
    return memset(p, v, n), cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)malloc(8), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::mutex> l(mu);
    drain(queue_of(s));
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { return *c = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)malloc(8), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return *e = (cudaGraphExec_t)malloc(8), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return free(e), cudaSuccess; }

cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t) new Event, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete (Event*)e, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::mutex> l(mu);
    ((Event*)e)->recorded = true;
    ((Event*)e)->q = queue_of(s);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::mutex> l(mu);
    if (((Event*)e)->recorded) drain(((Event*)e)->q);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { return *t = 0.0f, cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { return memset(a, 0, sizeof *a), cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t, cudaStream_t) {
    if (!grid.x || !grid.y || !grid.z || !block.x || !block.y || !block.z) return set(cudaErrorInvalidConfiguration);
    return launch(f, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return cudaLaunchKernel(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}
}
