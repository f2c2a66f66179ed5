// fake_cuda.h: the functions of the CUDA runtime that the library calls.
#include "fake_cuda.h"

#include <cxxabi.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <set>

namespace fake {
std::vector<Launch> launches;
std::vector<Copy> copies;
uint64_t memory_limit = 1ull << 40;
bool reads_pageable = false;
}  // namespace fake

using Op = std::function<void()>;

struct CUstream_st {
    std::deque<Op> queue;
    uint64_t issued = 0, done = 0;
    bool capturing = false;
    std::vector<Op> captured;
};
struct CUevent_st {
    CUstream_st* stream = nullptr;
    uint64_t at = 0;
};
struct CUgraph_st {
    std::vector<Op> ops;
};
struct CUgraphExec_st {
    std::vector<Op> ops;
};

namespace {

std::recursive_mutex mu;
std::set<CUstream_st*> streams;
std::map<uintptr_t, size_t> device_mem, pinned;
std::map<uintptr_t, int> devices;  // of the allocations
uint64_t used = 0;
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
// (made on first use: objects register their kernels before main)
std::map<const void*, std::string>& names() {
    static auto* m = new std::map<const void*, std::string>;
    return *m;
}
std::map<const void*, size_t>& vars() {
    static auto* m = new std::map<const void*, size_t>;
    return *m;
}
std::map<std::pair<int, const void*>, int> max_smem;
std::vector<std::pair<std::string, std::function<Op(void**)>>> hooks;

struct Lock {
    std::lock_guard<std::recursive_mutex> g{mu};
};

cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}

CUstream_st* stream(cudaStream_t s) {
    static CUstream_st* legacy = new CUstream_st;
    if (!s || s == cudaStreamLegacy) return legacy;
    if (!streams.count(s)) {
        fprintf(stderr, "fake cuda: a stream that does not exist\n");
        abort();
    }
    return s;
}

void drain(CUstream_st* s, uint64_t upto) {
    while (s->done < upto && !s->queue.empty()) {
        Op op = std::move(s->queue.front());
        s->queue.pop_front();
        s->done++;
        op();
    }
}
void drain_all() {
    drain(stream(nullptr), ~0ull);
    for (CUstream_st* s : streams) drain(s, ~0ull);
}

void push(cudaStream_t st, Op op) {
    CUstream_st* s = stream(st);
    if (s->capturing) {
        s->captured.push_back(std::move(op));
        return;
    }
    s->queue.push_back(std::move(op));
    s->issued++;
}

size_t room(const std::map<uintptr_t, size_t>& m, const void* p) {  // bytes from p to its allocation's end
    const uintptr_t a = (uintptr_t)p;
    auto it = m.upper_bound(a);
    if (it == m.begin()) return 0;
    --it;
    return a < it->first + it->second ? it->first + it->second - a : 0;
}

void in_device(const void* p, size_t n, const char* what) {
    if (n && room(device_mem, p) < n) {
        fprintf(stderr, "fake cuda: %s of %zu bytes outside device memory\n", what, n);
        abort();
    }
}

void check_copy(const void* dst, const void* src, size_t n, cudaMemcpyKind k) {
    if (k == cudaMemcpyHostToDevice || k == cudaMemcpyDeviceToDevice) in_device(dst, n, "copy to");
    if (k == cudaMemcpyDeviceToHost || k == cudaMemcpyDeviceToDevice) in_device(src, n, "copy from");
}

}  // namespace

namespace fake {
void on_launch(const char* kernel, std::function<std::function<void()>(void**)> f) {
    Lock l;
    hooks.emplace_back(kernel, std::move(f));
}
bool launched(const char* kernel) {
    Lock l;
    for (const Launch& x : launches)
        if (x.kernel.find(kernel) != std::string::npos) return true;
    return false;
}
int device_of(const void* p) {
    Lock l;
    if (!room(device_mem, p)) return -1;
    return std::prev(devices.upper_bound((uintptr_t)p))->second;
}
}  // namespace fake

extern "C" {

// ------------------------------------------------- what compiled code calls
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    int st = 0;
    char* d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
    names()[host] = d ? d : name;
    free(d);
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) { vars()[host] = size; }

static thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} call;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* st) {
    call = {grid, block, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
    *grid = call.grid;
    *block = call.block;
    *smem = call.smem;
    *static_cast<cudaStream_t*>(st) = call.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t) const_cast<void*>(f);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t st) {
    Lock l;
    if (!grid.x || !grid.y || !grid.z || !block.x) return ret(cudaErrorInvalidConfiguration);
    if (smem > 48 * 1024 && (size_t)max_smem[{current, f}] < smem) return ret(cudaErrorInvalidValue);
    const std::string& name = names()[f];
    fake::launches.push_back({name, current, st, smem});
    Op op = [] {};
    for (auto& h : hooks)
        if (name.find(h.first) != std::string::npos) op = h.second(args);
    push(st, op);
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t st) {
    return cudaLaunchKernel((const void*)k, grid, block, args, smem, st);
}

// --------------------------------------------------------------- devices
cudaError_t cudaSetDevice(int d) {
    current = d;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = current;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? fake::reads_pageable : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
    *lo = 0;
    *hi = -1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake cuda error"; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
    Lock l;
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) max_smem[{current, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}

// ---------------------------------------------------------------- memory
cudaError_t cudaMemGetInfo(size_t* free_, size_t* total) {
    Lock l;
    *free_ = fake::memory_limit > used ? fake::memory_limit - used : 0;
    *total = fake::memory_limit;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    Lock l;
    if (used + n > fake::memory_limit) return ret(cudaErrorMemoryAllocation);
    void* a = mmap(nullptr, n + 4096, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (a == MAP_FAILED) return ret(cudaErrorMemoryAllocation);
    if (n <= (64u << 20)) memset(a, fake::kPoison, n);
    device_mem[(uintptr_t)a] = n;
    devices[(uintptr_t)a] = current;
    used += n;
    *p = a;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    Lock l;
    if (!p) return cudaSuccess;
    drain_all();
    auto it = device_mem.find((uintptr_t)p);
    if (it == device_mem.end()) return ret(cudaErrorInvalidValue);
    used -= it->second;
    munmap(p, it->second + 4096);
    devices.erase(it->first);
    device_mem.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    Lock l;
    *p = malloc(n ? n : 1);
    pinned[(uintptr_t)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    Lock l;
    drain_all();
    pinned.erase((uintptr_t)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
    Lock l;
    *a = {};
    if (room(device_mem, p)) a->type = cudaMemoryTypeDevice;
    else if (room(pinned, p)) a->type = cudaMemoryTypeHost;
    if (a->type != cudaMemoryTypeUnregistered) a->devicePointer = const_cast<void*>(p);
    if (a->type == cudaMemoryTypeHost) a->hostPointer = const_cast<void*>(p);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
    return cudaMalloc(p, vars()[sym]);
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind k) {
    Lock l;
    check_copy(dst, src, n, k);
    fake::copies.push_back({src, dst, n, k});
    drain(stream(nullptr), ~0ull);
    memcpy(dst, src, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    Lock l;
    check_copy(dst, src, n, k);
    fake::copies.push_back({src, dst, n, k});
    if (k == cudaMemcpyHostToDevice && !room(pinned, src)) {  // pageable memory is staged at the call
        auto staged = std::make_shared<std::vector<uint8_t>>((const uint8_t*)src, (const uint8_t*)src + n);
        push(st, [dst, staged] { memcpy(dst, staged->data(), staged->size()); });
    } else {
        push(st, [dst, src, n] { memcpy(dst, src, n); });
    }
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
    Lock l;
    in_device(p, n, "clear");
    drain(stream(nullptr), ~0ull);
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    Lock l;
    in_device(p, n, "clear");
    push(st, [p, v, n] { memset(p, v, n); });
    return cudaSuccess;
}

// --------------------------------------------------- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    Lock l;
    *s = new CUstream_st;
    streams.insert(*s);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    Lock l;
    drain(stream(s), ~0ull);
    streams.erase(s);  // (not freed: events may still name it)
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    Lock l;
    if (stream(s)->capturing) return ret(cudaErrorStreamCaptureUnsupported);
    drain(stream(s), ~0ull);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* st) {
    Lock l;
    *st = stream(s)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode* m) {
    static thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
    std::swap(*m, mode);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode) {
    Lock l;
    stream(s)->capturing = true;
    stream(s)->captured.clear();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    Lock l;
    stream(s)->capturing = false;
    *g = new CUgraph_st{stream(s)->captured};
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
    *x = new CUgraphExec_st{g->ops};
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t st) {
    Lock l;
    for (const Op& op : x->ops) push(st, op);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete g;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    delete x;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = new CUevent_st;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }  // (not freed: queued waits may name it)
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    Lock l;
    e->stream = stream(st);
    e->at = e->stream->issued;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
    Lock l;
    CUstream_st* s = e->stream;
    const uint64_t at = e->at;
    if (s) push(st, [s, at] { drain(s, at); });
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    Lock l;
    if (e->stream) drain(e->stream, e->at);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1;
    return cudaSuccess;
}

}  // extern "C"
