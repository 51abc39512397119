// A CUDA runtime without a GPU, for the host code of the library: two devices whose memory is host
// memory, and streams that run nothing until something waits for them, i.e. as late as the runtime's
// documentation allows. An asynchronous copy reads its source when it runs; a blocking copy to the
// device has read its source on return but reaches the device later, in the legacy stream; a stream
// made with cudaStreamNonBlocking is not ordered against the legacy stream. Kernels do nothing. What a
// program must not rely on is recorded as a violation:
//   * a copy whose source changed (or was freed) between the call and the copy;
//   * a kernel launched into a non-blocking stream while legacy-stream work is pending;
//   * a stream, pool or launch used with another device current than its own.
// fake_* below are the test's handles.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <vector>

#define FAKE extern "C" __attribute__((visibility("default")))

namespace {

struct Op {
    uint64_t seq;
    std::function<void()> run;
};
struct Stream {
    int dev = 0;
    bool blocking = false;
    bool capturing = false;
    std::deque<Op> q;
};
struct Event {
    Stream* s = nullptr;
    uint64_t seq = 0;
};
struct Pool {
    int dev = 0;
    uint64_t keep = 0, reserved = 0, used = 0;
};
struct Block {
    size_t bytes;
    Pool* pool;
};

std::recursive_mutex mx;
uint64_t seq_now = 0, host_news = 0;
uint64_t capacity = ~0ull, in_use = 0;  // device memory (both devices together)
std::string violations;
std::map<void*, Block> blocks;
std::set<Stream*> live;
Stream legacy[2];
uint32_t status_script = 0;  // statuses the next small-result read-backs report, one a call
int scripted_reads = 0;
thread_local int cur = 0;
thread_local cudaError_t last = cudaSuccess;

// Held by every call of the runtime; what the fake itself allocates is not counted (host_news).
thread_local int inside = 0;
struct Lock {
    Lock() {
        mx.lock();
        ++inside;
    }
    ~Lock() {
        --inside;
        mx.unlock();
    }
};

void violation(const std::string& s) { violations += s + "\n"; }
cudaError_t err(cudaError_t e) {
    if (e) last = e;
    return e;
}
Stream* get(cudaStream_t st) {
    if (!st) {
        legacy[0].dev = 0;
        legacy[1].dev = 1;
        legacy[0].blocking = legacy[1].blocking = true;
        return &legacy[cur];
    }
    Stream* s = reinterpret_cast<Stream*>(st);
    if (!live.count(s)) violation("use of a destroyed stream");
    return s;
}
void drain(Stream* s, uint64_t upto) {
    while (!s->q.empty() && s->q.front().seq <= upto) {
        Op op = std::move(s->q.front());
        s->q.pop_front();
        op.run();
    }
}
void put(Stream* s, std::function<void()> f) {
    if (!s->capturing) s->q.push_back(Op{++seq_now, std::move(f)});
}
uint64_t sum(const void* p, size_t n) {
    uint64_t h = 1469598103934665603ull;
    for (size_t i = 0; i < n; ++i) h = (h ^ static_cast<const unsigned char*>(p)[i]) * 1099511628211ull;
    return h;
}
bool on_device(const void* p) {
    auto it = blocks.upper_bound(const_cast<void*>(p));
    if (it == blocks.begin()) return false;
    --it;
    return static_cast<const char*>(p) < static_cast<const char*>(it->first) + it->second.bytes;
}
cudaError_t take(void** out, size_t bytes, Pool* pool) {
    if (pool) {
        const uint64_t idle = pool->reserved - pool->used;
        const uint64_t more = bytes > idle ? bytes - idle : 0;
        if (in_use + more > capacity) return cudaErrorMemoryAllocation;
        in_use += more;
        pool->reserved += more;
        pool->used += bytes;
    } else {
        if (in_use + bytes > capacity) return cudaErrorMemoryAllocation;
        in_use += bytes;
    }
    *out = std::calloc(1, bytes + 16);
    blocks[*out] = Block{bytes, pool};
    return cudaSuccess;
}
void give(void* p) {
    auto it = blocks.find(p);
    if (it == blocks.end()) return violation("free of unknown device memory");
    if (Pool* pool = it->second.pool) pool->used -= it->second.bytes;
    else in_use -= it->second.bytes;
    blocks.erase(it);
    std::free(p);
}
void trim(Pool* p, uint64_t keep) {
    const uint64_t to = p->used > keep ? p->used : (p->reserved < keep ? p->reserved : keep);
    in_use -= p->reserved - to;
    p->reserved = to;
}
std::set<Pool*> pools;
void trim_all() {  // a synchronisation gives memory above the release threshold back
    for (Pool* p : pools) trim(p, p->keep);
}
cudaError_t launch(cudaStream_t st) {
    Lock lk;
    Stream* s = get(st);
    if (s->dev != cur) {
        violation("launch into a stream of another device");
        return err(cudaErrorInvalidResourceHandle);
    }
    if (!s->blocking && !s->capturing && !legacy[s->dev].q.empty())
        violation("kernel launched into a non-blocking stream while legacy-stream work is pending");
    put(s, [] {});
    return cudaSuccess;
}

}  // namespace

FAKE const char* fake_violations() { return violations.c_str(); }
FAKE void fake_reset() {
    Lock lk;
    violations.clear();
    host_news = 0;
    capacity = ~0ull;
    scripted_reads = 0;
}
FAKE uint64_t fake_in_use() { return in_use; }
FAKE void fake_set_free(uint64_t bytes) { capacity = bytes == ~0ull ? bytes : in_use + bytes; }
FAKE uint64_t fake_host_news() { return host_news; }
FAKE void fake_set_device(int d) { cur = d; }
// the next `reads` copies back report `status` in the first whole-test result
FAKE void fake_script_status(uint32_t status, int reads) {
    status_script = status;
    scripted_reads = reads;
}

// host allocations by the library's C++ code
void* operator new(size_t n) {
    if (!inside) ++host_news;
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }

// ---- what nvcc's host stubs call ---------------------------------------------------------------

static thread_local cudaStream_t pushed;
FAKE unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t st) {
    pushed = st;
    return 0;
}
FAKE cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sh, void* st) {
    *g = *b = dim3(1);
    *sh = 0;
    *static_cast<cudaStream_t*>(st) = pushed;
    return cudaSuccess;
}
FAKE void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
FAKE void __cudaRegisterFatBinaryEnd(void**) {}
FAKE void __cudaUnregisterFatBinary(void**) {}
FAKE void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
FAKE void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

FAKE cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t st) { return launch(st); }
FAKE cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) { return launch(c->stream); }
FAKE cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int) { return cudaSuccess; }

// ---- devices -----------------------------------------------------------------------------------

FAKE cudaError_t cudaGetDeviceCount(int* n) {
    *n = 2;
    return cudaSuccess;
}
FAKE cudaError_t cudaGetDevice(int* d) {
    *d = cur;
    return cudaSuccess;
}
FAKE cudaError_t cudaSetDevice(int d) {
    cur = d;
    return cudaSuccess;
}
FAKE cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
FAKE cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    std::strcpy(p->name, "fake");
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
FAKE const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
FAKE cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
FAKE cudaError_t cudaDeviceSynchronize() {
    Lock lk;
    drain(&legacy[cur], ~0ull);
    for (Stream* s : live)
        if (s->dev == cur) drain(s, ~0ull);
    trim_all();
    return cudaSuccess;
}

// ---- streams and events ------------------------------------------------------------------------

FAKE cudaError_t cudaStreamCreateWithFlags(cudaStream_t* out, unsigned flags) {
    Lock lk;
    Stream* s = new Stream;
    s->dev = cur;
    s->blocking = !(flags & cudaStreamNonBlocking);
    live.insert(s);
    *out = reinterpret_cast<cudaStream_t>(s);
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamDestroy(cudaStream_t st) {
    Lock lk;
    Stream* s = get(st);
    drain(s, ~0ull);
    live.erase(s);
    return cudaSuccess;  // the object itself is kept: events may name it
}
FAKE cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    Lock lk;
    drain(get(st), ~0ull);
    trim_all();
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned) {
    Lock lk;
    const Event e = *reinterpret_cast<Event*>(ev);
    if (e.s) put(get(st), [e] { drain(e.s, e.seq); });
    return cudaSuccess;
}
FAKE cudaError_t cudaEventCreate(cudaEvent_t* out) {
    Lock lk;
    *out = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
FAKE cudaError_t cudaEventCreateWithFlags(cudaEvent_t* out, unsigned) { return cudaEventCreate(out); }
FAKE cudaError_t cudaEventDestroy(cudaEvent_t ev) {
    delete reinterpret_cast<Event*>(ev);
    return cudaSuccess;
}
FAKE cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st) {
    Lock lk;
    Stream* s = get(st);
    put(s, [] {});
    *reinterpret_cast<Event*>(ev) = Event{s, seq_now};
    return cudaSuccess;
}
FAKE cudaError_t cudaEventSynchronize(cudaEvent_t ev) {
    Lock lk;
    const Event e = *reinterpret_cast<Event*>(ev);
    if (e.s) drain(e.s, e.seq);
    return cudaSuccess;
}
FAKE cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamBeginCapture(cudaStream_t st, enum cudaStreamCaptureMode) {
    get(st)->capturing = true;
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g) {
    get(st)->capturing = false;
    *g = nullptr;
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamIsCapturing(cudaStream_t st, enum cudaStreamCaptureStatus* out) {
    *out = get(st)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
FAKE cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    static int dummy;
    *e = reinterpret_cast<cudaGraphExec_t>(&dummy);
    return cudaSuccess;
}
FAKE cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) { return launch(st); }

// ---- memory ------------------------------------------------------------------------------------

FAKE cudaError_t cudaMalloc(void** out, size_t bytes) {
    Lock lk;
    return err(take(out, bytes, nullptr));
}
FAKE cudaError_t cudaFree(void* p) {
    Lock lk;
    cudaDeviceSynchronize();
    if (p) give(p);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemPoolCreate(cudaMemPool_t* out, const cudaMemPoolProps* props) {
    Lock lk;
    Pool* p = new Pool;
    p->dev = props->location.id;
    pools.insert(p);
    *out = reinterpret_cast<cudaMemPool_t>(p);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t pool, enum cudaMemPoolAttr a, void* v) {
    if (a == cudaMemPoolAttrReleaseThreshold) reinterpret_cast<Pool*>(pool)->keep = *static_cast<uint64_t*>(v);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) {
    Lock lk;
    trim(reinterpret_cast<Pool*>(pool), keep);
    return cudaSuccess;
}
FAKE cudaError_t cudaMallocFromPoolAsync(void** out, size_t bytes, cudaMemPool_t pool, cudaStream_t st) {
    Lock lk;
    Pool* p = reinterpret_cast<Pool*>(pool);
    if (p->dev != get(st)->dev) violation("pool memory of one device taken in a stream of another");
    return err(take(out, bytes, p));
}
FAKE cudaError_t cudaFreeAsync(void* p, cudaStream_t st) {
    Lock lk;
    put(get(st), [p] { give(p); });
    return cudaSuccess;
}
FAKE cudaError_t cudaGetSymbolAddress(void** out, const void*) {
    static unsigned char symbol[1 << 20];
    *out = symbol;
    return cudaSuccess;
}
FAKE cudaError_t cudaMemset(void* p, int v, size_t n) {
    Lock lk;
    put(get(nullptr), [=] { std::memset(p, v, n); });
    return cudaSuccess;
}
FAKE cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    Lock lk;
    put(get(st), [=] { std::memset(p, v, n); });
    return cudaSuccess;
}
FAKE cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
    Lock lk;
    if (k == cudaMemcpyHostToDevice) {  // staged: the copy to the device follows
        std::vector<char> stage(static_cast<const char*>(s), static_cast<const char*>(s) + n);
        put(get(nullptr), [=] { std::memcpy(d, stage.data(), n); });
        return cudaSuccess;
    }
    drain(get(nullptr), ~0ull);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    Lock lk;
    if (k == cudaMemcpyDeviceToHost) {  // to pageable memory: complete on return
        drain(get(st), ~0ull);
        std::memcpy(d, s, n);
        if (scripted_reads > 0 && on_device(s) && n >= 32) {
            --scripted_reads;
            std::memcpy(static_cast<char*>(d) + 24, &status_script, sizeof status_script);
        }
        return cudaSuccess;
    }
    const uint64_t was = sum(s, n);
    put(get(st), [=] {
        if (sum(s, n) != was) violation("the source of an asynchronous copy changed before the copy ran");
        std::memcpy(d, s, n);
    });
    return cudaSuccess;
}
