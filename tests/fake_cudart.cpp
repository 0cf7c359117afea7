// A CUDA runtime of two devices in host memory, for tests of what the engine
// asks of the real one: which device is current at each launch, what is
// allocated and when, what is launched, and how errors are passed on. Kernels
// do not run; copies and fills are done at once. A launch, or an event record,
// on a stream of another device than the thread's current one fails as it does
// there. Linked with the library's objects in place of the CUDA runtime.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <mutex>
#include <string>

namespace {

std::mutex mu;
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local struct { dim3 grid, block; size_t smem; cudaStream_t stream; } pushed;

struct Stream {
    int device;
    long captured;
    Stream *capture;            // the stream whose capture takes what is launched here
    bool busy;
    std::set<Stream *> after;   // streams whose work it has waited for
};
struct Event { int device; Stream *stream, *capture; };
struct Graph { long launches; };

std::map<void *, std::pair<int, size_t>> memory;
std::map<Stream *, int> streams;
std::map<const void *, std::string> kernels;
std::map<std::string, long> counts;
long copies_left = -1;   // copies until one fails (-1: none does)
double static_scratch[1 << 17];
float elapsed = 1.f, elapsed_factor = 1.f;   // what the next pair of events measures, and how it changes

Stream *S(cudaStream_t s) { return reinterpret_cast<Stream *>(s); }
cudaError_t ret(cudaError_t e) { return e == cudaSuccess ? e : last = e; }

void settle(Stream *s) {   // what s has, and what it has waited for, is done
    std::lock_guard<std::mutex> l(mu);
    if (!streams.count(s)) return;
    s->busy = false;
    for (Stream *t : s->after)
        if (streams.count(t)) t->busy = false;
}

cudaError_t launch(const void *f, dim3 grid, cudaStream_t stream) {
    std::lock_guard<std::mutex> l(mu);
    if (!grid.x || !grid.y || !grid.z) return ret(cudaErrorInvalidConfiguration);
    if (S(stream)->device != current) return ret(cudaErrorInvalidResourceHandle);
    if (S(stream)->capture) {
        S(stream)->capture->captured++;
        return cudaSuccess;
    }
    S(stream)->busy = true;
    counts["launch"]++;
    counts[kernels[f]]++;
    return cudaSuccess;
}

CUresult encode(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// what the tests ask: "malloc", "free", "free in flight" (with launches that nothing has waited for), "live" (bytes), "up" (copies to the device), "launch", "graph" (replays), "capture", or a kernel's name
__attribute__((visibility("default"))) long fake_count(const char *what) {
    std::lock_guard<std::mutex> l(mu);
    if (!std::strcmp(what, "live")) {
        long n = 0;
        for (auto &m : memory) n += (long)m.second.second;
        return n;
    }
    long n = 0;
    for (auto &c : counts)
        if (c.first == what || (c.first.size() > std::strlen(what) && c.first.find("cb2") != std::string::npos &&
                                c.first.find(what) != std::string::npos))
            n += c.second;
    return n;
}
__attribute__((visibility("default"))) void fake_fail_copy(long after) {
    copies_left = after;
    last = cudaSuccess;
}
__attribute__((visibility("default"))) void fake_elapsed(float ms, float factor) { elapsed = ms; elapsed_factor = factor; }
__attribute__((visibility("default"))) int fake_current() { return current; }
__attribute__((visibility("default"))) void fake_set_current(int d) { current = d; }

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    kernels[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *stream) {
    pushed = {g, b, smem, static_cast<cudaStream_t>(stream)};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *stream) {
    *g = pushed.grid; *b = pushed.block; *smem = pushed.smem;
    *static_cast<cudaStream_t *>(stream) = pushed.stream;
    return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **, size_t, cudaStream_t s) { return launch(f, g, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) { return launch(f, c->gridDim, c->stream); }
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 1) return ret(cudaErrorInvalidDevice);
    current = d;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::mutex> l(mu);
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    std::memset(*p, 0xff, n);
    memory[*p] = {current, n};
    counts["malloc"]++;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> l(mu);
    if (!p) return cudaSuccess;
    if (!memory.erase(p)) return ret(cudaErrorInvalidValue);
    std::free(p);
    counts["free"]++;
    for (auto &s : streams)
        if (s.first->busy) { counts["free in flight"]++; break; }
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    if (kind == cudaMemcpyHostToDevice) {
        std::lock_guard<std::mutex> l(mu);
        counts["up"]++;
    }
    if (copies_left >= 0 && copies_left-- == 0) return ret(cudaErrorUnknown);
    std::memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidResourceHandle ? "invalid resource handle" : "fake error"; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = static_scratch; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **f, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *f = reinterpret_cast<void *>(&encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    std::lock_guard<std::mutex> l(mu);
    Stream *n = new Stream{current, 0, nullptr, false, {}};
    streams[n] = 1;
    *s = reinterpret_cast<cudaStream_t>(n);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::lock_guard<std::mutex> l(mu);
    streams.erase(S(s));
    delete S(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { settle(S(s)); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { return ret(S(s)->busy ? cudaErrorNotReady : cudaSuccess); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    const Event *ev = reinterpret_cast<Event *>(e);
    if (ev->stream) S(s)->after.insert(ev->stream);
    if (ev->capture && ev->capture->capture) S(s)->capture = ev->capture;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(new Event{current, nullptr, nullptr});
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    reinterpret_cast<Event *>(e)->stream = S(s);
    reinterpret_cast<Event *>(e)->capture = S(s)->capture;
    return ret(reinterpret_cast<Event *>(e)->device == S(s)->device ? cudaSuccess : cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {   // (of all that its stream has: enough for a wait at the end)
    Stream *s = reinterpret_cast<Event *>(e)->stream;
    if (s) settle(s);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = elapsed;
    elapsed *= elapsed_factor;
    return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    S(s)->capture = S(s);
    S(s)->captured = 0;
    std::lock_guard<std::mutex> l(mu);
    counts["capture"]++;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
    {
        std::lock_guard<std::mutex> l(mu);
        for (auto &t : streams)
            if (t.first->capture == S(s)) t.first->capture = nullptr;
    }
    *g = reinterpret_cast<cudaGraph_t>(new Graph{S(s)->captured});
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph *>(g); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
    *x = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph *>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete reinterpret_cast<Graph *>(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
    std::lock_guard<std::mutex> l(mu);
    if (S(s)->device != current) return ret(cudaErrorInvalidResourceHandle);
    S(s)->busy = true;
    counts["graph"]++;
    return cudaSuccess;
}

}  // extern "C"
