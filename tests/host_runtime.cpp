// Stand-ins for the CUDA runtime calls of libsph_cuda's host code, linked
// around its objects with ld's --wrap, so that the order of its copies, waits
// and launches can be tested without a GPU.
//
// Device memory is host memory.  A stream is a queue: what is put on it runs
// when something waits for it and not before, the latest that a GPU may run
// it; copies without a stream run at once, past every (non-blocking) stream.
// Kernels do nothing.  host_fail() makes a coming call of a kind fail,
// host_hold() makes a coming host-to-device copy wait until host_release().
#include <cuda_runtime_api.h>

#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {

struct Stream {
    std::deque<std::function<void()>> work;
    bool capturing = false;
};
struct Event {
    Stream *stream = nullptr;
    size_t until = 0;  // items of the stream's queue that it waits for
};

std::recursive_mutex g_mu;
std::vector<Stream *> g_streams;
std::vector<Event *> g_events;
std::map<std::string, std::pair<int, cudaError_t>> g_fail;  // call -> (calls until it fails, error)
thread_local cudaError_t g_last = cudaSuccess;
std::string g_log;

std::mutex g_hold_mu;
std::condition_variable g_hold_cv;
bool g_hold = false, g_held = false;

void note(const std::string &s)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    g_log += s + "\n";
}

cudaError_t failing(const std::string &call)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    auto f = g_fail.find(call);
    if (f != g_fail.end() && f->second.first >= 0 && f->second.first-- == 0) return g_last = f->second.second;
    return cudaSuccess;
}

void drain(Stream *s, size_t items)
{
    for (; items > 0 && !s->work.empty(); --items) {
        auto f = std::move(s->work.front());
        s->work.pop_front();
        for (Event *e : g_events)
            if (e->stream == s && e->until > 0) --e->until;
        f();
    }
}

cudaError_t put(cudaStream_t st, std::function<void()> f)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    Stream *s = reinterpret_cast<Stream *>(st);
    if (!s) f();
    else if (!s->capturing) s->work.push_back(std::move(f));
    return cudaSuccess;
}

std::string number(const void *p, size_t n)
{
    return std::to_string((size_t)p) + " " + std::to_string(n);
}

}  // namespace

extern "C" {

void host_fail(const char *call, int after, int error)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    g_fail[call] = {after, (cudaError_t)error};
}
void host_reset(void)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    g_fail.clear();
    g_log.clear();
    g_last = cudaSuccess;
}
const char *host_log(void)  // and starts a new one
{
    static std::string out;
    std::lock_guard<std::recursive_mutex> l(g_mu);
    out.swap(g_log);
    g_log.clear();
    return out.c_str();
}
void *host_stream(int capturing)
{
    Stream *s = new Stream;
    s->capturing = capturing != 0;
    return s;
}
void host_hold(void)
{
    std::lock_guard<std::mutex> l(g_hold_mu);
    g_hold = true;
}
int host_wait_held(void)  // 1 once a copy is held, 0 after 10 s
{
    std::unique_lock<std::mutex> l(g_hold_mu);
    return g_hold_cv.wait_for(l, std::chrono::seconds(10), [] { return g_held; });
}
void host_release(void)
{
    std::lock_guard<std::mutex> l(g_hold_mu);
    g_held = false;
    g_hold_cv.notify_all();
}

#define W(name) __wrap_##name

cudaError_t W(cudaGetLastError)()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t W(cudaGetDevice)(int *d) { *d = 0; return cudaSuccess; }
cudaError_t W(cudaDeviceGetAttribute)(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;  // no shared page tables: buffers are copied
    return cudaSuccess;
}
cudaError_t W(cudaPointerGetAttributes)(cudaPointerAttributes *a, const void *)
{
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t W(cudaMalloc)(void **p, size_t n)
{
    const cudaError_t e = failing("cudaMalloc");
    *p = e ? nullptr : std::calloc(n ? n : 1, 1);
    if (!e) note("malloc " + number(*p, n));
    return e;
}
cudaError_t W(cudaFree)(void *p)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    for (Stream *s : g_streams) drain(s, s->work.size());
    if (p) note("free " + number(p, 0));
    std::free(p);
    return cudaSuccess;
}
cudaError_t W(cudaHostAlloc)(void **p, size_t n, unsigned) { *p = std::calloc(n ? n : 1, 1); return cudaSuccess; }
cudaError_t W(cudaFreeHost)(void *p) { std::free(p); return cudaSuccess; }
cudaError_t W(cudaFuncSetAttribute)(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t W(cudaGetSymbolAddress)(void **p, const void *) { *p = nullptr; return cudaErrorInvalidSymbol; }

cudaError_t W(cudaMemcpy)(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t W(cudaMemset)(void *d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t W(cudaMemcpyAsync)(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st)
{
    if (k == cudaMemcpyHostToDevice) {
        note("h2d " + number(d, n));
        std::unique_lock<std::mutex> l(g_hold_mu);
        if (g_hold) {
            g_hold = false;
            g_held = true;
            g_hold_cv.notify_all();
            g_hold_cv.wait_for(l, std::chrono::seconds(20), [] { return !g_held; });
        }
        std::vector<char> copy((const char *)s, (const char *)s + n);  // pageable: taken at the call
        return put(st, [=] { std::memcpy(d, copy.data(), n); });
    }
    return put(st, [=] { std::memcpy(d, s, n); });
}
cudaError_t W(cudaMemsetAsync)(void *d, int v, size_t n, cudaStream_t st)
{
    note("memset " + number(d, n));
    return put(st, [=] { std::memset(d, v, n); });
}

cudaError_t W(cudaStreamCreateWithFlags)(cudaStream_t *s, unsigned)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    g_streams.push_back(new Stream);
    *s = reinterpret_cast<cudaStream_t>(g_streams.back());
    return cudaSuccess;
}
cudaError_t W(cudaStreamDestroy)(cudaStream_t) { return cudaSuccess; }
cudaError_t W(cudaStreamSynchronize)(cudaStream_t st)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    Stream *s = reinterpret_cast<Stream *>(st);
    if (s && s->capturing) return cudaErrorStreamCaptureUnsupported;
    if (s) drain(s, s->work.size());
    return cudaSuccess;
}
cudaError_t W(cudaStreamIsCapturing)(cudaStream_t st, cudaStreamCaptureStatus *c)
{
    Stream *s = reinterpret_cast<Stream *>(st);
    *c = s && s->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t W(cudaStreamWaitEvent)(cudaStream_t, cudaEvent_t ev, unsigned)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    Event *e = reinterpret_cast<Event *>(ev);
    if (e->stream) drain(e->stream, e->until);
    return cudaSuccess;
}
cudaError_t W(cudaEventCreate)(cudaEvent_t *e)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    g_events.push_back(new Event);
    *e = reinterpret_cast<cudaEvent_t>(g_events.back());
    return cudaSuccess;
}
cudaError_t W(cudaEventCreateWithFlags)(cudaEvent_t *e, unsigned) { return W(cudaEventCreate)(e); }
cudaError_t W(cudaEventDestroy)(cudaEvent_t) { return cudaSuccess; }
cudaError_t W(cudaEventRecord)(cudaEvent_t ev, cudaStream_t st)
{
    std::lock_guard<std::recursive_mutex> l(g_mu);
    Event *e = reinterpret_cast<Event *>(ev);
    e->stream = reinterpret_cast<Stream *>(st);
    e->until = e->stream ? e->stream->work.size() : 0;
    return cudaSuccess;
}
cudaError_t W(cudaEventSynchronize)(cudaEvent_t ev) { return W(cudaStreamWaitEvent)(nullptr, ev, 0); }
cudaError_t W(cudaEventElapsedTime)(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t W(cudaStreamBeginCapture)(cudaStream_t st, cudaStreamCaptureMode)
{
    const cudaError_t e = failing("cudaStreamBeginCapture");
    reinterpret_cast<Stream *>(st)->capturing = e == cudaSuccess;
    return e;
}
cudaError_t W(cudaStreamEndCapture)(cudaStream_t st, cudaGraph_t *g)
{
    reinterpret_cast<Stream *>(st)->capturing = false;
    *g = reinterpret_cast<cudaGraph_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t W(cudaGraphInstantiate)(cudaGraphExec_t *x, cudaGraph_t, unsigned long long)
{
    const cudaError_t e = failing("cudaGraphInstantiate");
    *x = e ? nullptr : reinterpret_cast<cudaGraphExec_t>(std::malloc(1));
    note(std::string("instantiate ") + (e ? "failed" : "ok"));
    return e;
}
cudaError_t W(cudaGraphDestroy)(cudaGraph_t g) { std::free(g); return cudaSuccess; }
cudaError_t W(cudaGraphExecDestroy)(cudaGraphExec_t x) { std::free(x); return cudaSuccess; }
cudaError_t W(cudaGraphLaunch)(cudaGraphExec_t x, cudaStream_t)
{
    note("graph " + number(x, 0));
    return cudaSuccess;
}
cudaError_t W(cudaLaunchKernelExC)(const cudaLaunchConfig_t *, const void *, void **)
{
    note("launch");
    return failing("launch");
}
cudaError_t W(__cudaLaunchKernel)(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t)
{
    note("launch");
    return failing("launch");
}

}  // extern "C"
