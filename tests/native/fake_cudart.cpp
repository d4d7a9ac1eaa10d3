// A stand-in for the CUDA runtime, for CPU tests of the library's host code: linked with the
// library's own objects in place of the runtime.  Device memory is host memory, copies happen at
// once, kernels do nothing.  What is modelled is what host code can get wrong without a GPU
// noticing at once:
//   order    a vector clock per stream, event and the host: fake_pending() counts the operations
//            a call queued that nothing the host waited for is known to come after
//   errors   fake_fail makes the n-th next call of a function fail; the last error sticks until
//            cudaGetLastError takes it; null pointers, streams and events are counted
//   capture  captures begun and not ended, and captures in which a call failed
//   kernels  the names launched
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {
using Clock = std::map<const void*, long long>;
void join(Clock& a, const Clock& b)
{
    for (const auto& kv : b)
        if (a[kv.first] < kv.second) a[kv.first] = kv.second;
}

struct State
{
    Clock                              host, done;   // done: operations queued per stream
    std::map<const void*, Clock>       streams, events;
    std::set<const void*>              live_streams, live_events, pinned;
    std::map<const void*, std::string> names;        // kernels by their host stub
    std::vector<std::string>           launched;
    std::map<std::string, std::pair<int, int>> fail; // function -> (calls to go, error)
    cudaError_t                        last = cudaSuccess;
    long long                          nulls = 0, poll_value = 0;
    const void*                        capturing = nullptr;
    std::set<const void*>              captured;     // streams that joined the capture
    bool                               capture_bad = false;
    long long                          open_captures = 0;
};
State& S()
{
    static State s;
    return s;
}

cudaError_t result(const char* fn)
{
    auto it = S().fail.find(fn);
    if (it == S().fail.end() || --it->second.first > 0) return cudaSuccess;
    const cudaError_t e = static_cast<cudaError_t>(it->second.second);
    S().fail.erase(it);
    S().last = e;
    if (S().capturing) S().capture_bad = true;
    return e;
}
// an operation on a stream, after everything the host has waited for
void op(const void* st)
{
    if (S().capturing && S().captured.count(st)) return;
    Clock& c = S().streams[st];
    join(c, S().host);
    c[st] = ++S().done[st];
}
void must(const void* p)
{
    if (!p) ++S().nulls;
}

struct Config
{
    dim3   grid, block;
    size_t shared;
    void*  stream;
};
std::vector<Config> configs;
}  // namespace

#define FAKE extern "C" __attribute__((visibility("hidden")))
#define TEST extern "C" __attribute__((visibility("default")))
#define TRY(fn)                          \
    do                                   \
    {                                    \
        cudaError_t e_ = result(fn);     \
        if (e_ != cudaSuccess) return e_; \
    } while (0)

TEST void      fake_fail(const char* fn, int nth, int error) { S().fail[fn] = {nth, error}; }
TEST int       fake_fails_left() { return static_cast<int>(S().fail.size()); }
TEST void      fake_poll(long long value) { S().poll_value = value; }  // what copies to page-locked memory read
TEST long long fake_nulls() { return S().nulls; }
TEST long long fake_open_captures() { return S().open_captures; }
TEST long long fake_pending()
{
    long long n = 0;
    for (const auto& kv : S().done) n += kv.second - S().host[kv.first];
    return n;
}
TEST int         fake_launches() { return static_cast<int>(S().launched.size()); }
TEST const char* fake_launch(int i) { return S().launched[i].c_str(); }
TEST void        fake_forget() { S().launched.clear(); }

// memory
FAKE cudaError_t cudaMalloc(void** p, size_t n)
{
    TRY("cudaMalloc");
    *p = std::calloc(1, n ? n : 1);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
FAKE cudaError_t cudaFree(void* p)
{
    std::free(p);
    return cudaSuccess;
}
FAKE cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    TRY("cudaHostAlloc");
    *p = std::calloc(1, n);
    S().pinned.insert(*p);
    return cudaSuccess;
}
static cudaError_t copy(void* d, const void* s, size_t n)
{
    must(d);
    must(s);
    for (const void* p : S().pinned)
        if (d >= p && d < static_cast<const char*>(p) + 64 && n == sizeof(long long))
        {
            std::memcpy(d, &S().poll_value, n);
            return cudaSuccess;
        }
    if (d && s) std::memcpy(d, s, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    TRY("cudaMemcpy");
    return copy(d, s, n);
}
FAKE cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    TRY("cudaMemcpyAsync");
    op(st);
    return copy(d, s, n);
}
FAKE cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
    TRY("cudaMemsetAsync");
    must(d);
    op(st);
    if (d) std::memset(d, v, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaGetSymbolAddress(void** p, const void* s)
{
    *p = const_cast<void*>(s);
    return cudaSuccess;
}

// streams and events
FAKE cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    TRY("cudaStreamCreateWithFlags");
    *s = static_cast<cudaStream_t>(std::malloc(1));
    S().live_streams.insert(*s);
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    S().live_streams.erase(s);  // (a capture that began on it stays begun)
    if (S().capturing == s) S().capturing = nullptr;
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    TRY("cudaStreamSynchronize");
    join(S().host, S().streams[s]);
    return cudaSuccess;
}
FAKE cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    TRY("cudaEventCreateWithFlags");
    *e = static_cast<cudaEvent_t>(std::malloc(1));
    S().live_events.insert(*e);
    S().events[*e].clear();
    return cudaSuccess;
}
FAKE cudaError_t cudaEventCreate(cudaEvent_t* e)
{
    TRY("cudaEventCreate");
    return cudaEventCreateWithFlags(e, 0);
}
FAKE cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    S().live_events.erase(e);
    return cudaSuccess;
}
FAKE cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    TRY("cudaEventRecord");
    must(e);
    if (S().capturing && S().captured.count(s)) return cudaSuccess;
    S().events[e] = S().streams[s];
    return cudaSuccess;
}
FAKE cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    TRY("cudaEventSynchronize");
    must(e);
    join(S().host, S().events[e]);
    return cudaSuccess;
}
FAKE cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.f;
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    TRY("cudaStreamWaitEvent");
    must(e);
    if (S().capturing)
    {
        S().captured.insert(s);
        return cudaSuccess;
    }
    join(S().streams[s], S().events[e]);
    return cudaSuccess;
}

// capture and graphs
FAKE cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
    TRY("cudaStreamBeginCapture");
    S().capturing = s;
    S().captured = {s};
    S().capture_bad = false;
    ++S().open_captures;
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
    S().capturing = nullptr;
    --S().open_captures;
    *g = nullptr;
    if (S().capture_bad)
    {
        S().last = cudaErrorStreamCaptureInvalidated;
        return cudaErrorStreamCaptureInvalidated;
    }
    *g = static_cast<cudaGraph_t>(std::malloc(1));
    return cudaSuccess;
}
FAKE cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long)
{
    TRY("cudaGraphInstantiate");
    *x = static_cast<cudaGraphExec_t>(std::malloc(1));
    return cudaSuccess;
}
FAKE cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s)
{
    TRY("cudaGraphLaunch");
    op(s);
    return cudaSuccess;
}
FAKE cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

// the device: 152 SMs, four blocks of any kernel on each
FAKE cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
FAKE cudaError_t cudaSetDevice(int) { return cudaSuccess; }
FAKE cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int)
{
    *v = 152;
    return cudaSuccess;
}
FAKE cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
FAKE cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}

// errors
FAKE const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
FAKE cudaError_t cudaGetLastError()
{
    const cudaError_t e = S().last;
    S().last = cudaSuccess;
    return e;
}

// kernel launches, as nvcc's host code makes them
FAKE void** __cudaRegisterFatBinary(void*)
{
    static void* handle;
    return &handle;
}
FAKE void __cudaRegisterFatBinaryEnd(void**) {}
FAKE void __cudaUnregisterFatBinary(void**) {}
FAKE void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
FAKE void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, void*, void*, void*, void*,
                                 int*)
{
    S().names[stub] = name;
}
FAKE unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, void* stream)
{
    configs.push_back({grid, block, shared, stream});
    return 0;
}
FAKE cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream)
{
    const Config c = configs.back();
    configs.pop_back();
    *grid = c.grid;
    *block = c.block;
    *shared = c.shared;
    *static_cast<void**>(stream) = c.stream;
    return cudaSuccess;
}
FAKE cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* stub)
{
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(stub));
    return cudaSuccess;
}
FAKE cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t st)
{
    TRY("cudaLaunchKernel");
    S().launched.push_back(S().names[reinterpret_cast<const void*>(k)]);
    op(st);
    return cudaSuccess;
}
