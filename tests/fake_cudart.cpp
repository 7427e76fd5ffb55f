// A CUDA runtime without a GPU, for tests of the library's host code: linked
// with the library's own objects in place of the CUDA runtime.  Device memory
// is host memory, kernels do nothing, streams only count what was ordered on
// them.  It keeps what the tests ask for: work pending on a stream, kernels
// launched while an upload of the legacy stream may be on its way, bytes
// allocated, the dynamic shared memory limit of every kernel, and it can fail
// the n-th call that may fail.
#include <cuda_runtime_api.h>

#include <sys/mman.h>

#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

struct CUstream_st
{
    long long ordered = 0, done = 0; // operations
    bool      capturing = false;
};
struct CUevent_st
{
    cudaStream_t s  = nullptr;
    long long    at = 0;
};

namespace {

std::recursive_mutex               g_mutex;
std::set<cudaStream_t>             g_streams;
CUstream_st                        g_legacy;
std::map<char*, size_t>            g_blocks;
size_t                             g_live = 0, g_peak = 0, g_limit = (size_t)180 << 30;
std::map<const void*, std::string>& names() // filled before this file's statics may be
{
    static auto& m = *new std::map<const void*, std::string>;
    return m;
}
std::map<const void*, std::set<int>> g_limits; // every dynamic shared memory limit a kernel was given
std::map<const void*, int>         g_limit_now;
long                               g_calls = 0, g_fail_at = 0;
int                                g_bad = 0; // streams destroyed with work pending
int                                g_early = 0; // launches while an upload may be on its way
cudaError_t                        g_last = cudaSuccess;

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t err(cudaError_t e)
{
    if (e != cudaSuccess)
        g_last = e;
    return e;
}

// Counts a call that may fail; true when this one is to.
bool fails() { return ++g_calls == g_fail_at; }

CUstream_st& stream_of(cudaStream_t s) { return s && s != cudaStreamLegacy ? *s : g_legacy; }

void order(cudaStream_t s)
{
    CUstream_st& st = stream_of(s);
    if (!st.capturing)
        ++st.ordered;
}

// A kernel or graph launch: the library's streams do not wait for the legacy one.
void launch(cudaStream_t s)
{
    CUstream_st& st = stream_of(s);
    if (&st != &g_legacy && !st.capturing)
        g_early += g_legacy.ordered > g_legacy.done;
    order(s);
}

struct Config
{
    dim3         g, b;
    size_t       smem;
    cudaStream_t s;
};
thread_local Config t_config;

} // namespace

extern "C" {

// ---- for the tests ---------------------------------------------------------
void fake_reset(long fail_at)
{
    Lock l(g_mutex);
    g_calls   = 0;
    g_fail_at = fail_at;
    g_bad     = 0;
    g_early   = 0;
    g_peak    = g_live;
    g_last    = cudaSuccess;
}
long fake_calls()
{
    Lock l(g_mutex);
    return g_calls;
}
int fake_pending()
{
    Lock l(g_mutex);
    int  n = 0;
    for (cudaStream_t s : g_streams)
        n += s->ordered > s->done;
    return n;
}
int    fake_bad() { return g_bad; }
int    fake_early() { return g_early; }
size_t fake_live() { return g_live; }
size_t fake_peak() { return g_peak; }
void   fake_limit(size_t bytes) { g_limit = bytes; }
// Kernels whose dynamic shared memory limit was set to more than one value.
int fake_varying_limits(char* out, int len)
{
    Lock        l(g_mutex);
    int         n = 0;
    std::string all;
    for (auto& [f, v] : g_limits)
        if (v.size() > 1)
        {
            ++n;
            all += names()[f] + " ";
        }
    std::strncpy(out, all.c_str(), (size_t)len - 1);
    out[len - 1] = 0;
    return n;
}
// Kernels that were given a limit at all.
int fake_limited()
{
    Lock l(g_mutex);
    return (int)g_limits.size();
}

// ---- the runtime -----------------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int)
{
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int)
{
    std::memset(p, 0, sizeof(*p));
    p->major               = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "failed"; }
cudaError_t cudaGetLastError()
{
    Lock              l(g_mutex);
    const cudaError_t e = g_last;
    g_last              = cudaSuccess;
    return e;
}
cudaError_t cudaMalloc(void** p, size_t n)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorMemoryAllocation);
    if (g_live + n > g_limit)
        return err(cudaErrorMemoryAllocation);
    void* q = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (q == MAP_FAILED)
        return err(cudaErrorMemoryAllocation);
    g_blocks[(char*)q] = n;
    g_live += n;
    g_peak = g_live > g_peak ? g_live : g_peak;
    *p     = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    Lock l(g_mutex);
    for (cudaStream_t s : g_streams) // waits for the device
        s->done = s->ordered;
    g_legacy.done = g_legacy.ordered;
    auto it = g_blocks.find((char*)p);
    if (it == g_blocks.end())
        return p ? err(cudaErrorInvalidValue) : cudaSuccess;
    munmap(p, it->second);
    g_live -= it->second;
    g_blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*)
{
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol)
{
    *p = const_cast<void*>(symbol);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    std::memcpy(d, s, n);
    g_legacy.done = g_legacy.ordered; // the stream is synchronised before the copy
    if (kind == cudaMemcpyHostToDevice)
        ++g_legacy.ordered; // from pageable memory: on its way when the call returns
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind)
{
    for (size_t i = 0; i < h; ++i)
        std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    std::memcpy(d, s, n);
    order(st);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n)
{
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    std::memset(d, v, n);
    order(st);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    *s = new CUstream_st;
    g_streams.insert(*s);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    Lock l(g_mutex);
    g_bad += s->ordered > s->done;
    g_streams.erase(s);
    delete s;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    Lock         l(g_mutex);
    CUstream_st& st = stream_of(s);
    if (st.capturing)
        return err(cudaErrorStreamCaptureUnsupported);
    st.done = st.ordered;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c)
{
    *c = s && s->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
    s->capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g)
{
    s->capturing = false;
    *g           = (cudaGraph_t)s;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    *e = (cudaGraphExec_t)g;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    launch(s);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e)
{
    *e = new CUevent_st;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    delete e;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    if (s && !s->capturing)
    {
        e->s  = s;
        e->at = s->ordered;
    }
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    Lock l(g_mutex);
    if (e->s && g_streams.count(e->s) && e->s->done < e->at)
        e->s->done = e->at;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v)
{
    Lock l(g_mutex);
    if (fails())
        return err(cudaErrorUnknown);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize)
    {
        g_limits[f].insert(v);
        g_limit_now[f] = v;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t smem, cudaStream_t s)
{
    Lock      l(g_mutex);
    auto      it    = g_limit_now.find(f);
    const int limit = it == g_limit_now.end() ? 48 * 1024 : it->second;
    if (fails() || g.x == 0 || g.y == 0 || b.x == 0 || b.x > 1024 || smem > (size_t)limit)
        return err(cudaErrorInvalidValue);
    launch(s);
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s)
{
    t_config = Config{g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s)
{
    *g                 = t_config.g;
    *b                 = t_config.b;
    *smem              = t_config.smem;
    *(cudaStream_t*)s = t_config.s;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*)
{
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*)
{
    names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

} // extern "C"
