// A CUDA runtime of bookkeeping alone, for the host side of the library.
//
// The translation units that hold no kernels are compiled with the host compiler and
// linked with this file in place of the CUDA runtime and the kernel launchers.
// "Device" memory is host memory; nothing is computed.  What is kept is what the host
// code is responsible for: which stream work goes to, what it is ordered after (a
// vector clock per stream, carried by events and host synchronisation), what was
// allocated and freed, and what each projection launch reads.  The sim_* functions set
// the scene (memory size, errors to return) and read the record.
#include "internal.cuh"

#include <sys/mman.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

using namespace ctlcu;

namespace {

using Clock = std::map<int, long>;  // stream id -> last operation known to be done before

void merge(Clock& to, const Clock& from)
{
    for (const auto& kv : from)
        if (to[kv.first] < kv.second)
            to[kv.first] = kv.second;
}

struct Alloc {
    size_t bytes;
    int device;
};
struct Built {
    int stream;
    long at;
    Clock reads;  // the last launch of each stream that read it
};

std::mutex mu;
std::map<const void*, Alloc> allocs;        // device memory
std::map<const void*, size_t> pinned;
std::map<const void*, Built> built;         // derived arrays and the operation that wrote them
std::map<cudaStream_t, int> ids;
std::map<int, Clock> clocks;
std::map<cudaEvent_t, Clock> events;
Clock host;
std::map<std::string, int> failures;        // operation -> calls until the one that fails
std::map<int, float> mode_ms;               // loop -> time of a launch, for event timing
std::vector<uint64_t> free_answers;         // what cudaMemGetInfo answers next
std::string record;
uint64_t capacity = 180ull << 30, used = 0;
int capturing = 0, capture_mode = 0, foreign_capture = 0, unsafe_calls = 0;
int last_mode = 0, info_calls = 0;
long next_handle = 16;
thread_local int current = 0;
std::atomic<int> news_left{ 0 };            // allocations until the one that fails, counted from
int news_after_pin = 0;                     // the next pinned allocation on
std::map<int, uint64_t> free_of_device;     // what cudaMemGetInfo answers there, where set

void note(const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    record += buf;
    record += '\n';
}

bool fails(const char* op)
{
    auto it = failures.find(op);
    if (it == failures.end() || --it->second > 0)
        return false;
    failures.erase(it);
    return true;
}

int id_of(cudaStream_t s)
{
    auto it = ids.find(s);
    return it == ids.end() ? 0 : it->second;
}

// One operation on stream `s`: what the host knows to be done comes before it.
long op(cudaStream_t s)
{
    Clock& c = clocks[id_of(s)];
    merge(c, host);
    return ++c[id_of(s)];
}

void host_waits(cudaStream_t s) { merge(host, clocks[id_of(s)]); }

// A call that the runtime refuses while any thread captures in the global mode, unless
// this thread is in the relaxed mode; the capture is then lost.
bool unsafe()
{
    if (!foreign_capture || capture_mode == cudaStreamCaptureModeRelaxed)
        return false;
    ++unsafe_calls;
    return true;
}

cudaError_t take(void** p, size_t bytes, bool pooled)
{
    if (fails(pooled ? "mallocasync" : "malloc") || used + bytes > capacity) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    void* m = mmap(nullptr, bytes ? bytes : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED)
        return cudaErrorMemoryAllocation;
    allocs[m] = { bytes, current };
    used += bytes;
    *p = m;
    return cudaSuccess;
}

cudaError_t give(void* p)
{
    if (!p)
        return cudaSuccess;
    auto it = allocs.find(p);
    if (it == allocs.end())
        return cudaErrorInvalidValue;
    used -= it->second.bytes;
    munmap(p, it->second.bytes ? it->second.bytes : 1);
    allocs.erase(it);
    if (built.erase(p))
        note("freed_array %p", p);
    return cudaSuccess;
}

const Alloc* find(const void* p)
{
    auto it = allocs.upper_bound(p);
    if (it == allocs.begin())
        return nullptr;
    --it;
    return (const char*)p < (const char*)it->first + (it->second.bytes ? it->second.bytes : 1) ? &it->second : nullptr;
}

void wrote(void* p, cudaStream_t s) { built[p] = { id_of(s), op(s), {} }; }

// "-" without an array, "ok" after its build, "race" if nothing orders this stream after
// the build, "stale" if it was freed or never built.
const char* read(const void* p, cudaStream_t s)
{
    if (!p)
        return "-";
    auto it = built.find(p);
    if (it == built.end())
        return "stale";
    Clock& c = clocks[id_of(s)];
    it->second.reads[id_of(s)] = c[id_of(s)];
    return c[it->second.stream] >= it->second.at ? "ok" : "race";
}

}  // namespace

// the library's own allocations
thread_local int in_fake = 0;
struct InFake {
    InFake() { ++in_fake; }
    ~InFake() { --in_fake; }
};
void* operator new(size_t n)
{
    if (in_fake == 0 && news_left.load() > 0 && news_left.fetch_sub(1) == 1)
        throw std::bad_alloc();
    void* p = malloc(n ? n : 1);
    if (!p)
        throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

#define LOCK          \
    InFake in_fake_;  \
    std::lock_guard<std::mutex> lk_(mu)
#define SIM extern "C" __attribute__((visibility("default")))

SIM void sim_reset()
{
    LOCK;
    for (const auto& m : allocs)
        munmap(const_cast<void*>(m.first), m.second.bytes ? m.second.bytes : 1);
    allocs.clear();
    built.clear();
    used = 0;
    failures.clear();
    free_answers.clear();
    free_of_device.clear();
    mode_ms.clear();
    record.clear();
    capacity = 180ull << 30;
    capturing = foreign_capture = unsafe_calls = 0;
}
SIM const char* sim_record() { return record.c_str(); }
SIM void sim_clear_record() { LOCK; record.clear(); }
SIM void sim_capacity(uint64_t bytes) { LOCK; capacity = bytes; }
SIM uint64_t sim_used() { LOCK; return used; }
SIM void sim_free_answers(const uint64_t* v, int n) { LOCK; free_answers.assign(v, v + n); }
SIM void sim_free_of_device(int device, uint64_t bytes) { LOCK; free_of_device[device] = bytes; }
SIM void sim_fail_new_after_pin(int nth) { LOCK; news_after_pin = nth; }
SIM void sim_stop_failing_new() { news_left = 0; }
SIM void sim_fail(const char* what, int nth) { LOCK; failures[what] = nth; }
SIM void sim_mode_ms(int mode, float ms) { LOCK; mode_ms[mode] = ms; }
SIM void sim_capturing(int on) { LOCK; capturing = on; }
SIM void sim_foreign_capture(int on) { LOCK; foreign_capture = on; unsafe_calls = 0; }
SIM int sim_info_calls() { LOCK; return info_calls; }
SIM int sim_unsafe_calls() { LOCK; return unsafe_calls; }
SIM void* sim_device_memory(uint64_t bytes)
{
    LOCK;
    void* p = nullptr;
    take(&p, bytes, false);
    return p;
}
SIM void* sim_stream()
{
    LOCK;
    cudaStream_t s = (cudaStream_t)(next_handle += 16);
    ids[s] = (int)ids.size() + 1;
    return s;
}

// ---- the launchers ------------------------------------------------------------------------------

namespace ctlcu {

cudaError_t launch_setup(const double*, uint32_t, uint32_t, ViewGeom*, double*, double*, int*, cudaStream_t s)
{
    LOCK;
    op(s);
    return cudaSuccess;
}
cudaError_t launch_batch_setup(const BatchSetup*, uint32_t, uint32_t, ViewGeom*, int*, cudaStream_t s)
{
    LOCK;
    op(s);
    return cudaSuccess;
}
cudaError_t launch_pad_convert(const float*, void*, const int*, int, cudaStream_t s)
{
    LOCK;
    op(s);
    return fails("pad_convert") ? cudaErrorLaunchFailure : cudaSuccess;
}
cudaError_t launch_build_cells(const void*, const int*, int, const CellLayout&, void* cells, cudaStream_t s)
{
    LOCK;
    const bool bad = fails("build_cells");
    note("build_cells stream=%d %s", id_of(s), bad ? "failed" : "done");
    if (bad)
        return cudaErrorLaunchFailure;
    wrote(cells, s);
    return cudaSuccess;
}
cudaError_t launch_build_pairs(const void*, const int*, int, const PairLayout&, void* pairs, cudaStream_t s)
{
    LOCK;
    const bool bad = fails("build_pairs");
    note("build_pairs stream=%d %s", id_of(s), bad ? "failed" : "done");
    if (bad)
        return cudaErrorLaunchFailure;
    wrote(pairs, s);
    return cudaSuccess;
}
cudaError_t launch_project(const ProjectArgs& a, Mode mode, Accum, int, cudaStream_t s)
{
    LOCK;
    op(s);
    last_mode = (int)mode;
    note("project mode=%d views=%u stream=%d array=%p %s sub=%u,%u", (int)mode, a.n_views, id_of(s), a.cells,
         read(a.cells, s), a.sub_x, a.sub_y);
    return cudaSuccess;
}
cudaError_t launch_batch(const BatchReq*, uint32_t, uint32_t total, Mode mode, Accum, const LaunchShape& sh,
                         unsigned int*, int* blocks, cudaStream_t s)
{
    LOCK;
    op(s);
    *blocks = 1;
    note("batch mode=%d items=%u", (int)mode, total);
    // the limit of the launcher proper: items times warps per item in 32 bits
    return (uint64_t)total * (sh.block / 32) > 0xffffffffull - (1ull << 20) ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t launch_count(const ProjectArgs&, Mode, cudaStream_t s)
{
    LOCK;
    op(s);
    return cudaSuccess;
}
cudaError_t launch_mean(const void*, const int*, int, double*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_mean_volume(const double*, double, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_unpad_upsample(const void*, const int*, int, int, void*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_average_samples(const float*, uint32_t, uint64_t, float*, bool, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_combine_linear(const float*, const float*, const double*, uint64_t, uint32_t, float*, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_encode_geometry(const ctlcu_detector_desc&, const ctlcu_trajectory_desc&, uint32_t, const double*,
                                   uint32_t, double*, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_poisson_noise(float*, uint32_t, uint32_t, uint32_t, const float*, uint64_t, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_saturation(float*, uint32_t, uint32_t, uint64_t, int, const ctlcu_saturation_model&, const float*,
                              cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_spectral(const float*, uint32_t, uint64_t, uint32_t, const float*, const double*, const float*,
                            const int*, uint32_t, const double*, float*, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_spectral_noisy(const float*, uint32_t, uint32_t, uint32_t, uint32_t, const float*, const double*,
                                  const float*, const int*, const int*, uint32_t, const double*, const float*, uint64_t,
                                  float*, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_transform(float*, uint64_t, uint32_t, const double*, bool, cudaStream_t) { return cudaSuccess; }

}  // namespace ctlcu

// ---- the runtime --------------------------------------------------------------------------------

extern "C" {

cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "simulated"; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m)
{
    LOCK;
    const int old = capture_mode;
    capture_mode = *m;
    *m = (cudaStreamCaptureMode)old;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes)
{
    LOCK;
    if (unsafe()) {
        *p = nullptr;
        return cudaErrorStreamCaptureUnsupported;
    }
    return take(p, bytes, false);
}
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t s)
{
    LOCK;
    op(s);
    return take(p, bytes, true);
}
cudaError_t cudaFree(void* p)
{
    LOCK;
    for (const auto& c : clocks)
        merge(host, c.second);  // cudaFree waits for the device
    return give(p);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s)
{
    LOCK;
    op(s);
    auto it = built.find(p);
    if (it != built.end())
        for (const auto& r : it->second.reads)
            if (clocks[id_of(s)][r.first] < r.second)
                note("freed_while_read %p", p);
    return give(p);
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned)
{
    LOCK;
    *p = malloc(bytes);
    pinned[*p] = bytes;
    news_left = news_after_pin;
    news_after_pin = 0;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) { return cudaHostAlloc(p, bytes, 0); }
cudaError_t cudaFreeHost(void* p)
{
    LOCK;
    pinned.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t)
{
    LOCK;
    ++info_calls;
    *t = capacity;
    *f = used < capacity ? capacity - used : 0;
    if (free_of_device.count(current))
        *f = free_of_device[current];
    if (!free_answers.empty()) {
        *f = free_answers.front();
        free_answers.erase(free_answers.begin());
    }
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    LOCK;
    memset(a, 0, sizeof *a);
    const Alloc* m = find(p);
    a->device = m ? m->device : current;
    a->type = m ? cudaMemoryTypeDevice : pinned.count(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    LOCK;
    op(st);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s)
{
    LOCK;
    op(s);
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)sim_stream(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { LOCK; host_waits(s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize()
{
    LOCK;
    for (const auto& c : clocks)
        merge(host, c.second);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* st)
{
    *st = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)16; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long)
{
    *x = (cudaGraphExec_t)16;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    LOCK;
    *e = (cudaEvent_t)(next_handle += 16);
    events[*e];
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { LOCK; events.erase(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    LOCK;
    op(s);
    events[e] = clocks[id_of(s)];
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { LOCK; merge(host, events[e]); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    LOCK;
    *ms = mode_ms.count(last_mode) ? mode_ms[last_mode] : 10.0f;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    LOCK;
    merge(clocks[id_of(s)], events[e]);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*)
{
    static char scratch[1 << 20];
    *p = scratch;
    return cudaSuccess;
}
cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f) { return { x, y, z, w, f }; }
cudaError_t cudaMalloc3DArray(cudaArray_t* a, const cudaChannelFormatDesc*, cudaExtent, unsigned)
{
    *a = (cudaArray_t)16;
    return cudaSuccess;
}
cudaError_t cudaFreeArray(cudaArray_t) { return cudaSuccess; }
cudaError_t cudaCreateTextureObject(cudaTextureObject_t* t, const cudaResourceDesc*, const cudaTextureDesc*,
                                    const cudaResourceViewDesc*)
{
    *t = 1;
    return cudaSuccess;
}
cudaError_t cudaDestroyTextureObject(cudaTextureObject_t) { return cudaSuccess; }

}  // extern "C"
