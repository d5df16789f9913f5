// fake_cuda.cpp - A CUDA runtime without a GPU, for the host side of the library.
//
// tests/test_host_runtime.py links it with bh_capi.cpp (the C-ABI), bh_scene.cpp
// and bh_adjoint_frame.cpp, compiled as they are.  Device memory is host memory.
// A stream is a list of operations: they run when the stream, or one that waits
// for it, is synchronised, and every synchronisation lets each stream run up to its
// next copy into host memory (the device makes progress; a copy into the caller's
// memory stays outstanding until somebody waits for it).  The kernels' launch
// wrappers fill what the host looks at: the rays' counters, and pixels that
// hold their own index.
//
// fake_fail(name, nth) makes the nth call of a function from now on fail,
// fake_memory(bytes) bounds the device memory, fake_without_wait_value(1) takes
// cuStreamWaitValue32 away.
#include <cuda.h>
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "../../blackhole_b200/csrc/bh_adjoint.h"
#include "../../blackhole_b200/csrc/bh_display.h"
#include "../../blackhole_b200/csrc/bh_launch.h"
#include "../../include/bh_gpu.h"

namespace {

struct Op {
    std::function<void()> run;
    bool to_host;
};
struct Stream {
    std::vector<Op> ops;
    size_t done = 0;
};
struct Event {
    Stream* stream = nullptr;
    size_t upto = 0;
};

std::vector<Stream*> g_streams;
std::vector<std::unique_ptr<Stream>> g_graphs;      // captured operations
Stream* g_capturing = nullptr;
size_t g_capture_from = 0;
std::map<void*, size_t> g_blocks;
size_t g_used = 0, g_limit = SIZE_MAX;
bool g_no_wait_value = false;
std::map<std::string, int> g_fail;                  // calls until the failing one
std::map<std::string, long long> g_count;

bool fails(const char* name) {
    ++g_count[name];
    auto it = g_fail.find(name);
    if (it == g_fail.end() || it->second <= 0) return false;
    return --it->second == 0;
}

void run_to(Stream* s, size_t upto) {
    while (s->done < upto && s->done < s->ops.size()) {
        const size_t i = s->done++;
        s->ops[i].run();
    }
}
// Every stream up to its next copy into host memory.
void progress() {
    for (bool moved = true; moved;) {
        moved = false;
        for (Stream* s : g_streams)
            while (s != g_capturing && s->done < s->ops.size() && !s->ops[s->done].to_host) {
                run_to(s, s->done + 1);
                moved = true;
            }
    }
}
void push(Stream* s, std::function<void()> f, bool to_host = false) { s->ops.push_back({std::move(f), to_host}); }
Stream* stream_of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
Event* event_of(cudaEvent_t e) { return reinterpret_cast<Event*>(e); }

cudaError_t new_stream(cudaStream_t* out) {
    Stream* s = new Stream;
    g_streams.push_back(s);
    *out = reinterpret_cast<cudaStream_t>(s);
    return cudaSuccess;
}

CUresult wait_value(CUstream s, CUdeviceptr at, cuuint32_t value, unsigned int) {
    if (fails("cuStreamWaitValue32")) return CUDA_ERROR_UNKNOWN;
    push(reinterpret_cast<Stream*>(s), [at, value] {
        const volatile uint32_t* p = reinterpret_cast<const uint32_t*>(at);
        for (int i = 0; i < 4 && *p < value; ++i)
            for (Stream* t : g_streams)
                while (t->done < t->ops.size() && !t->ops[t->done].to_host && *p < value) run_to(t, t->done + 1);
        if (*p < value) {
            std::fprintf(stderr, "fake_cuda: a stream would wait for good\n");
            std::abort();
        }
    });
    return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

void fake_reset() {
    g_fail.clear();
    g_count.clear();
    g_limit = SIZE_MAX;
    g_no_wait_value = false;
}
void fake_fail(const char* name, int nth) { g_fail[name] = nth; }
long long fake_count(const char* name) { return g_count[name]; }
void fake_memory(long long bytes) { g_limit = bytes < 0 ? SIZE_MAX : static_cast<size_t>(bytes); }
long long fake_memory_used() { return static_cast<long long>(g_used); }
void fake_without_wait_value(int on) { g_no_wait_value = on != 0; }
// Copies into host memory that have been enqueued and have not run.
int fake_outstanding_copies() {
    int n = 0;
    for (Stream* s : g_streams)
        for (size_t i = s->done; i < s->ops.size(); ++i) n += s->ops[i].to_host;
    return n;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* most) { *least = 0; *most = -5; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *fn = g_no_wait_value ? nullptr : reinterpret_cast<void*>(wait_value);
    if (q) *q = g_no_wait_value ? cudaDriverEntryPointSymbolNotFound : cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) {
    if (fails("cudaMalloc") || g_used + n > g_limit) return cudaErrorMemoryAllocation;
    // zero pages that take no memory until they are written
    *p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (*p == MAP_FAILED) return cudaErrorMemoryAllocation;
    g_blocks[*p] = n;
    g_used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    for (Stream* s : g_streams) run_to(s, s->ops.size());      // cudaFree waits for the device
    g_used -= g_blocks[p];
    munmap(p, g_blocks[p]);
    g_blocks.erase(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
    *total = g_limit == SIZE_MAX ? (size_t)180 << 30 : g_limit;
    *free_bytes = *total - g_used;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) {
    if (fails("cudaHostAlloc")) return cudaErrorMemoryAllocation;
    *p = std::calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) { return new_stream(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned int, int) { return new_stream(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    run_to(stream_of(s), stream_of(s)->ops.size());
    for (size_t i = 0; i < g_streams.size(); ++i)
        if (g_streams[i] == stream_of(s)) g_streams.erase(g_streams.begin() + i);
    // kept: events may still point at it
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (!s) return cudaErrorInvalidResourceHandle;
    const bool bad = fails("cudaStreamSynchronize");
    if (bad) return cudaErrorUnknown;
    progress();
    run_to(stream_of(s), stream_of(s)->ops.size());
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned int) {
    if (!s || !e) return cudaErrorInvalidResourceHandle;
    if (fails("cudaStreamWaitEvent")) return cudaErrorUnknown;
    Stream* on = event_of(e)->stream;
    const size_t upto = event_of(e)->upto;
    push(stream_of(s), [on, upto] {
        if (on) run_to(on, upto);
    });
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) {
    if (fails("cudaEventCreateWithFlags")) return cudaErrorUnknown;
    *e = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete event_of(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (!e || !s) return cudaErrorInvalidResourceHandle;
    if (fails("cudaEventRecord")) return cudaErrorUnknown;
    event_of(e)->stream = stream_of(s);
    event_of(e)->upto = stream_of(s)->ops.size();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (event_of(e)->stream) run_to(event_of(e)->stream, event_of(e)->upto);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    if (fails("cudaMemcpyAsync")) return cudaErrorUnknown;
    if (k == cudaMemcpyHostToDevice) {
        // pageable memory is staged before the call returns
        auto held = std::make_shared<std::vector<char>>(static_cast<const char*>(s), static_cast<const char*>(s) + n);
        push(stream_of(st), [=] { std::memcpy(d, held->data(), n); });
    } else {
        push(stream_of(st), [=] { std::memcpy(d, s, n); }, true);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t st) {
    if (fails("cudaMemcpy2DAsync")) return cudaErrorUnknown;
    push(stream_of(st), [=] {
        for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
    }, true);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    if (fails("cudaMemsetAsync")) return cudaErrorUnknown;
    push(stream_of(st), [=] { std::memset(d, v, n); });
    return cudaSuccess;
}

// A graph is the list of operations that were captured on one stream.
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    g_capturing = stream_of(s);
    g_capture_from = g_capturing->ops.size();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    Stream* st = stream_of(s);
    g_graphs.emplace_back(new Stream);
    g_graphs.back()->ops.assign(st->ops.begin() + g_capture_from, st->ops.end());
    st->ops.resize(g_capture_from);
    g_capturing = nullptr;
    *g = reinterpret_cast<cudaGraph_t>(g_graphs.back().get());
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
    *x = reinterpret_cast<cudaGraphExec_t>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
    if (fails("cudaGraphLaunch")) return cudaErrorUnknown;
    for (const Op& op : reinterpret_cast<Stream*>(x)->ops) push(stream_of(s), op.run, op.to_host);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

int bh_gpu_fma_peak(int, int, double*) { return BH_ERR_NO_DEVICE; }

}  // extern "C"

// ---- the launch wrappers ----------------------------------------------------------
namespace bhg {

size_t deferred_record_bytes() { return kDeferredRecordBytes; }
int trace_blocks_per_sm(int, int, int) { return 4; }
int trace_registers(int, int variant) { return variant ? 232 : 128; }
int adjoint_block_size() { return 64; }
int adjoint_blocks_per_sm(int) { return 4; }
int reverse_blocks_per_sm() { return 6; }
int shade_blocks(long long pixels, int most) {
    const long long want = (pixels + 127) / 128;
    return (int)(want < 1 ? 1 : (want < most ? want : most));
}

cudaError_t launch_trace(const TraceLaunch& L, cudaStream_t s) {
    if (fails("launch_trace")) return cudaErrorLaunchFailure;
    push(stream_of(s), [L] {
        for (int b = 0; L.band_done && b < L.nbands; ++b) {
            const long long left = L.total_rays - b * L.rays_per_band;
            L.band_done[b] = (unsigned)(left < L.rays_per_band ? left : L.rays_per_band);
        }
    });
    return cudaSuccess;
}
cudaError_t launch_shade(const ShadeLaunch& L, cudaStream_t s) {
    if (fails("launch_shade")) return cudaErrorLaunchFailure;
    push(stream_of(s), [L] {
        for (int f = 0; f < L.nframes; ++f) {
            const FrameParams& F = L.frames[f];
            const long long n = (long long)F.width * F.height, hi = L.pixel_hi < n ? L.pixel_hi : n;
            for (long long p = L.pixel_lo; p < hi; ++p) {      // a launch covers whole rows
                bh_xyz& o = L.pixels[F.pixel_begin + p];
                o.x = o.y = o.z = (double)p;
            }
            L.stats[f].rays += (unsigned long long)(hi - L.pixel_lo) * F.S * F.S;
        }
    });
    return cudaSuccess;
}
cudaError_t launch_reduce(const ReduceLaunch&, cudaStream_t) {
    return fails("launch_reduce") ? cudaErrorLaunchFailure : cudaSuccess;
}
cudaError_t launch_display(const DisplayLaunch& L, cudaStream_t s) {
    if (fails("launch_display")) return cudaErrorLaunchFailure;
    push(stream_of(s), [L] {
        for (int i = 0; i < L.n && L.develop; ++i)
            std::memset(L.frames[i].rgb, 1 + L.frames[i].index, (size_t)L.frames[i].width * L.frames[i].height * 3);
    });
    return cudaSuccess;
}
cudaError_t launch_adjoint(const AdjointLaunch&, cudaStream_t) {
    return fails("launch_adjoint") ? cudaErrorLaunchFailure : cudaSuccess;
}
cudaError_t launch_eval_rhs(int, const FrameParams*, const double*, long long, double*, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_eval_shade(int, const FrameParams*, const double*, const double*, long long, double*, cudaStream_t) {
    return cudaSuccess;
}

}  // namespace bhg
