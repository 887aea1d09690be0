// fake_cuda.cpp — a CUDA runtime and kernel launchers made of host memory, linked with
// the library's host runtime (csrc/engine.cu) so that its handling of streams, page-locked
// memory and failing calls is tested without a GPU.
//
// Work put on a stream stays pending until something waits for it, as on a device: copies
// from or to page-locked memory read and write it only then; a copy to ordinary memory
// waits for its stream, a copy from ordinary memory takes the bytes at once.  Kernels
// do nothing (device memory starts as zeros).  A call can be made to fail.
#include <cuda_runtime.h>
#include <cuda.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "kernels.h"

namespace {

struct Op {
    cudaStream_t stream;
    bool host_write;
    std::function<void()> run;
};
std::vector<Op> g_ops;
std::map<char *, size_t> g_pinned;
std::map<std::string, int> g_fail;  // call -> how many calls from now fail (1: the next)
uint64_t g_pinned_bytes = 0, g_event = 0;
float g_ms = 1000.0f;

bool fails(const char *fn) {
    auto it = g_fail.find(fn);
    if (it == g_fail.end() || --it->second > 0) return false;
    g_fail.erase(it);
    return true;
}
void drain(cudaStream_t s, bool all = false) {
    for (size_t i = 0; i < g_ops.size();) {
        if (!all && g_ops[i].stream != s) {
            ++i;
            continue;
        }
        Op op = std::move(g_ops[i]);
        g_ops.erase(g_ops.begin() + (ptrdiff_t)i);
        op.run();
    }
}
bool pinned(const void *p) {
    auto it = g_pinned.upper_bound((char *)p);
    if (it == g_pinned.begin()) return false;
    --it;
    return (char *)p < it->first + it->second;
}

}  // namespace

extern "C" {
// ---- what a test controls and asks -------------------------------------------
void fake_fail(const char *call, int nth) { g_fail[call] = nth; }
int fake_pending_host_writes() {
    int n = 0;
    for (const Op &o : g_ops) n += o.host_write;
    return n;
}
uint64_t fake_pinned_bytes() { return g_pinned_bytes; }
void *__real_malloc(size_t);
void *__wrap_malloc(size_t n) { return fails("malloc") ? nullptr : __real_malloc(n); }

// ---- runtime -----------------------------------------------------------------
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof(*p));
    p->major = 10;
    p->multiProcessorCount = 148;
    p->sharedMemPerBlockOptin = 227u << 10;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = 180ull << 30, cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
    if (fails("cudaMalloc")) return cudaErrorMemoryAllocation;
    return (*p = std::calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) { return drain(nullptr, true), std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (fails("cudaHostAlloc")) return cudaErrorMemoryAllocation;
    *p = std::calloc(n, 1);
    g_pinned[(char *)*p] = n;
    g_pinned_bytes += n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    drain(nullptr, true);
    g_pinned_bytes -= g_pinned[(char *)p];
    g_pinned.erase((char *)p);
    return std::free(p), cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::memset(a, 0, sizeof(*a));
    a->type = pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    a->devicePointer = pinned(p) ? const_cast<void *>(p) : nullptr;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    if (fails(k == cudaMemcpyDeviceToHost ? "copy to host" : "copy to device")) return cudaErrorUnknown;
    if (k == cudaMemcpyDeviceToHost) {
        g_ops.push_back({st, true, [=] { std::memcpy(d, s, n); }});
        if (!pinned(d)) drain(st);
    } else if (k == cudaMemcpyHostToDevice && !pinned(s)) {
        std::vector<char> b((const char *)s, (const char *)s + n);
        g_ops.push_back({st, false, [d, b] { std::memcpy(d, b.data(), b.size()); }});
    } else {
        g_ops.push_back({st, false, [=] { std::memcpy(d, s, n); }});
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
    drain(nullptr, true);
    if (fails(k == cudaMemcpyDeviceToHost ? "copy to host" : "copy to device")) return cudaErrorUnknown;
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    g_ops.push_back({st, false, [=] { std::memset(d, v, n); }});
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    return *s = (cudaStream_t)std::malloc(1), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drain(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return drain(s), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaLaunchHostFunc(cudaStream_t st, cudaHostFn_t fn, void *u) {
    g_ops.push_back({st, false, [=] { fn(u); }});
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)++g_event, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
// each timing is shorter than the one before: an autotuner takes its last candidate
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = g_ms *= 0.99f, cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorUnknown; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorUnknown; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorUnknown; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
static CUresult fake_encode(...) { return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **f, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *f = (void *)fake_encode;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}  // extern "C"

// ---- launchers ---------------------------------------------------------------
namespace mrc {
cudaError_t occupancy_launch(const OccupancyArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t snapshot_launch(const SnapshotArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t overuse_launch(const OveruseArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t dirty_launch(const DirtyArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t group_overuse_launch(const GroupArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t halo_launch(const HaloArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t emit_launch(const EmitArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t footprint_reduce(const unsigned long long *, const uint32_t *, unsigned long long *, uint32_t *,
                             unsigned long long *, uint32_t *, uint32_t *, uint64_t, int, void *, size_t *b, cudaStream_t) {
    return *b = 16, cudaSuccess;
}
cudaError_t override_launch(const OverrideArgs &, cudaStream_t) { return cudaSuccess; }
uint32_t warp_relax_threads() { return 128; }
cudaError_t warp_relax_occupancy(int *n) { return *n = 1, cudaSuccess; }
cudaError_t warp_relax_launch(const RelaxArgs &, uint32_t, cudaStream_t) { return cudaSuccess; }
uint64_t planes_chunks(uint32_t, uint32_t, uint32_t) { return 1; }
cudaError_t planes_launch(const DevBoard *, const uint64_t *, uint32_t, uint64_t, uint32_t, bool, cudaStream_t) {
    return cudaSuccess;
}
size_t relax_smem_bytes(uint32_t layers, uint32_t tile_h, bool) { return (size_t)layers * tile_h * 1088; }
cudaError_t relax_configure(uint32_t, uint32_t, size_t, bool, bool) { return cudaSuccess; }
cudaError_t relax_occupancy(uint32_t, uint32_t, size_t, int *n, bool, bool) { return *n = 1, cudaSuccess; }
cudaError_t relax_launch(const RelaxArgs &, uint32_t, uint32_t, size_t, cudaStream_t, bool, bool) { return cudaSuccess; }
size_t layer_smem_bytes(uint32_t layers, uint32_t tile_h) { return (size_t)layers * tile_h * 1024; }
cudaError_t layer_configure(uint32_t, uint32_t, size_t, bool, bool, bool, int *n) { return *n = 1, cudaSuccess; }
cudaError_t layer_launch(const RelaxArgs &, uint32_t, size_t, cudaStream_t, bool, bool, bool) { return cudaSuccess; }
cudaError_t mark_over_tiles_launch(const DevField *, uint32_t, const DevBoard *, uint32_t, uint8_t *, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t path_launch(const PathArgs &, cudaStream_t) { return cudaSuccess; }
cudaError_t fields_launch(const PathArgs &, uint32_t *, uint64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t plain_round_launch(const PlainArgs &, uint64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t wait_selftest_launch(Ctl *, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t combine_flags_launch(uint8_t *, const uint8_t *, uint64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t host_gather_launch(const HostSpan *, const uint64_t *, uint32_t, uint64_t, uint32_t, cudaStream_t) {
    return cudaSuccess;
}
uint64_t host_gather_chunks(uint64_t b) { return b / 65536 + 1; }
}  // namespace mrc
