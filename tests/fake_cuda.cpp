// A CUDA runtime on host memory for tests of the host code (api.cpp,
// engine.cpp, server.cpp) without a GPU: two devices, allocations that
// remember the device current when they were made, copies that run at once,
// launches that only write down what they were given, and calls that fail on
// request.  Linked with those sources in place of the runtime and the kernels
// (tests/fake_cuda.py).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "kernels.hpp"
#include "rvsb.h"

namespace {

constexpr int kDevices = 2;
thread_local int t_device = 0;
thread_local cudaError_t t_last = cudaSuccess;

struct Block {
    size_t bytes;
    int device;
};
std::mutex g_mu;
std::map<char*, Block> g_blocks;
std::map<cudaStream_t, int> g_pending;  // copies issued since the stream was last waited for
std::string g_fail_call;
int g_fail_after = -1;

const Block* block_of(const void* p) {
    auto it = g_blocks.upper_bound(const_cast<char*>(static_cast<const char*>(p)));
    if (it == g_blocks.begin()) return nullptr;
    --it;
    return static_cast<const char*>(p) < it->first + it->second.bytes ? &it->second : nullptr;
}

// Whether `bytes` from `p` on lie in one allocation.
bool backed(const void* p, size_t bytes) {
    auto it = g_blocks.upper_bound(const_cast<char*>(static_cast<const char*>(p)));
    if (it == g_blocks.begin()) return false;
    --it;
    return static_cast<const char*>(p) + bytes <= it->first + it->second.bytes;
}

// The error of the call `name` where the test asked for one.
cudaError_t result(const char* name) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (g_fail_after < 0 || g_fail_call != name || g_fail_after-- > 0) return cudaSuccess;
    return t_last = cudaErrorUnknown;
}

}  // namespace

extern "C" {

// What one launch_batch got (its first slot's table).
struct FakeLaunch {
    int device, out_device, slots, variant, small, views, decodes_before, decodes_at_resolve;
    float precision;
    int unbacked;  // workspace buffers without an allocation of their size behind them
};

}  // extern "C"

namespace {

std::vector<FakeLaunch> g_launches;
int g_decodes = 0;

}  // namespace

extern "C" {

void fake_reset() {
    std::lock_guard<std::mutex> lock(g_mu);
    g_launches.clear();
    g_decodes = 0;
    g_pending.clear();
    g_fail_after = -1;
}
void fake_fail(const char* call, int after) {
    std::lock_guard<std::mutex> lock(g_mu);
    g_fail_call = call;
    g_fail_after = after;
}
int fake_pending_copies() {
    std::lock_guard<std::mutex> lock(g_mu);
    int n = 0;
    for (const auto& p : g_pending) n += p.second;
    return n;
}
int fake_launches() { return (int)g_launches.size(); }
void fake_launch(int k, FakeLaunch* out) { *out = g_launches[k]; }
int fake_device() { return t_device; }
void fake_set_device(int d) { t_device = d; }

// --- runtime -----------------------------------------------------------------

cudaError_t cudaGetDeviceCount(int* n) {
    *n = kDevices;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    t_device = d;
    return result("cudaSetDevice");
}
cudaError_t cudaMalloc(void** p, size_t n) {
    const cudaError_t e = result("cudaMalloc");
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_mu);
    *p = std::calloc(n, 1);
    g_blocks[static_cast<char*>(*p)] = Block{n, t_device};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lock(g_mu);
    g_blocks.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = std::calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return result("cudaMemcpy");
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t stream) {
    const cudaError_t e = result("cudaMemcpyAsync");
    if (e != cudaSuccess) return e;
    std::memcpy(d, s, n);
    std::lock_guard<std::mutex> lock(g_mu);
    ++g_pending[stream];
    return e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    const cudaError_t e = result("cudaStreamSynchronize");
    std::lock_guard<std::mutex> lock(g_mu);
    g_pending[s] = 0;
    return e;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return result("cudaStreamWaitEvent"); }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return result("cudaEventRecord"); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaPeekAtLastError() { return t_last; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = t_last;
    t_last = cudaSuccess;
    return e;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

rvsb_status rvsb_inpaint_sources_noalloc(const uint8_t*, int, int, int32_t*, void*, char*, size_t) {
    return RVSB_E_UNSUPPORTED;
}

}  // extern "C"

// --- kernels -----------------------------------------------------------------

namespace rvsb {

size_t inpaint_sum_words(int wo, int ho) { return (size_t)3 * ((ho + 31) / 32) * wo; }

// What the kernels of a slot write beside its outputs.
static int unbacked_buffers(const SlotTable& t) {
    const size_t n = (size_t)t.t.wo * t.t.ho;
    int bad = 0;
    auto need = [&](const void* p, size_t bytes) { bad += !backed(p, bytes); };
    need(t.b.status, sizeof(DevStatus));
    // and the huge triangles after it
    need(t.b.large, sizeof(uint4) * (size_t)t.b.large_capacity + 8 * (size_t)t.b.huge_capacity);
    need(t.b.codes, 8 * n);
    need(t.b.holes, 4 * (size_t)((t.t.wo + 31) / 32) * t.t.ho);
    for (const uint64_t* p : t.b.scan) need(p, 8 * n);
    need(t.b.inpaint_sum, 8 * inpaint_sum_words(t.t.wo, t.t.ho));
    for (int v = 0; v < t.t.n_views; ++v) {
        need(t.v[v].vert, sizeof(float4) * (size_t)t.v[v].w * t.v[v].h);
        need(t.v[v].z, 8 * n);
    }
    if (t.t.rescale) {
        need(t.b.pcolor, sizeof(float4) * n);
        need(t.b.psrc, 8 * n);
    }
    if (t.aux.on) {
        need(t.aux.acc_depth, 4 * n);
        need(t.aux.acc_valid, 4 * n);
    }
    if (t.ms.on) {
        need(t.ms.yq, 8 * n * t.t.n_views);
        need(t.ms.uv, 8 * n * t.t.n_views);
        need(t.ms.hsum, 8 * n * t.t.n_views);
        need(t.ms.hcnt, 4 * n * t.t.n_views);
        need(t.ms.blur, 4 * n * t.t.n_views);
    }
    return bad;
}

template <class Tabs>
int launch_batch(const Tabs& tabs, const BatchShape& sh, cudaStream_t, cudaEvent_t*,
                 const std::function<void()>& before_resolve) {
    const SlotTable& t = tabs.at(0);
    FakeLaunch f{};
    f.device = t_device;
    const Block* b = block_of(t.out_y);
    f.out_device = b ? b->device : -1;
    f.slots = sh.slots;
    f.variant = sh.variant;
    f.small = t.t.small;
    f.views = t.t.n_views;
    f.precision = t.t.precision;
    for (int k = 0; k < sh.slots; ++k) f.unbacked += unbacked_buffers(tabs.at(k));
    f.decodes_before = g_decodes;
    if (before_resolve) before_resolve();
    f.decodes_at_resolve = g_decodes;
    g_launches.push_back(f);
    return cudaPeekAtLastError() == cudaSuccess ? 10 : -1;
}
template int launch_batch<TableParam>(const TableParam&, const BatchShape&, cudaStream_t, cudaEvent_t*,
                                      const std::function<void()>&);
template int launch_batch<TablePtr>(const TablePtr&, const BatchShape&, cudaStream_t, cudaEvent_t*,
                                    const std::function<void()>&);

void launch_decode_color(const uint16_t*, const uint16_t*, const uint16_t*, int, int, uint64_t*, cudaStream_t) {
    ++g_decodes;
}
void launch_decode_views(const DecodeJobs&, int n, int, int, cudaStream_t) { g_decodes += n; }
void launch_depth_lut(float, float, float, int, float, float, float4*, cudaStream_t) {}
void launch_tile_depth(const TileDepthJobs&, int, int, int, cudaStream_t) {}
void prepare_ms_kernels(int) {}

}  // namespace rvsb
