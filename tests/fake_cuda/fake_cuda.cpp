// The CUDA runtime calls and kernel launches that the C ABI's host code
// (csrc/grt_api.cu, grt_host.cpp) makes, on host memory and without a GPU:
// "device" memory is malloc'd and counted against a limit, copies are checked
// against the allocations they touch, launches are only written down.  Tests
// make calls fail here that a GPU cannot be made to fail on purpose.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "grt.h"
#include "grt_kparams.h"
#include "grt_launch.h"

namespace {

std::map<char*, size_t> device, pinned;
size_t limit = 1ull << 34, used = 0;
bool refuse_pinned = false, fail_init = false;
int bad_accesses = 0;
std::string launches;  // one line per launch
std::vector<unsigned> last_order;

// The device allocation that holds p, or device.end().
std::map<char*, size_t>::iterator owner(const void* p) {
    auto it = device.upper_bound(static_cast<char*>(const_cast<void*>(p)));
    if (it == device.begin()) return device.end();
    --it;
    return static_cast<const char*>(p) < it->first + it->second ? it : device.end();
}

bool on_device(const void* p) { return owner(p) != device.end(); }

bool within(const void* p, size_t n) {
    const auto it = owner(p);
    return it == device.end() || static_cast<const char*>(p) + n <= it->first + it->second;
}

cudaError_t copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
    if ((kind == cudaMemcpyDeviceToHost && on_device(dst)) || (kind == cudaMemcpyHostToDevice && on_device(src)))
        return cudaErrorInvalidValue;
    if (!within(dst, n) || !within(src, n)) {
        ++bad_accesses;  // counted, not made
        return cudaSuccess;
    }
    std::memcpy(dst, src, n);
    return cudaSuccess;
}

}  // namespace

extern "C" {

void fake_reset(size_t memory) {
    limit = memory;
    refuse_pinned = fail_init = false;
    bad_accesses = 0;
    launches.clear();
    last_order.clear();
}
void fake_limit(size_t memory) { limit = memory; }
size_t fake_used(void) { return used; }
void fake_refuse_pinned(int on) { refuse_pinned = on != 0; }
void fake_fail_init(int on) { fail_init = on != 0; }
int fake_bad_accesses(void) { return bad_accesses; }
const char* fake_launches(void) { return launches.c_str(); }
void fake_clear(void) { launches.clear(); }
void* fake_malloc(size_t n) {
    void* p = nullptr;
    return cudaMalloc(&p, n) == cudaSuccess ? p : nullptr;
}

cudaError_t cudaMalloc(void** p, size_t n) {
    if (used + n > limit) return cudaErrorMemoryAllocation;
    char* q = static_cast<char*>(std::malloc(n ? n : 1));
    if (!q) return cudaErrorMemoryAllocation;
    device[q] = n;
    used += n;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    const auto it = device.find(static_cast<char*>(p));
    if (it == device.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    used -= it->second;
    device.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
    *total = limit;
    *free_bytes = limit > used ? limit - used : 0;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    if (refuse_pinned) return cudaErrorMemoryAllocation;
    char* q = static_cast<char*>(std::malloc(n ? n : 1));
    pinned[q] = n;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    pinned.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return copy(d, s, n, k); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    if (!within(d, n)) ++bad_accesses;
    else std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::memset(a, 0, sizeof(*a));
    a->type = on_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    for (const auto& b : pinned)
        if (p >= b.first && p < b.first + b.second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake CUDA error"; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) {
    launches += "wait\n";
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {  // any handle that is not null
    static size_t events = 0;
    return *e = reinterpret_cast<cudaEvent_t>(++events), cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

// entry points of the library's other files
grt_status grt_measure_fma_peaks(double*, double*) { return GRT_ENODEV; }
grt_status grt_trace_device_noalloc(const grt_params*, const grt_device_grid*, const grt_photon_soa*, uint64_t,
                                    grt_run_stats*, void*, char*, size_t) {
    return GRT_ENODEV;
}

}  // extern "C"

namespace grt {

cudaError_t launch_init_image(const InitImageArgs&, cudaStream_t) {
    launches += "init\n";
    return fail_init ? cudaErrorLaunchFailure : cudaSuccess;
}
// every queue position is its own photon
cudaError_t launch_screen_order(const ScreenOrderArgs& a, cudaStream_t) {
    launches += "screen_order\n";
    for (unsigned long long i = 0; i < a.n; ++i) a.order[i] = static_cast<unsigned>(i);
    return cudaSuccess;
}
// "trace <leg> n=<queue> refill=<threshold> order=<largest entry, - without an order> [hands_on] [resume]"
cudaError_t launch_trace(const KParams& kp, bool, int leg, int, int, int blocks_per_sm, int, size_t, cudaStream_t) {
    std::string order = "-";
    if (kp.order && !kp.resume) {
        unsigned largest = 0;
        if (!within(kp.order, kp.n * sizeof(unsigned))) ++bad_accesses;
        else
            for (unsigned long long i = 0; i < kp.n; ++i) largest = kp.order[i] > largest ? kp.order[i] : largest;
        order = std::to_string(largest);
    }
    launches += "trace " + std::to_string(leg) + " n=" + std::to_string(kp.n) + " refill=" +
                std::to_string(kp.refill_threshold) + " blocks=" + std::to_string(blocks_per_sm) + " order=" + order +
                (kp.stragglers ? " hands_on" : "") + (kp.resume ? " resume" : "") + "\n";
    if (kp.stragglers && !within(kp.stragglers, kp.n * sizeof(unsigned))) ++bad_accesses;
    const size_t cells = static_cast<size_t>(kp.grid.nr) * kp.grid.nth * kp.grid.nph;
    for (const double* m : {kp.m_abs, kp.m_emis})
        if (m && !within(m, cells * sizeof(double))) ++bad_accesses;
    if (kp.m_abs || kp.m_emis) launches += "multipliers\n";
    if (leg != 1) kp.counters->terminated = kp.n;
    return cudaSuccess;
}
cudaError_t launch_generate_pending(const KParams&, int, size_t, cudaStream_t) {
    launches += "generate\n";
    return cudaSuccess;
}
cudaError_t launch_init_disk(const DiskInitArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_image_products(ProductsSet&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_gather_fields(const GatherArgs&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_count_terminated(const uint8_t*, unsigned long long, unsigned long long* out, int, cudaStream_t) {
    *out = 0;
    return cudaSuccess;
}
cudaError_t launch_adjoint_forward(const KParams& kp, const AdjointArgs& aa, int, size_t, cudaStream_t) {
    launches += "forward cap=" + std::to_string(aa.full_cap) + "\n";
    if (aa.full_cap && !within(aa.full, kp.n * aa.full_cap * 6 * sizeof(double))) ++bad_accesses;
    return cudaSuccess;
}
cudaError_t launch_adjoint_sweep(const KParams&, const AdjointArgs& aa, cudaStream_t) {
    launches += aa.full && on_device(aa.full) ? "sweep\n" : "sweep without a record\n";
    return cudaSuccess;
}
cudaError_t launch_adjoint_reverse(const KParams&, const AdjointArgs&, int, size_t, cudaStream_t) {
    launches += "reverse\n";
    return cudaSuccess;
}

}  // namespace grt
