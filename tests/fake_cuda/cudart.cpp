// A CUDA runtime of two devices in host memory, as far as the engine's host
// code uses one.  Copies and launches run at once, a captured graph is the
// list of its launches, freed memory stays unmapped for good, and an access
// to memory that is not a live allocation of the device it runs on is counted
// (fake_faults) and skipped.
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "fake_cuda.h"

namespace {
struct Alloc {
    size_t bytes;
    int dev;
    bool live;
};
struct Graph {
    std::vector<std::function<void()>> launches;
};
std::mutex g_mu;
std::map<const char *, Alloc> g_allocs;
int g_faults = 0, g_execs = 0;
thread_local int t_dev = 0;
thread_local Graph *t_capture = nullptr;

// the allocation that p lies in, or null (host memory)
const Alloc *alloc_of(const void *p, size_t *left) {
    auto it = g_allocs.upper_bound((const char *)p);
    if (it == g_allocs.begin()) return nullptr;
    --it;
    const size_t at = (size_t)((const char *)p - it->first);
    if (at >= it->second.bytes) return nullptr;
    *left = it->second.bytes - at;
    return &it->second;
}
bool host_or_live(const void *p, size_t bytes) {
    std::lock_guard<std::mutex> lk(g_mu);
    size_t left = 0;
    const Alloc *a = alloc_of(p, &left);
    const bool ok = !a || (a->live && bytes <= left);
    g_faults += !ok;
    return ok;
}
cudaError_t copy(void *d, const void *s, size_t n) {
    if (n && host_or_live(d, n) && host_or_live(s, n)) memcpy(d, s, n);
    return cudaSuccess;
}
}  // namespace

int fake_stream_device(cudaStream_t s) { return *(int *)s; }
bool fake_access(const void *p, size_t bytes, int dev) {
    std::lock_guard<std::mutex> lk(g_mu);
    size_t left = 0;
    const Alloc *a = alloc_of(p, &left);
    const bool ok = a && a->live && a->dev == dev && bytes <= left;
    g_faults += !ok;
    return ok;
}
void fake_launch(std::function<void()> kernel) {
    if (t_capture) t_capture->launches.push_back(kernel);
    else kernel();
}

extern "C" {
int fake_faults() { return g_faults; }
int fake_live_execs() { return g_execs; }
size_t fake_live_bytes() {
    std::lock_guard<std::mutex> lk(g_mu);
    size_t n = 0;
    for (auto &a : g_allocs) n += a.second.live ? a.second.bytes : 0;
    return n;
}

cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_dev = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = t_dev; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    strcpy(p->name, "host memory");
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = *hi = 0; return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t bytes) {
    *p = aligned_alloc(256, (bytes + 511) / 256 * 256);
    if (!*p) return cudaErrorMemoryAllocation;
    std::lock_guard<std::mutex> lk(g_mu);
    g_allocs[(const char *)*p] = Alloc{bytes, t_dev, true};
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_allocs.find((const char *)p);
    if (it != g_allocs.end()) it->second.live = false;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) { *p = malloc(bytes); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { return copy(d, s, n); }
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t i = 0; i < h; i++) copy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    if (n && host_or_live(p, n)) memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t) new int(t_dev); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete (int *)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t) new int(0); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (int *)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    t_capture = new Graph;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    *g = (cudaGraph_t)t_capture;
    t_capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
    *x = (cudaGraphExec_t) new Graph(*(Graph *)g);
    g_execs++;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph *)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    delete (Graph *)x;
    g_execs--;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    for (auto &k : ((Graph *)x)->launches) k();
    return cudaSuccess;
}

cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidSymbol; }

// registration hooks and launch stubs of nvcc's host code
void *__cudaRegisterFatBinary() { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd() {}
void __cudaUnregisterFatBinary() {}
void __cudaRegisterVar() {}
void __cudaRegisterFunction() {}
int __cudaGetKernel() { return cudaErrorUnknown; }
int __cudaLaunchKernel() { return cudaErrorUnknown; }
int __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
}
