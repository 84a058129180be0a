// A CUDA runtime without a device, for tests of the library's host code: every call is written to a log
// and succeeds, unless a test has planned a failure for it; device memory is host memory, copies are
// copies, kernels do not run.  Linked with the compiled library object in place of libcudart.
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <cxxabi.h>
#include <stdint.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

static std::vector<std::string> g_log;
static std::map<std::string, std::map<long, int>> g_plan;  // call -> n-th from now -> error
static std::map<std::string, long> g_calls;
static std::map<const void *, std::string> g_kernels;
static std::map<void *, int> g_ids;  // streams and events by their order of creation
struct HostRange { char *p; size_t n; int access; };
static std::vector<HostRange> g_host;  // pinned ranges
static int g_next = 1;
static cudaError_t g_last = cudaSuccess;
static std::vector<std::pair<cudaStream_t, dim3>> g_push;

static int id_of(const void *p) { return p ? g_ids[(void *)p] : 0; }
// a call that fails by plan has "failed" in front of its name in the log
static cudaError_t call(const char *name, const std::string &what = "") {
    const long n = ++g_calls[name];
    auto it = g_plan.find(name);
    const int error = it != g_plan.end() && it->second.count(n) ? it->second[n] : 0;
    g_log.push_back((error ? "failed " : "") + std::string(name) + (what.empty() ? "" : " " + what));
    if (error) g_last = (cudaError_t)error;
    return (cudaError_t)error;
}
static std::string num(long long x) { return std::to_string(x); }
template <class T> static cudaError_t create(const char *name, T *out) {
    const cudaError_t e = call(name, num(g_next));
    if (e) return e;
    void *p = malloc(8);
    g_ids[p] = g_next++;
    *out = (T)p;
    return e;
}
static const HostRange *range_of(const void *p) {
    for (const HostRange &r : g_host)
        if ((char *)p >= r.p && (char *)p < r.p + r.n) return &r;
    return nullptr;
}

extern "C" {
// ---- for the tests
void fake_reset(void) { g_log.clear(); g_plan.clear(); g_calls.clear(); g_last = cudaSuccess; }
void fake_fail(const char *name, long nth, int error) { g_calls[name] = 0; g_plan[name][nth] = error; }
long fake_log_size(void) { return (long)g_log.size(); }
const char *fake_log_line(long i) { return g_log[i].c_str(); }
void fake_pin(void *p, size_t n, int read_only) {
    g_host.push_back({(char *)p, n, read_only ? CU_MEM_ACCESS_FLAGS_PROT_READ : CU_MEM_ACCESS_FLAGS_PROT_READWRITE});
}
void fake_unpin_all(void) { g_host.clear(); }

// ---- kernels
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    int st = 0;
    char *d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
    g_kernels[(const void *)host] = st == 0 && d ? d : name;
    free(d);
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3, size_t, struct CUstream_st *st) { g_push.push_back({st, grid}); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *, size_t *, void *st) {
    *(cudaStream_t *)st = g_push.back().first;
    *grid = g_push.back().second;
    g_push.pop_back();
    return cudaSuccess;
}
static std::string shape(dim3 g) { return " grid " + num(g.x) + " " + num(g.y) + " " + num(g.z); }
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t st) {
    return call("launch", num(id_of(st)) + " plain " + g_kernels[f] + shape(grid));
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
    bool chained = false;
    for (unsigned i = 0; i < c->numAttrs; i++)
        chained = chained || (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                              c->attrs[i].val.programmaticStreamSerializationAllowed);
    return call("launch", num(id_of(c->stream)) + (chained ? " chained " : " plain ") + g_kernels[f] + shape(c->gridDim));
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) { return call("cudaFuncSetAttribute", num(a) + " " + num(v) + " " + g_kernels[f]); }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) { memset(a, 0, sizeof *a); return call("cudaFuncGetAttributes"); }

// ---- devices, errors
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 232448; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return call("cudaDeviceSynchronize"); }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorName(cudaError_t) { return "fake error"; }
const char *cudaGetErrorString(cudaError_t) { return "planned by the test"; }

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n) {
    const cudaError_t e = call("cudaMalloc", num((long long)n));
    *p = e ? nullptr : calloc(1, n ? n : 1);
    return e;
}
cudaError_t cudaFree(void *p) { free(p); return call("cudaFree"); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    const cudaError_t e = call("cudaHostAlloc", num((long long)n));
    *p = e ? nullptr : aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    if (!e) g_host.push_back({(char *)*p, n, CU_MEM_ACCESS_FLAGS_PROT_READWRITE});
    return e;
}
cudaError_t cudaFreeHost(void *p) {
    for (size_t i = 0; i < g_host.size(); i++)
        if (g_host[i].p == p) { g_host.erase(g_host.begin() + i); break; }
    free(p);
    return call("cudaFreeHost");
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return call("cudaHostGetDevicePointer"); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    a->type = range_of(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    a->hostPointer = a->devicePointer = range_of(p) ? (void *)p : nullptr;
    return call("cudaPointerGetAttributes");
}
// as the driver: an address it does not know gives zeros and no error
static CUresult fake_attributes(unsigned n, CUpointer_attribute *at, void **out, CUdeviceptr p) {
    const HostRange *r = range_of((const void *)p);
    call("cuPointerGetAttributes");
    for (unsigned i = 0; i < n && r; i++) {
        unsigned long long v = 0;
        size_t bytes = sizeof v;
        switch (at[i]) {
            case CU_POINTER_ATTRIBUTE_MEMORY_TYPE: v = CU_MEMORYTYPE_HOST; bytes = 4; break;
            case CU_POINTER_ATTRIBUTE_IS_MANAGED: bytes = 4; break;
            case CU_POINTER_ATTRIBUTE_DEVICE_POINTER: v = p; break;
            case CU_POINTER_ATTRIBUTE_RANGE_START_ADDR: v = (uintptr_t)r->p; break;
            case CU_POINTER_ATTRIBUTE_RANGE_SIZE: v = r->n; break;
            case CU_POINTER_ATTRIBUTE_ACCESS_FLAGS: v = r->access; break;
            default: return CUDA_ERROR_INVALID_VALUE;
        }
        memcpy(out[i], &v, bytes);
    }
    return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *) {
    *f = strcmp(name, "cuPointerGetAttributes") == 0 ? (void *)fake_attributes : nullptr;
    return *f ? cudaSuccess : cudaErrorSymbolNotFound;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return call("cudaMemcpy"); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    const cudaError_t e = call("cudaMemcpyAsync", num(id_of(st)) + " " + num((long long)n));
    if (!e) memcpy(d, s, n);
    return e;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return call("cudaMemcpyToSymbol"); }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static char mem[1 << 20]; *p = mem; return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return call("cudaMemset"); }
// not written: fresh memory is zero already, and the pages of large arrays stay untouched
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return call("cudaMemsetAsync"); }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return create("cudaStreamCreate", s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { const int i = id_of(s); free(s); g_ids.erase(s); return call("cudaStreamDestroy", num(i)); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return call("cudaStreamSynchronize", num(id_of(s))); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return call("cudaStreamWaitEvent", num(id_of(s)) + " " + num(id_of(e))); }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) { *c = cudaStreamCaptureStatusNone; return call("cudaStreamIsCapturing"); }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return call("cudaStreamBeginCapture"); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = nullptr; return call("cudaStreamEndCapture"); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return create("cudaEventCreate", e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return create("cudaEventCreate", e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { const int i = id_of(e); free(e); g_ids.erase(e); return call("cudaEventDestroy", num(i)); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return call("cudaEventRecord", num(id_of(e)) + " " + num(id_of(s))); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return call("cudaEventSynchronize", num(id_of(e))); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) { *g = nullptr; return call("cudaGraphInstantiate"); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return call("cudaGraphLaunch"); }
}
