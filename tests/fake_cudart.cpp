// fake_cudart.cpp -- a CUDA runtime without a GPU, for tests of the library's
// host code: device memory is host memory (filled with 0xa5), copies are
// memcpy, kernels do nothing. The k-th allocation from fake_fail_at(k) on fails.
// Launches of the re-sampling builder's scans (k_r_scan) are checked: their
// workspaces must be live allocations, their flags cleared once.
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

#include <cuda_runtime.h>

namespace {
struct Block {
    size_t bytes;
    bool cleared;
};
std::map<char *, Block> g_live;
std::map<const void *, std::string> g_name;
size_t g_bytes = 0;
long g_fail = 0, g_allocs = 0, g_bad = 0, g_scans = 0;
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;

cudaError_t take(void **p, size_t n) {
    g_allocs++;
    *p = nullptr;
    if (g_fail && --g_fail == 0) return cudaErrorMemoryAllocation;
    char *q = static_cast<char *>(malloc(n ? n : 1));
    memset(q, 0xa5, n);
    g_live[q] = Block{n, false};
    g_bytes += n;
    *p = q;
    return cudaSuccess;
}
cudaError_t give(void *p) {
    auto it = g_live.find(static_cast<char *>(p));
    if (it == g_live.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    g_bytes -= it->second.bytes;
    g_live.erase(it);
    free(p);
    return cudaSuccess;
}
const Block *block_of(const void *p) {
    auto it = g_live.find(static_cast<char *>(const_cast<void *>(p)));
    return it == g_live.end() ? nullptr : &it->second;
}
cudaError_t launched(const void *f, size_t ctas, void **args) {
    if (g_name[f].find("k_r_scan") == std::string::npos) return cudaSuccess;
    g_scans++;
    // ScanPtrs: flags, ticket, err, aggs, incls; a CTA has a tile at least
    void *const *sp = static_cast<void *const *>(args[1]);
    const Block *flags = block_of(sp[0]), *aggs = block_of(sp[3]), *incls = block_of(sp[4]);
    if (!flags || !flags->cleared || !aggs || !incls || flags->bytes < 4 * ctas || aggs->bytes < 16 * ctas ||
        incls->bytes < 16 * ctas)
        g_bad++;
    return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_fail_at(long k) { g_fail = k; }
long fake_allocs() { return g_allocs; }
long fake_bad_launches() { return g_bad; }
long fake_scan_launches() { return g_scans; }
size_t fake_live_bytes() { return g_bytes; }

void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    g_name[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
    g_grid = g;
    g_block = b;
    g_smem = s;
    g_stream = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
    *g = g_grid;
    *b = g_block;
    *s = g_smem;
    *static_cast<cudaStream_t *>(st) = g_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **args, size_t, cudaStream_t) {
    return launched(f, g.x, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    return launched(f, c->gridDim.x, args);
}
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return take(p, n); }
cudaError_t cudaFreeHost(void *p) { return give(p); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    memset(p, v, n);
    auto it = g_live.find(static_cast<char *>(p));
    if (it != g_live.end() && v == 0 && n == it->second.bytes) it->second.cleared = true;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.0f;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    memset(a, 0, sizeof *a);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *, size_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
}
