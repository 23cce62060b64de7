// A stand-in for libcudart on a machine without a GPU: device memory is a range of
// addresses that nothing reads, kernels and copies do nothing (copies to the host
// give zeros), and every call is counted.  The library's host code runs on it as it
// does on the real one, so a test can have the n-th call fail, look at what was left
// allocated, and at the shared-memory limits that the launches were given.
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

namespace {
std::map<const void *, size_t> live;
std::map<const void *, int> smem_limit;
long long calls = 0, fail_at = 0;
int lowered = 0, refused = 0, launches = 0;
std::map<const void *, std::string> names;
std::string watched;
int watched_arg = 0;
std::vector<int> seen;
char *next_address = (char *)(1ull << 40);

// The n-th call that can fail (fake_fail_at) does.
cudaError_t step(cudaError_t e) { return ++calls == fail_at ? e : cudaSuccess; }

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local Config config;
}  // namespace

extern "C" {
long long fake_live() { return (long long)live.size(); }
long long fake_calls() { return calls; }
int fake_lowered() { return lowered; }
int fake_refused() { return refused; }
int fake_launches() { return launches; }
// From here on, note the arg-th (an int) of every launch of a kernel named `name`.
void fake_watch(const char *name, int arg) {
    watched = name;
    watched_arg = arg;
    seen.clear();
}
int fake_seen(int i) { return i < (int)seen.size() ? seen[i] : -1; }
void fake_fail_at(long long n) {
    calls = 0;
    fail_at = n;
}

cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t) {
    if (cudaError_t e = step(cudaErrorMemoryAllocation)) return e;
    *p = next_address;
    next_address += (bytes + 511) & ~(size_t)255;
    live[*p] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return live.erase(p) ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaMemcpyAsync(void *d, const void *, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    if (cudaError_t e = step(cudaErrorUnknown)) return e;
    if (kind == cudaMemcpyDeviceToHost) memset(d, 0, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return step(cudaErrorUnknown); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return step(cudaErrorUnknown); }

cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    int &limit = smem_limit[f];
    lowered += v < limit;
    limit = v;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t smem, cudaStream_t) {
    if (!watched.empty() && names[f].find(watched) != std::string::npos) seen.push_back(*(int *)args[watched_arg]);
    const auto i = smem_limit.find(f);
    const size_t limit = i == smem_limit.end() || i->second < 48 * 1024 ? 48 * 1024 : (size_t)i->second;
    ++launches;
    refused += smem > limit;
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    config = {g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
    *g = config.grid;
    *b = config.block;
    *smem = config.smem;
    *(cudaStream_t *)st = config.stream;
    return cudaSuccess;
}

cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount            ? 148
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448
         : a == cudaDevAttrComputeCapabilityMajor       ? 10
         : a == cudaDevAttrComputeCapabilityMinor       ? 0
                                                        : 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = next_address, cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void *d, const void *, size_t n, size_t, cudaMemcpyKind) {
    memset(d, 0, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    return *s = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *) {
    names[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
