// fake_cudart.h -- a stand-in for the CUDA runtime, for tests of host code on
// the CPU: memory is host memory, copies are done at once, kernels do not run,
// time is a counter that the test advances, and each launch's grid is noted.
// Linked in place of the runtime with objects that nvcc compiled.
#pragma once

#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace fake {
struct Launch {
    dim3 grid, block;
    size_t smem;
};
inline std::vector<Launch> launches;
inline double clock_ms = 0.0;
inline int captured = -1;                     // steps captured so far; -1: no capture
inline cudaError_t (*graph_launch)(long) = nullptr;  // a graph of that many captured steps
inline int resident = 4;                      // blocks per SM that the occupancy call answers

// the kernels' (mangled) names, and what a test does in a kernel's place
inline std::map<const void *, std::string> &names()
{
    static std::map<const void *, std::string> m;
    return m;
}
inline void (*on_kernel)(const std::string &name, void **args) = nullptr;

// buffers that count as a caller's device memory, and the copies from and to them
struct Range {
    char *base;
    size_t size;
};
inline std::vector<Range> device;
inline long device_copies = 0;
inline Range *holding(const void *p)
{
    for (Range &r : device)
        if (p >= r.base && p < r.base + r.size) return &r;
    return nullptr;
}
// As the runtime's copy checks: both ends inside their allocation.
inline bool copies(const void *p, size_t n)
{
    Range *r = holding(p);
    if (!r) return true;
    ++device_copies;
    return n <= size_t(r->base + r->size - static_cast<const char *>(p));
}
inline CUresult address_range(CUdeviceptr *base, size_t *size, CUdeviceptr p)
{
    Range *r = holding(reinterpret_cast<void *>(p));
    if (!r) return CUDA_ERROR_NOT_FOUND;
    *base = reinterpret_cast<CUdeviceptr>(r->base), *size = r->size;
    return CUDA_SUCCESS;
}

// As the runtime's launch checks: the grid's limits.
inline cudaError_t note(dim3 grid, dim3 block, size_t smem)
{
    if (grid.x < 1 || grid.x > 2147483647u || grid.y < 1 || grid.y > 65535u || grid.z < 1 || grid.z > 65535u)
        return cudaErrorInvalidConfiguration;
    launches.push_back({grid, block, smem});
    return cudaSuccess;
}
} // namespace fake

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::calloc(n ? n : 1, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (!fake::copies(d, n) || !fake::copies(s, n)) return cudaErrorInvalidValue;
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    std::memset(a, 0, sizeof *a);
    if (fake::holding(p)) a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *found)
{
    const bool known = !std::strcmp(name, "cuMemGetAddressRange");
    *f = known ? reinterpret_cast<void *>(fake::address_range) : nullptr;
    *found = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = size_t(1) << 33; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new double(0)); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { fake::captured = 0; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    *g = reinterpret_cast<cudaGraph_t>(long(fake::captured));
    fake::captured = -1;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long) { *e = reinterpret_cast<cudaGraphExec_t>(g); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) { return fake::graph_launch(reinterpret_cast<long>(e)); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(new double(0)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<double *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { *reinterpret_cast<double *>(e) = fake::clock_ms; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b)
{
    *ms = float(*reinterpret_cast<double *>(b) - *reinterpret_cast<double *>(a));
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = fake::resident;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t m, cudaStream_t)
{
    if (cudaError_t e = fake::note(g, b, m)) return e;
    if (fake::on_kernel) fake::on_kernel(fake::names()[f], args);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **)
{
    return fake::note(c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
// what nvcc's host stubs call
static struct { dim3 g, b; size_t m; void *s; } fake_config;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void *s) { fake_config = {g, b, m, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s)
{
    *g = fake_config.g, *b = fake_config.b, *m = fake_config.m, *static_cast<void **>(s) = fake_config.s;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *)
{
    fake::names()[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
} // extern "C"
