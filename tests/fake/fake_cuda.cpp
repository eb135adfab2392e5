// fake_cuda.cpp - the CUDA runtime functions that the library calls, on host memory,
// so that its host code runs without a GPU: device memory is malloc'ed, copies
// happen at the call, kernels do nothing.  Every call is logged; a named function can be
// made to fail.  The library's objects are linked with this file in the runtime's place
// (tests/test_host_paths_cpu.py).
#include <cuda_runtime_api.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {

std::string g_log, g_fail_name;
int g_fail_in = 0, g_host_pages = 0, g_next = 0;
float g_fast_grid = 0, g_fast_block = 0;
std::map<const void *, size_t> g_pinned;
cudaError_t g_last = cudaSuccess;  // a launch's error, read by cudaGetLastError
struct Config { dim3 grid, block; size_t smem; cudaStream_t stream; } g_config;

void *handle() { return reinterpret_cast<void *>((size_t)(++g_next)); }

// Log one call (and the stream it names); its status.
cudaError_t called(const char *name, const void *stream = nullptr, const std::string &more = "")
{
    g_log += std::string(name) + " " + std::to_string((size_t)stream) + more + "\n";
    if (g_fail_in > 0 && g_fail_name == name && --g_fail_in == 0) return cudaErrorUnknown;
    return cudaSuccess;
}
cudaError_t allocate(const char *name, void **p, size_t bytes)
{
    const cudaError_t e = called(name);
    if (e != cudaSuccess) return e;
    *p = std::calloc(bytes ? bytes : 1, 1);
    return cudaSuccess;
}

}  // namespace

#define FAKE extern "C" __attribute__((visibility("default")))

// ---- control -------------------------------------------------------------------

// Fail the nth call of `name` from now (0: none).
FAKE void fake_fail(const char *name, int nth) { g_fail_name = name; g_fail_in = nth; }
FAKE void fake_host_pages(int on) { g_host_pages = on; }
FAKE void fake_pin(const void *p, size_t bytes, int on)
{
    if (on) g_pinned[p] = bytes;
    else g_pinned.erase(p);
}
FAKE void fake_fastest(int grid, int block) { g_fast_grid = (float)grid; g_fast_block = (float)block; }
// The calls since the last fake_clear, one per line: name, stream, and for a launch its
// grid, block and dynamic shared memory.
FAKE const char *fake_log() { return g_log.c_str(); }
FAKE void fake_clear() { g_log.clear(); }

// ---- memory ----------------------------------------------------------------------

FAKE cudaError_t cudaMalloc(void **p, size_t n) { return allocate("cudaMalloc", p, n); }
FAKE cudaError_t cudaFree(void *p) { std::free(p); return called("cudaFree"); }
FAKE cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    const cudaError_t e = allocate("cudaHostAlloc", p, n);
    if (e == cudaSuccess) g_pinned[*p] = n;
    return e;
}
FAKE cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
FAKE cudaError_t cudaFreeHost(void *p)
{
    g_pinned.erase(p);
    std::free(p);
    return called("cudaFreeHost");
}
FAKE cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    const cudaError_t e = called("cudaMemcpy");
    if (e == cudaSuccess) std::memcpy(d, s, n);
    return e;
}
FAKE cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t q)
{
    const cudaError_t e = called("cudaMemcpyAsync", q);
    if (e == cudaSuccess) std::memcpy(d, s, n);
    return e;
}
FAKE cudaError_t cudaMemset(void *p, int v, size_t n) { std::memset(p, v, n); return called("cudaMemset"); }
FAKE cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t q)
{
    std::memset(p, v, n);
    return called("cudaMemsetAsync", q);
}
FAKE cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = size_t(1) << 36; return cudaSuccess; }
FAKE cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    for (const auto &m : g_pinned)
        if (p >= m.first && p < static_cast<const char *>(m.first) + m.second)
            a->type = cudaMemoryTypeHost;
    return called("cudaPointerGetAttributes");
}
FAKE cudaError_t cudaGetSymbolAddress(void **p, const void *)
{
    static char scratch[4 << 20];
    *p = scratch;
    return called("cudaGetSymbolAddress");
}

// ---- devices, streams, events, graphs ----------------------------------------------

FAKE cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
FAKE cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
FAKE cudaError_t cudaSetDevice(int) { return cudaSuccess; }
FAKE cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
FAKE cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152
         : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? g_host_pages
         : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 228 * 1024
         : a == cudaDevAttrMaxRegistersPerMultiprocessor ? 65536
         : a == cudaDevAttrMaxThreadsPerMultiProcessor ? 2048
         : a == cudaDevAttrMaxBlocksPerMultiprocessor ? 32
         : a == cudaDevAttrReservedSharedMemoryPerBlock ? 1024 : 0;
    return cudaSuccess;
}
FAKE cudaError_t cudaDeviceSynchronize() { return called("cudaDeviceSynchronize"); }
FAKE cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
FAKE const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
FAKE cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = static_cast<cudaStream_t>(handle());
    return called("cudaStreamCreateWithFlags");
}
FAKE cudaError_t cudaStreamDestroy(cudaStream_t s) { return called("cudaStreamDestroy", s); }
FAKE cudaError_t cudaStreamSynchronize(cudaStream_t s) { return called("cudaStreamSynchronize", s); }
FAKE cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned)
{
    return called("cudaStreamWaitEvent", s);
}
FAKE cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = static_cast<cudaEvent_t>(handle());
    return called("cudaEventCreateWithFlags");
}
FAKE cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
FAKE cudaError_t cudaEventDestroy(cudaEvent_t) { return called("cudaEventDestroy"); }
FAKE cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { return called("cudaEventRecord", s); }
FAKE cudaError_t cudaEventSynchronize(cudaEvent_t) { return called("cudaEventSynchronize"); }
FAKE cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
// A launch takes as many ms as its grid and block differ from fake_fastest's.
FAKE cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.0f + std::abs((float)g_config.block.x - g_fast_block) +
          std::abs((float)g_config.grid.x - g_fast_grid);
    return called("cudaEventElapsedTime");
}
FAKE cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorUnknown; }
FAKE cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorUnknown; }
FAKE cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long)
{
    return cudaErrorUnknown;
}
FAKE cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
FAKE cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

// ---- kernels -------------------------------------------------------------------------

FAKE cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
FAKE cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *)
{
    std::memset(a, 0, sizeof *a);
    a->numRegs = 128;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
FAKE cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int,
                                                                        size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}
FAKE cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t)
{
    *n = 4;
    return cudaSuccess;
}
FAKE unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s)
{
    g_config = {grid, block, smem, s};
    return 0;
}
FAKE cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s)
{
    *grid = g_config.grid;
    *block = g_config.block;
    *smem = g_config.smem;
    *static_cast<cudaStream_t *>(s) = g_config.stream;
    return cudaSuccess;
}
FAKE cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
FAKE cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3 grid, dim3 block, void **, size_t smem,
                                    cudaStream_t s)
{
    return g_last = called("launch", s, " " + std::to_string(grid.x) + " " +
                                            std::to_string(block.x) + " " + std::to_string(smem));
}
FAKE void **__cudaRegisterFatBinary(void *) { static void *none; return &none; }
FAKE void __cudaRegisterFatBinaryEnd(void **) {}
FAKE void __cudaUnregisterFatBinary(void **) {}
FAKE void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *,
                                 void *, void *, int *)
{
}
FAKE void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
