// A fake of the CUDA runtime calls the library makes, on host memory, for
// tests of its error paths without a GPU (tests/test_cuda_failures_host.py
// links the library's objects against it).  Kernels are registered and counted
// but not run; memory is zeroed host memory.  A chosen launch or allocation
// fails with the runtime's own code and sets the thread's last error.
//
//   fake_fail_launch(n)   the n-th launch from now on fails (0: none)
//   fake_fail_malloc(n)   the n-th allocation from now on fails (0: none)
//   fake_launches() / fake_mallocs()   so far
//   fake_device_word(v)   4-byte reads of device memory give v (0: what it holds): the flags a step polls
//   fake_null_uses()      copies from or to, downloads into, and key scans of a null pointer
//   fake_launched(name)   launches of kernels whose name contains `name`
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string>& names()
{
    static std::map<const void*, std::string> m;
    return m;
}
std::map<std::string, int> launched;
unsigned device_word = 0;
int fail_launch = 0, fail_malloc = 0, launches = 0, mallocs = 0, null_uses = 0;
cudaError_t last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t st;
} config;

cudaError_t fail(cudaError_t e) { return last = e; }
cudaError_t launch(const void* f, void** args)
{
    ++launches;
    const std::string& n = names()[f];
    if (fail_launch > 0 && --fail_launch == 0) return fail(cudaErrorLaunchOutOfResources);
    ++launched[n];
    // k_scan_tiles(nkeys, count, starts, tile_sums); k_download(n, v4, s, id, cell, g, h, kind, out)
    if (n.find("k_scan_tiles") != std::string::npos)
        for (int k = 1; k < 4; ++k) null_uses += !*(void**)args[k];
    if (n.find("k_download") != std::string::npos && !*(void**)args[8]) ++null_uses;
    return cudaSuccess;
}
cudaError_t copy(void* d, const void* s, size_t n)
{
    if (n && (!d || !s)) {
        ++null_uses;
        return fail(cudaErrorInvalidValue);
    }
    if (n) std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t take(void** p, size_t n)
{
    *p = std::calloc(n ? n : 1, 1);
    return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
}  // namespace

extern "C" {
void fake_fail_launch(int n) { fail_launch = n; }
void fake_fail_malloc(int n) { fail_malloc = n; }
void fake_device_word(unsigned v) { device_word = v; }
int fake_launches() { return launches; }
int fake_mallocs() { return mallocs; }
int fake_null_uses() { return null_uses; }
int fake_launched(const char* part)
{
    int k = 0;
    for (const auto& q : launched)
        if (q.first.find(part) != std::string::npos) k += q.second;
    return k;
}

// ---- what nvcc's host code calls --------------------------------------------
void** __cudaRegisterFatBinary(void*)
{
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names()[f] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st)
{
    config = Config{grid, block, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st)
{
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(cudaStream_t*)st = config.st;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t, cudaStream_t) { return launch(k, args); }

// ---- the runtime ---------------------------------------------------------------
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { return launch(f, args); }
cudaError_t cudaMalloc(void** p, size_t n)
{
    ++mallocs;
    if (fail_malloc > 0 && --fail_malloc == 0) return fail(cudaErrorMemoryAllocation);
    return take(p, n);
}
cudaError_t cudaFree(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFreeHost(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    if (device_word && n == 4 && kind == cudaMemcpyDeviceToHost && d && s) return copy(d, &device_word, 4);
    return copy(d, s, n);
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t)
{
    if (!d) return copy(d, d, n);
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaSuccess ? "no error" : "launch failed"; }
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int)
{
    std::memset(p, 0, sizeof *p);
    std::strcpy(p->name, "fake");
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int)
{
    *v = 152;  // multiprocessors
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return take(p, 4u << 20); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return take((void**)s, 1); }
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return take((void**)e, 1); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return take((void**)e, 1); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 0.f;
    return cudaSuccess;
}
// graphs: not faked
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return fail(cudaErrorNotSupported); }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                          cudaStreamCaptureMode)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return fail(cudaErrorNotSupported); }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus*, unsigned long long*, cudaGraph_t*, const cudaGraphNode_t**,
                                     const cudaGraphEdgeData**, size_t*)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, unsigned)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, cudaGraphNodeParams*)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned)
{
    return fail(cudaErrorNotSupported);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
