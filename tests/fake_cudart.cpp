// A CUDA runtime that launches nothing, for CPU tests of the host side: device memory is host
// memory out of a settable budget, kernels have a settable register count, every launch succeeds.
// Linked with the library's own objects in place of libcudart.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

namespace {
std::mutex mu;
std::map<void *, size_t> blocks;
size_t used = 0, peak = 0, budget = (size_t)1 << 40;
int regs = 96, waits = 0;
cudaError_t last = cudaSuccess;

cudaError_t fail(cudaError_t e)
{
    last = e;
    return e;
}

cudaError_t take(void **p, size_t n)
{
    std::lock_guard<std::mutex> l(mu);
    n = (n + 511) & ~(size_t)511;
    if (n > budget - used || !(*p = std::aligned_alloc(512, n))) return fail(cudaErrorMemoryAllocation);
    blocks[*p] = n;
    used += n;
    peak = used > peak ? used : peak;
    return cudaSuccess;
}

cudaError_t give(void *p)
{
    std::lock_guard<std::mutex> l(mu);
    if (!p) return cudaSuccess;
    auto f = blocks.find(p);
    if (f == blocks.end()) return fail(cudaErrorInvalidValue);
    used -= f->second;
    blocks.erase(f);
    std::free(p);
    return cudaSuccess;
}

CUresult tensor_map() { return CUDA_SUCCESS; }
int handle;
}  // namespace

extern "C" {
void fake_budget(size_t n) { budget = n; }
void fake_registers(int n) { regs = n; }
int fake_waits()
{
    const int n = waits;
    waits = 0;
    return n;
}
size_t fake_used() { return used; }
size_t fake_peak()
{
    const size_t p = peak;
    peak = used;
    return p;
}

cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return give(p); }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }

cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    p->sharedMemPerBlockOptin = 232448;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "error of the stand-in runtime"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return *p = const_cast<void *>(s), cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned, unsigned long long, cudaDriverEntryPointQueryResult *q)
{
    *f = reinterpret_cast<void *>(&tensor_map);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = reinterpret_cast<cudaStream_t>(&handle), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return waits++, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = reinterpret_cast<cudaEvent_t>(&handle), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { return *t = 0.f, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }

cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *)
{
    std::memset(a, 0, sizeof *a);
    a->numRegs = regs;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) { return cudaSuccess; }

// what nvcc's host code calls
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *) { return *k = reinterpret_cast<cudaKernel_t>(&handle), cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { return reinterpret_cast<void **>(&handle); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
