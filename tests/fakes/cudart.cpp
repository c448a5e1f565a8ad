// The runtime calls of cudart.hpp.
#include "cudart.hpp"

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = fake::current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { fake::current = d; fake::bound = true; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = fake::devices; return cudaSuccess; }
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = fake::last_error;
    fake::last_error = cudaSuccess;
    return e;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t)
{
    return fake::last_error = fake::cooperative;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void)
{
    fake::bound = true;
    fake::note("wait", fake::current);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { fake::bound = true; return fake::give(p, n); }
cudaError_t cudaFree(void* p)
{
    fake::bound = true;
    if (!p) return cudaSuccess;
    int dev;
    {
        std::lock_guard<std::mutex> l(fake::mu);
        dev = fake::device_of.at(p);
        fake::device_of.erase(p);
    }
    fake::note("free", dev);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t)
{
    fake::bound = true;
    return fake::give(p, n);
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*)
{
    std::lock_guard<std::mutex> l(fake::mu);
    *p = reinterpret_cast<cudaMemPool_t>((uintptr_t)(++fake::pools_made));
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep)
{
    fake::note("trim" + std::to_string((uintptr_t)p) + "to" + std::to_string(keep), fake::current);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 1; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    fake::bound = true;
    *s = reinterpret_cast<cudaStream_t>((uintptr_t)64);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int value)
{
    fake::note("attribute" + std::to_string(value), fake::current);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    fake::bound = true;
    std::lock_guard<std::mutex> l(fake::mu);
    *p = std::malloc(n);
    fake::pinned[*p] = n;
    ++fake::pinned_made;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    std::lock_guard<std::mutex> l(fake::mu);
    auto it = fake::device_of.find(const_cast<void*>(p));
    if (it == fake::device_of.end()) return cudaErrorInvalidValue;
    a->type = cudaMemoryTypeDevice;
    a->device = it->second;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q)
{
    *q = cudaDriverEntryPointSuccess;
    if (!std::strcmp(name, "cuCtxGetCurrent")) *f = reinterpret_cast<void*>(&fake::get_current);
    else if (!std::strcmp(name, "cuCtxGetId")) *f = reinterpret_cast<void*>(&fake::get_id);
    else *q = cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
// what nvcc's host code calls for the kernels of the headers (none is launched)
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return 0; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
char __cudaInitModule(void**) { return 1; }
}
