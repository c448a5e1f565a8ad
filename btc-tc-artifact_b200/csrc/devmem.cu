// devmem.cu -- the library's device memory: one stream-ordered pool per device (and context).
//
// Handles that live for one graph allocate some 20 buffers; with cudaMalloc and cudaFree
// each of them maps and unmaps memory and waits for the device.  The pool keeps up to
// kKeepBytes of freed memory for the next handle; what is above that goes back to the
// device at the next wait, and all of it on btc_trim_memory.  Allocations are made on a stream of the pool's own and are
// complete when dev_alloc returns, so a caller may use the memory on any stream; freed
// memory is idle (dev_free's callers have waited), so it may be handed to any other.
// Allocations of kDirectBytes and more come from cudaMalloc: the pool would not keep them
// and maps them more slowly (a new R-MAT scale 22 handle of 9 GB: 69 ms to build and count
// with all of it pooled, 19.4 like this; scale 20, 1.9 GB: 9.6 / 3.7 ms).
#include "common.cuh"

#include <cuda.h>

#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace btc200 {

unsigned long long current_context_id()
{
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
        cudaGetLastError();
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
    if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

namespace {

constexpr uint64_t kKeepBytes = 1ull << 30;
constexpr size_t kDirectBytes = 256ull << 20;

struct DevicePool {
    cudaMemPool_t pool = nullptr;  // null: no pool support
    cudaStream_t stream = nullptr;
};

// The id of the context the calling thread works in, made current if the thread had none yet (a
// new thread's first call here comes before anything has bound it); 0 when it cannot be read.
unsigned long long bound_context_id()
{
    unsigned long long id = current_context_id();
    int dev = 0;
    if (id == 0 && cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess)
        id = current_context_id();
    return id;
}

// The current device's pool, made on first use in each context; false without pool support.  A
// context's pool is kept for as long as the process runs: contexts come and go seldom, and one
// that is met again (a second context on the device) finds its pool.
bool pool_for_current_device(cudaMemPool_t* pool, cudaStream_t* stream)
{
    static std::mutex mu;
    static auto& pools = *new std::map<std::pair<int, unsigned long long>, DevicePool>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const unsigned long long id = bound_context_id();
    std::lock_guard<std::mutex> lock(mu);
    const auto found = pools.find({dev, id});
    if (found != pools.end()) {
        *pool = found->second.pool;
        *stream = found->second.stream;
        return *pool != nullptr;
    }
    DevicePool& p = pools[{dev, id}];
    int supported = 0;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    uint64_t keep = kKeepBytes;
    if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess ||
        !supported || cudaMemPoolCreate(&p.pool, &props) != cudaSuccess) {
        p.pool = nullptr;
    } else if (cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
               cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaMemPoolDestroy(p.pool);
        p.pool = nullptr;
    }
    if (!p.pool) cudaGetLastError();
    *pool = p.pool;
    *stream = p.stream;
    return p.pool != nullptr;
}

}  // namespace

// Pinned, mapped host slots of kHostSlotWords uint64, carved from blocks that stay until the
// process ends (64 KB holds 512 handles; cudaHostAlloc and cudaFreeHost cost 0.01 to 5 ms a
// handle).  A block belongs to the context that made it (a device reset takes its memory with
// it), and its slots are handed out in that context only: whoever gives one back names it.
namespace {

constexpr size_t kSlotsPerBlock = 512;

struct HostSlots {
    std::mutex mu;
    std::map<unsigned long long, std::vector<unsigned long long*>> free_slots;  // by context
};
HostSlots& host_slots()
{
    static HostSlots* h = new HostSlots;  // (outlives handles freed at exit)
    return *h;
}

}  // namespace

unsigned long long* host_slot_alloc(unsigned long long* context)
{
    HostSlots& h = host_slots();
    *context = bound_context_id();
    std::lock_guard<std::mutex> lock(h.mu);
    std::vector<unsigned long long*>& free_slots = h.free_slots[*context];
    if (free_slots.empty()) {
        void* p = nullptr;
        if (cudaHostAlloc(&p, sizeof(unsigned long long) * kHostSlotWords * kSlotsPerBlock,
                          cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        for (size_t i = kSlotsPerBlock; i-- > 0;)
            free_slots.push_back(static_cast<unsigned long long*>(p) + i * kHostSlotWords);
    }
    unsigned long long* s = free_slots.back();
    free_slots.pop_back();
    std::memset(s, 0, sizeof(unsigned long long) * kHostSlotWords);
    return s;
}

void host_slot_free(unsigned long long* s, unsigned long long context)
{
    if (!s) return;
    HostSlots& h = host_slots();
    std::lock_guard<std::mutex> lock(h.mu);
    h.free_slots[context].push_back(s);
}

cudaError_t dev_alloc(void** ptr, size_t bytes)
{
    cudaMemPool_t pool;
    cudaStream_t stream;
    const bool pooled = pool_for_current_device(&pool, &stream);
    if (bytes >= kDirectBytes || !pooled) {
        cudaError_t e = cudaMalloc(ptr, bytes);
        if (e == cudaErrorMemoryAllocation && pooled) {
            // (the memory that the pool keeps may be what is missing)
            cudaGetLastError();
            cudaMemPoolTrimTo(pool, 0);
            e = cudaMalloc(ptr, bytes);
        }
        return e;
    }
    cudaError_t e = cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
    if (e == cudaErrorMemoryAllocation) {
        // give the kept memory back and try once more
        cudaGetLastError();
        cudaMemPoolTrimTo(pool, 0);
        e = cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
    }
    return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
}

bool allow_dynamic_smem(const void* kernel, size_t bytes, std::atomic<unsigned long long>* done)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
    const unsigned long long id = bound_context_id();
    if (id != 0 && done[dev].load(std::memory_order_acquire) == id) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    done[dev].store(id, std::memory_order_release);
    return true;
}

cudaError_t wait_device(int dev)
{
    int cur = 0;
    if (dev < 0 || cudaGetDevice(&cur) != cudaSuccess || cur == dev) return cudaDeviceSynchronize();
    cudaError_t e = cudaSetDevice(dev);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    const cudaError_t back = cudaSetDevice(cur);
    return e != cudaSuccess ? e : back;
}

void dev_free(void* p)
{
    // (cudaFree of pool memory returns it to its pool without a wait)
    if (p) cudaFree(p);
}

void free_arrays(void* const* arrays, int n)
{
    const void* any = nullptr;
    for (int i = 0; i < n && !any; ++i) any = arrays[i];
    if (!any) return;
    cudaPointerAttributes a{};
    const bool known = cudaPointerGetAttributes(&a, any) == cudaSuccess && a.type == cudaMemoryTypeDevice;
    if (!known) cudaGetLastError();
    if (wait_device(known ? a.device : -1) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    for (int i = 0; i < n; ++i) dev_free(arrays[i]);
}

}  // namespace btc200

extern "C" int btc_trim_memory(uint64_t keep_bytes)
{
    using namespace btc200;
    cudaMemPool_t pool;
    cudaStream_t stream;
    if (!pool_for_current_device(&pool, &stream)) return BTC_OK;  // (nothing is kept)
    BTC_CUDA_TRY(cudaMemPoolTrimTo(pool, keep_bytes));
    return BTC_OK;
}
