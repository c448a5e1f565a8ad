// A CUDA runtime of two devices on the host, for checks of what the library asks of the real
// one: every call that waits, allocates or frees is logged with the device it acted on.  A
// program that includes it links no CUDA runtime.
#pragma once

#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace fake {
inline std::mutex mu;
inline std::vector<std::string> log;
inline std::map<void*, int> device_of;         // live device allocations
inline std::map<void*, size_t> pinned;         // live pinned blocks
inline std::map<CUcontext, unsigned long long> ids;
inline int devices = 2;
inline cudaError_t cooperative = cudaSuccess;  // what a cooperative launch answers
inline cudaError_t last_error = cudaSuccess;
inline int pools_made = 0, pinned_made = 0;
inline unsigned long long context_id[2] = {101, 102};  // of each device's context
inline thread_local int current = 0;
inline thread_local bool bound = false;        // a call has made the thread's context current

inline void note(const std::string& what, int dev)
{
    std::lock_guard<std::mutex> l(mu);
    log.push_back(what + "@" + std::to_string(dev));
}
inline cudaError_t give(void** p, size_t n)
{
    *p = std::malloc(n ? n : 1);
    std::lock_guard<std::mutex> l(mu);
    device_of[*p] = current;
    return cudaSuccess;
}
// what a device reset does: the device's context gets a new id, its memory is gone
inline void reset(int dev)
{
    std::lock_guard<std::mutex> l(mu);
    context_id[dev] += 1000;
    for (auto& b : pinned) std::memset(b.first, 0xEE, b.second);
    bound = false;
}
inline CUresult get_current(CUcontext* c)
{
    *c = bound ? reinterpret_cast<CUcontext>((uintptr_t)current + 1) : nullptr;
    return CUDA_SUCCESS;
}
inline CUresult get_id(CUcontext c, unsigned long long* id)
{
    *id = context_id[reinterpret_cast<uintptr_t>(c) - 1];
    return CUDA_SUCCESS;
}
}  // namespace fake
