// csrc/small.cu on the GPU with a wait that runs out at once: the launch ends, reports that it gave
// up, writes nothing past the cell words and leaves its counters ready for the next build, which
// then builds the tiles of a path.
#include "common.cuh"

#include <cstdio>
#include <cstring>
#include <vector>

namespace btc200 {
void note_cuda_error(cudaError_t, const char*, const char*, int) {}
int device_sm_count()
{
    int n = 148;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, 0);
    return n;
}
}  // namespace btc200

using namespace btc200;

#define CHECK(c)                                               \
    do {                                                       \
        if (!(c)) {                                            \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c); \
            return 1;                                          \
        }                                                      \
    } while (0)

template <class T>
static T* device(size_t n)
{
    void* p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess || cudaMemset(p, 0, n * sizeof(T)) != cudaSuccess) return nullptr;
    return static_cast<T*>(p);
}

int main()
{
    const int n = 4096, m = 40000;  // 20 CTAs; every pair (i, i + 1) many times over
    std::vector<int32_t> u(m), v(m);
    for (int i = 0; i < m; ++i) {
        u[i] = i % (n - 1);
        v[i] = u[i] + 1;
    }
    const uint32_t R = n / 16, cells = R * (n / 32);
    SmallBuild b{};
    int32_t *src = device<int32_t>(m), *dst = device<int32_t>(m);
    unsigned long long* small = device<unsigned long long>(4);
    void* host = nullptr;
    CHECK(cudaHostAlloc(&host, 128, cudaHostAllocMapped) == cudaSuccess);
    std::memset(host, 0, 128);
    void* d_host = nullptr;
    CHECK(cudaHostGetDevicePointer(&d_host, host, 0) == cudaSuccess);
    CHECK(cudaMemcpy(src, u.data(), m * 4, cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(cudaMemcpy(dst, v.data(), m * 4, cudaMemcpyHostToDevice) == cudaSuccess);
    b.src = src;
    b.dst = dst;
    b.m = m;
    b.n = n;
    b.tile_cols = 32;
    b.words = device<uint32_t>(R * (n / 32 / 32));
    b.counts = device<uint32_t>(2 * device_sm_count());
    b.cellpp = device<uint2>(R * (n / 32 / 32));
    b.indices = device<uint32_t>(cells);
    b.row_indices = device<uint32_t>(cells);
    b.indptr = device<uint32_t>(R + 1);
    b.blocks = device<uint32_t>(16 * (size_t)cells);
    b.rowmask = device<uint32_t>(cells);
    b.cap128 = b.cap32 = cells;
    b.meta = device<unsigned long long>(kMetaSlots);
    b.host = static_cast<unsigned long long*>(d_host);
    b.policy_sums = small;
    b.bar = reinterpret_cast<unsigned int*>(small + 2);
    b.step = 1;
    b.samples = m;
    CHECK(src && dst && small && b.words && b.counts && b.cellpp && b.indices && b.row_indices && b.indptr && b.blocks &&
          b.rowmask && b.meta);

    volatile unsigned long long* h = static_cast<unsigned long long*>(host);
    b.max_spins = 0;  // every wait has run out when it begins
    CHECK(launch_build_small(b, nullptr) == BTC_OK);
    CHECK(cudaDeviceSynchronize() == cudaSuccess);
    CHECK(h[kMetaOverflow] == kGaveUp && h[kMetaTiles] == 0);
    unsigned long long counters[4] = {1, 1, 1, 1};
    CHECK(cudaMemcpy(counters, small, sizeof(counters), cudaMemcpyDeviceToHost) == cudaSuccess);
    for (unsigned long long c : counters) CHECK(c == 0);
    uint32_t t = 1;
    CHECK(cudaMemcpy(&t, b.indptr + R, 4, cudaMemcpyDeviceToHost) == cudaSuccess && t == 0);

    b.max_spins = SmallBuild{}.max_spins;
    CHECK(launch_build_small(b, nullptr) == BTC_OK);
    CHECK(cudaDeviceSynchronize() == cudaSuccess);
    CHECK(h[kMetaOverflow] == 0 && h[kMetaBad] == 0);
    // a row block I holds the pairs (16 I + r, 16 I + r - 1): its own column block, and from every
    // even I on the last column of the block before
    CHECK(h[kMetaTiles] == R + R / 2 - 1);
    std::printf("small wait ok\n");
    return 0;
}
