// small.cu -- Bit-BSR builder for small graphs in natural order: the tile policy's sample and
// the whole cell-bitmap build (bitmap.cu) in one cooperative launch.
//
// A graph of a few thousand edges spends its step on launches, not on work: sample, two
// memsets, mark, popcount scan, emit, fill and the longest list are eight enqueued
// operations and two waits (Erdos-Renyi 256 / 24,
// 3,072 draws: 72 us a step, 54 like this).  Here one grid
// of co-resident CTAs (about 2,048 edges each) runs them as phases between grid barriers,
// and the tile width it picks reaches the host with the build's status.
//
//   phase 0  cell words and metadata zeroed; the sample of the tile policy (policy.cu)
//   phase 1  the width is known: mark the cells
//   phase 2  popcount of each CTA's share of the words
//   phase 3  tile prefix: pairs, indices, row_indices, indptr; tiles and row masks zeroed
//   phase 4  tiles and row masks filled, the longest row-block list
//
// A barrier counts arrivals; its wait is bounded (a cooperative launch's CTAs are all resident, so
// the bound is not met unless they are kept from running; past it the build reports that it gave
// up, and the caller builds otherwise).
#include "common.cuh"

#include <algorithm>
#include <atomic>

namespace btc200 {
namespace sm {

constexpr int kThreads = 256;
constexpr int kEdges = 8;  // edges in flight per thread

struct Args {
    const int32_t* src;
    const int32_t* dst;
    int64_t m;
    int32_t n;
    int tile_cols;  // 0: the policy's
    uint32_t* words;  // cell words of the wider grid (16x32 tiles)
    uint32_t* counts; // one per CTA
    uint2* cellpp;
    uint32_t* indices;
    uint32_t* row_indices;
    uint32_t* indptr;
    uint32_t* blocks;
    uint32_t* rowmask;
    uint32_t cap128, cap32;  // tiles the arrays hold at either width
    unsigned long long* meta;
    unsigned long long* host;   // mapped status slots
    unsigned long long* words3; // the policy's two sums (zero at the start)
    unsigned int* bar;          // arrivals, CTAs done (zero at the start)
    int64_t step;               // the policy's sample
    uint32_t samples;
    uint32_t max_spins;         // of a barrier's wait
};

__device__ __forceinline__ bool barrier(unsigned int* bar, unsigned target, uint32_t max_spins)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        uint32_t spins = 0;
        while (*(volatile unsigned int*)bar < target && ++spins < max_spins) {
        }
        s_ok = spins < max_spins;
        __threadfence();
    }
    __syncthreads();
    return s_ok;
}

// Phases 1 to 4 at one tile width.  false: a barrier gave up.
template <int LOG2C>
__device__ __forceinline__ bool build(const Args& a, uint32_t cap, uint32_t* s_scan)
{
    constexpr int C = 1 << LOG2C, TW = 16 * (C / 32);
    const uint32_t R = (uint32_t)((a.n + 15) / 16);
    const uint32_t wpr = (((uint32_t)a.n + C - 1) / C + 31) / 32;
    const uint32_t W = R * wpr;
    const uint32_t G = gridDim.x;
    const int64_t stride = (int64_t)G * kThreads;
    uint32_t nbad = 0;
    for (int64_t i0 = (int64_t)blockIdx.x * kThreads + threadIdx.x; i0 < a.m; i0 += kEdges * stride) {
        int32_t u[kEdges], v[kEdges];
#pragma unroll
        for (int k = 0; k < kEdges; ++k) {
            const int64_t i = i0 + k * stride;
            u[k] = i < a.m ? a.src[i] : 0;
            v[k] = i < a.m ? a.dst[i] : 0;
        }
#pragma unroll
        for (int k = 0; k < kEdges; ++k) {
            if ((u[k] < 0) | (v[k] < 0) | (u[k] >= a.n) | (v[k] >= a.n)) {
                ++nbad;
            } else if (u[k] != v[k]) {
                const uint32_t cb = (uint32_t)min(u[k], v[k]) >> LOG2C;
                uint32_t* w = &a.words[((uint32_t)max(u[k], v[k]) >> 4) * wpr + (cb >> 5)];
                const uint32_t bit = 1u << (cb & 31u);
                if (!(*(volatile uint32_t*)w & bit)) atomicOr(w, bit);
            }
        }
    }
    nbad = __reduce_add_sync(kFull, nbad);
    if ((threadIdx.x & 31) == 0 && nbad) atomicAdd(&a.meta[kMetaBad], (unsigned long long)nbad);
    if (!barrier(a.bar, 2 * G, a.max_spins)) return false;

    // this CTA's words: whole runs of kThreads
    const uint32_t per = (W + G * kThreads - 1) / (G * kThreads) * kThreads;
    const uint32_t wa = min(blockIdx.x * per, W), wb = min(wa + per, W);
    uint32_t cnt = 0;
    for (uint32_t w = wa + threadIdx.x; w < wb; w += kThreads) cnt += __popc(__ldcg(&a.words[w]));
    uint32_t mine;
    cta_exclusive_scan<kThreads>(cnt, s_scan, mine);
    if (threadIdx.x == 0) a.counts[blockIdx.x] = mine;
    if (!barrier(a.bar, 3 * G, a.max_spins)) return false;

    uint32_t before = 0, all = 0;
    for (uint32_t b = threadIdx.x; b < G; b += kThreads) {
        const uint32_t c = __ldcg(&a.counts[b]);
        all += c;
        before += b < blockIdx.x ? c : 0u;
    }
    uint32_t base, T;
    cta_exclusive_scan<kThreads>(before, s_scan, base);
    cta_exclusive_scan<kThreads>(all, s_scan, T);
    const bool fits = T <= cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.meta[kMetaTiles] = T;
        a.indptr[R] = T;
        if (!fits) a.meta[kMetaOverflow] = 1ull;
    }
    if (fits) {
        for (uint32_t i = base * (TW / 4) + threadIdx.x; i < (base + mine) * (TW / 4); i += kThreads)
            reinterpret_cast<uint4*>(a.blocks)[i] = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t i = base + threadIdx.x; i < base + mine; i += kThreads) a.rowmask[i] = 0u;
        for (uint32_t w0 = wa; w0 < wb; w0 += kThreads) {
            const uint32_t w = w0 + threadIdx.x;
            uint32_t x = w < wb ? __ldcg(&a.words[w]) : 0u;
            uint32_t total;
            uint32_t t = base + cta_exclusive_scan<kThreads>(__popc(x), s_scan, total);
            if (w < wb) {
                const uint32_t rb = w / wpr, cw = w - rb * wpr;
                a.cellpp[w] = make_uint2(x, t);
                if (cw == 0) a.indptr[rb] = t;
                while (x) {
                    a.indices[t] = cw * 32 + (__ffs(x) - 1);
                    a.row_indices[t] = rb;
                    x &= x - 1;
                    ++t;
                }
            }
            base += total;
        }
    }
    if (!barrier(a.bar, 4 * G, a.max_spins)) return false;
    if (!fits) return true;

    uint32_t longest = 0;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < R; i += G * kThreads)
        longest = max(longest, __ldcg(&a.indptr[i + 1]) - __ldcg(&a.indptr[i]));
    longest = __reduce_max_sync(kFull, longest);
    if ((threadIdx.x & 31) == 0 && longest) atomicMax(&a.meta[kMetaRowMax], (unsigned long long)longest);
    for (int64_t i0 = (int64_t)blockIdx.x * kThreads + threadIdx.x; i0 < a.m; i0 += kEdges * stride) {
        uint32_t tile[kEdges], at[kEdges];
        int32_t u[kEdges], v[kEdges];
        bool ok[kEdges];
#pragma unroll
        for (int k = 0; k < kEdges; ++k) {
            const int64_t i = i0 + k * stride;
            u[k] = i < a.m ? a.src[i] : 0;
            v[k] = i < a.m ? a.dst[i] : 0;
        }
#pragma unroll
        for (int k = 0; k < kEdges; ++k) {
            ok[k] = !((u[k] < 0) | (v[k] < 0) | (u[k] >= a.n) | (v[k] >= a.n)) && u[k] != v[k];
            const uint32_t r = (uint32_t)max(u[k], v[k]), c = (uint32_t)min(u[k], v[k]), cb = c >> LOG2C;
            tile[k] = 0;
            if (ok[k]) {
                const uint2 cp = __ldcg(&a.cellpp[(r >> 4) * wpr + (cb >> 5)]);
                tile[k] = cp.y + __popc(cp.x & ((1u << (cb & 31u)) - 1u));
            }
            at[k] = ((r & 15u) << LOG2C) | (c & (C - 1));
        }
#pragma unroll
        for (int k = 0; k < kEdges; ++k)
            u[k] = ok[k] ? (int32_t)atomicOr(&a.blocks[tile[k] * TW + (at[k] >> 5)], 1u << (at[k] & 31u)) : 1;
#pragma unroll
        for (int k = 0; k < kEdges; ++k)
            if (u[k] == 0)
                atomicOr(&a.rowmask[tile[k]],
                         1u << ((at[k] >> LOG2C) + (C == 128 ? (at[k] & 64u) / 4u : 0u)));
    }
    return true;
}

__global__ void __launch_bounds__(kThreads) k_build_small(Args a)
{
    __shared__ uint32_t s_scan[kThreads / kWarp];
    // ---- phase 0 ------------------------------------------------------------------------
    const uint32_t gid = blockIdx.x * kThreads + threadIdx.x, all = gridDim.x * kThreads;
    const uint32_t R = (uint32_t)((a.n + 15) / 16);
    const uint32_t c0 = a.tile_cols ? a.tile_cols : 32;
    const uint32_t W = R * ((((uint32_t)a.n + c0 - 1) / c0 + 31) / 32);
    for (uint32_t w = gid; w < W; w += all) a.words[w] = 0u;
    if (gid < kMetaSlots) a.meta[gid] = 0ull;
    if (a.tile_cols == 0) {
        unsigned long long local = 0, expect = 0;
        for (uint32_t i = gid; i < a.samples; i += all)
            policy_sample(a.src[i * a.step], a.dst[i * a.step], a.n, local, expect);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            local += __shfl_xor_sync(kFull, local, d);
            expect += __shfl_xor_sync(kFull, expect, d);
        }
        if ((threadIdx.x & 31) == 0) {
            if (local) atomicAdd(&a.words3[0], local);
            if (expect) atomicAdd(&a.words3[1], expect);
        }
    }
    bool ok = barrier(a.bar, gridDim.x, a.max_spins);
    int tile_cols = a.tile_cols;
    if (ok) {
        if (tile_cols == 0)
            tile_cols = policy_is_local(__ldcg(&a.words3[0]), __ldcg(&a.words3[1])) ? 128 : 32;
        ok = tile_cols == 128 ? build<7>(a, a.cap128, s_scan) : build<5>(a, a.cap32, s_scan);
    }
    // ---- the last CTA hands the status to the host and leaves the counters at zero --------
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!ok) a.meta[kMetaOverflow] = kGaveUp;
        __threadfence();
        if (atomicAdd(&a.bar[1], 1u) == gridDim.x - 1) {
            __threadfence();
            volatile unsigned long long* h = a.host;
            const unsigned long long over = __ldcg(&a.meta[kMetaOverflow]);
            h[kMetaBad] = __ldcg(&a.meta[kMetaBad]);
            h[kMetaTiles] = __ldcg(&a.meta[kMetaTiles]);
            h[kMetaOverflow] = over;
            h[kHostTileCols] = (unsigned long long)tile_cols;
            a.words3[0] = a.words3[1] = 0ull;
            a.bar[0] = a.bar[1] = 0u;
            __threadfence_system();
        }
    }
}

}  // namespace sm

// CTAs for m edges: 2,048 each, at most two per SM (they must all be resident at once).
static int small_grid(int64_t m)
{
    const int64_t want = (m + sm::kThreads * sm::kEdges - 1) / (sm::kThreads * sm::kEdges);
    return (int)std::max<int64_t>(1, std::min<int64_t>(want, 2 * (int64_t)device_sm_count()));
}

int launch_build_small(const SmallBuild& b, cudaStream_t s)
{
    static std::atomic<int> per_sm[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return BTC_E_CUDA;
    int p = per_sm[dev].load(std::memory_order_relaxed);
    if (p == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, sm::k_build_small, sm::kThreads, 0) != cudaSuccess || p < 2) {
            cudaGetLastError();
            return kNotLaunched;
        }
        per_sm[dev].store(p, std::memory_order_relaxed);
    }
    sm::Args a{b.src, b.dst, b.m, b.n, b.tile_cols, b.words, b.counts, b.cellpp, b.indices, b.row_indices, b.indptr,
               b.blocks, b.rowmask, b.cap128, b.cap32, b.meta, b.host, b.policy_sums, b.bar, b.step, b.samples,
               b.max_spins};
    void* args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel(sm::k_build_small, dim3((unsigned)small_grid(b.m)),
                                                      dim3(sm::kThreads), args, 0, s);
    if (e == cudaSuccess) return BTC_OK;
    cudaGetLastError();  // (refused: the next check of an error is not to find it)
    return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported ? kNotLaunched : BTC_E_CUDA;
}

}  // namespace btc200
