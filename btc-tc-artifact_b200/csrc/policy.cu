// policy.cu -- tile width and tau per graph class (the engine's autotuned policy; the
// reference's policy is the fixed BTC-Lite rule, apps/btc_tc_lite.cu:45-65, which stays
// available as btc_lite_select_tile_cols).
//
// The rule comes from a sweep on one B200 of 37 graphs over five families (Erdos-Renyi,
// 27- and 7-point stencils, R-MAT in natural and descending-degree order, 8-block SBMs,
// complete graphs) at both tile widths and three taus (btc_b200/tune.py --sweep; table in
// the autotune profile).  Features, all cheap, in this order:
//   * average degree d = 2m/n >= 512 (dense communities, near-cliques): 16x32, whose
//     dense path packs four matches into one k = 128 MMA;
//   * descending-degree order requested (BTC_ORIENT_DEGREE): power-law graphs whose hubs
//     sit in the first column blocks -> 16x128;
//   * id locality L: the share of sampled input edges with |u - v| < 128 over the share
//     uniform ids would give (about 255/n); L >= 16 (banded or clustered ids: stencils)
//     -> 16x128, else (random ids: Erdos-Renyi, natural-order R-MAT, SBM) 16x32.
// tau: 1024 for 16x128 (dense SBM communities near 30% tile density run 2.6-2.9x faster
// on the sparse path than on the b1 MMA path at the reference's 512, while full tiles
// keep the MMA path), 64 for 16x32 (the reference's: its four-match packing wins there).
#include "common.cuh"
#include "handle.cuh"

#include <algorithm>
#include <cstdlib>
#include <vector>

namespace btc200 {
namespace pol {

constexpr int kThreads = 256;
constexpr int kGrid = 64;
constexpr uint32_t kSamples = kPolicySamples;
constexpr int32_t kNear = kPolicyNear;
// Skew of the row blocks, for lists the grouped builder would take in natural order:
// 65,536 samples over 16,384 counters leave at most some 20 in one where row blocks are alike; 64
// in one are a row block of a 1,024th of the edges.  Above that the grouped builder's CTA for it
// is the last to end (build, grouped / sorted: R-MAT scale 20, edge factor 2, 16x32 2.05 / 0.68 ms;
// a vertex of 3.9M neighbours among 8M pairs 111 / 3.3 ms), below it the sort's passes cost more
// (7-point grid 144^3: 0.54 / 0.95 ms).
constexpr uint32_t kSkewSlots = 1u << 14;
constexpr uint32_t kSkewed = 64;
__host__ __device__ __forceinline__ uint32_t skew_slot(int32_t u, int32_t v)
{
    return ((uint32_t)(u > v ? u : v) >> 4) * 0x9E3779B1u >> (32 - 14);
}

// Sample i reads edge i * step.  Adds the number of local edges and their expectation
// under uniform ids (per sampled edge: the chance that two uniform ids in [0, n) lie
// closer than kNear, about (2 kNear - 1) / n), scaled by 2^20 to stay integer.  With
// e_off / nv (a batch), an edge's n is its own graph's.  skew (nullable): kSkewSlots counters of the
// samples' row blocks (of the oriented edge, hashed) and the most that one got.  out: two sums and a
// ticket.  All are zero at the start; the last CTA hands the sums and the most to the host (mapped
// memory) and zeroes them.
__global__ void k_locality(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t m,
                           int32_t n, const int64_t* __restrict__ e_off, const int32_t* __restrict__ nv,
                           uint32_t G, int64_t step, unsigned int* __restrict__ skew,
                           unsigned long long* __restrict__ out, volatile unsigned long long* host)
{
    constexpr int U = 4;  // samples in flight per thread
    unsigned long long local = 0, expect = 0;
    unsigned int most = 0;
    const uint64_t stride = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i0 = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i0 < kSamples; i0 += U * stride) {
        int32_t u[U], v[U];
        int64_t e[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const uint64_t i = i0 + k * stride;
            e[k] = i < kSamples && (int64_t)i * step < m ? (int64_t)i * step : -1;
            u[k] = e[k] >= 0 ? src[e[k]] : 0;
            v[k] = e[k] >= 0 ? dst[e[k]] : 0;
        }
        if (skew) {
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (e[k] >= 0) most = max(most, atomicAdd(&skew[skew_slot(u[k], v[k])], 1u) + 1u);
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (e[k] < 0) continue;
            int32_t ng = n;
            if (e_off) {
                uint32_t lo = 0, hi = G;  // last g with e_off[g] <= e
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (e_off[mid] <= e[k]) lo = mid;
                    else hi = mid;
                }
                ng = nv[lo];
            }
            policy_sample(u[k], v[k], ng, local, expect);
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        local += __shfl_xor_sync(kFull, local, d);
        expect += __shfl_xor_sync(kFull, expect, d);
    }
    most = __reduce_max_sync(kFull, most);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&out[0], local);
        atomicAdd(&out[1], expect);
        if (skew) atomicMax(&skew[kSkewSlots], most);
        __threadfence();
    }
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&out[2], 1ull) == gridDim.x - 1;
        if (s_last) {
            host[0] = atomicExch(&out[0], 0ull);
            host[1] = atomicExch(&out[1], 0ull);
            if (skew) host[2] = atomicMax(&skew[kSkewSlots], 0u);
            out[2] = 0ull;
            __threadfence_system();
        }
    }
    __syncthreads();
    if (s_last && skew)
        for (uint32_t i = threadIdx.x; i <= kSkewSlots; i += kThreads) skew[i] = 0u;
}

double locality_host(const int32_t* src, const int32_t* dst, int64_t m, int32_t n,
                     const int64_t* e_off, const int32_t* nv, uint32_t G)
{
    const int64_t step = m > (int64_t)kSamples ? m / (int64_t)kSamples : 1;
    double local = 0.0, expect = 0.0;
    uint32_t g = 0;
    for (uint64_t i = 0; i < kSamples; ++i) {
        const int64_t e = (int64_t)i * step;
        if (e >= m) break;
        int32_t ng = n;
        if (e_off) {
            while (g + 1 < G && e_off[g + 1] <= e) ++g;
            ng = nv[g];
        }
        const int32_t u = src[e], v = dst[e];
        if (u == v || u < 0 || v < 0 || u >= ng || v >= ng) continue;
        local += std::abs((int64_t)u - (int64_t)v) < kNear ? 1.0 : 0.0;
        expect += ng > 2 * kNear ? (2.0 * kNear - 1.0) / (double)ng : 1.0;
    }
    return expect > 0.0 ? local / expect : 0.0;
}

uint32_t skew_host(const int32_t* src, const int32_t* dst, int64_t m)
{
    const int64_t step = m > (int64_t)kSamples ? m / (int64_t)kSamples : 1;
    std::vector<uint32_t> count(kSkewSlots, 0u);
    uint32_t most = 0;
    for (uint64_t i = 0; i < kSamples && (int64_t)i * step < m; ++i)
        most = std::max(most, ++count[skew_slot(src[i * step], dst[i * step])]);
    return most;
}

// Average degree 2m/n of at least 512.
bool dense(int64_t m, int32_t n)
{
    return n > 0 && 2.0 * (double)m / (double)n >= 512.0;
}

}  // namespace pol

bool policy_dense(int64_t m, int32_t n) { return pol::dense(m, n); }

// Id locality of an edge list (see above): host arrays are sampled on the host, device
// arrays by one small kernel and one wait on `s`.  e_off / nv (optional, num_graphs + 1 and
// num_graphs entries, host or device like src/dst): batch layout.  w: the caller's words (a
// handle keeps them: an allocation, a memset and a copy back cost a small graph's step 15 us).
int policy_locality(const int32_t* src, const int32_t* dst, int64_t m, int32_t n, bool on_host,
                    const int64_t* e_off, const int32_t* nv, uint32_t G, cudaStream_t s, PolicyWords& w,
                    double* L, bool* skewed)
{
    *L = 0.0;
    if (skewed) *skewed = false;
    if (m <= 0) return BTC_OK;
    if (on_host) {
        *L = pol::locality_host(src, dst, m, n, e_off, nv, G);
        if (skewed) *skewed = pol::skew_host(src, dst, m) >= pol::kSkewed;
        return BTC_OK;
    }
    if (!w.host && !(w.host = host_slot_alloc(&w.host_context))) return BTC_E_NOMEM;
    void* d_host = nullptr;
    BTC_CUDA_TRY(cudaHostGetDevicePointer(&d_host, w.host, 0));
    const bool fresh = w.dev.ptr == nullptr, fresh_skew = w.skew.ptr == nullptr;
    BTC_TRY(w.dev.reserve(3 * sizeof(unsigned long long)));
    // (a call that failed on its way may have left something in them)
    if (fresh || w.dirty) BTC_CUDA_TRY(cudaMemsetAsync(w.dev.ptr, 0, 3 * sizeof(unsigned long long), s));
    constexpr size_t skew_bytes = sizeof(unsigned int) * (pol::kSkewSlots + 1);
    if (skewed) BTC_TRY(w.skew.reserve(skew_bytes));
    if (w.skew.ptr && (fresh_skew || w.dirty)) BTC_CUDA_TRY(cudaMemsetAsync(w.skew.ptr, 0, skew_bytes, s));
    unsigned int* skew = skewed ? w.skew.as<unsigned int>() : nullptr;
    w.dirty = true;
    const int64_t step = m > (int64_t)pol::kSamples ? m / (int64_t)pol::kSamples : 1;
    const int64_t samples = m < (int64_t)pol::kSamples ? m : (int64_t)pol::kSamples;
    const int grid = (int)((samples + 4 * pol::kThreads - 1) / (4 * pol::kThreads));
    pol::k_locality<<<grid, pol::kThreads, 0, s>>>(src, dst, m, n, e_off, nv, G, step, skew,
                                                   w.dev.as<unsigned long long>(),
                                                   static_cast<unsigned long long*>(d_host));
    BTC_CUDA_TRY(cudaGetLastError());
    BTC_CUDA_TRY(cudaStreamSynchronize(s));
    w.dirty = false;
    const volatile unsigned long long* h = w.host;
    *L = h[1] ? (double)h[0] / (double)h[1] : 0.0;
    if (skewed) *skewed = h[2] >= pol::kSkewed;
    return BTC_OK;
}

int policy_select(const int32_t* src, const int32_t* dst, int64_t m, int32_t n, uint32_t flags, cudaStream_t s,
                  PolicyWords& w, int* tile_cols, int* tau, int* skewed)
{
    if (n < 0 || m < 0 || !tile_cols || (m > 0 && (!src || !dst))) return BTC_E_INVAL;
    double L = 0.0;
    // (the locality decides only where neither the degree nor the ordering does)
    if (!(flags & BTC_ORIENT_DEGREE) && !pol::dense(m, n)) {
        bool is = false;
        BTC_TRY(policy_locality(src, dst, m, n, (flags & BTC_INPUT_ON_HOST) != 0, nullptr, nullptr, 0, s, w, &L,
                                skewed ? &is : nullptr));
        if (skewed) *skewed = is;
    }
    return btc_tile_policy_from_features(m, n, flags, L, tile_cols, tau);
}

}  // namespace btc200

using namespace btc200;

extern "C" {

int btc_tile_policy_from_features(int64_t m, int32_t n, uint32_t flags, double locality,
                                  int* tile_cols, int* tau)
{
    if (m < 0 || n < 0 || !tile_cols) return BTC_E_INVAL;
    int C;
    if (pol::dense(m, n)) C = 32;
    else if (flags & BTC_ORIENT_DEGREE) C = 128;
    else C = locality >= 16.0 ? 128 : 32;
    *tile_cols = C;
    if (tau) *tau = default_tau(C);
    return BTC_OK;
}

int btc_select_tile_policy(const int32_t* src, const int32_t* dst, int64_t m, int32_t n,
                           uint32_t flags, btc_stream_t stream, int* tile_cols, int* tau)
{
    PolicyWords w;
    const int st = policy_select(src, dst, m, n, flags, stream, w, tile_cols, tau);
    w.release();
    return st;
}

}  // extern "C"
