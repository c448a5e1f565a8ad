// group.cu -- Bit-BSR builder for large edge lists: the edges are grouped by row block, then a
// CTA builds each row block's tiles in shared memory.
//
// Replaces what convert_coo_to_bcsr_16x128_gpu / _16x32_gpu do after their sort
// (btc/operations/bcsr_16x128.h:136-241, bcsr_16x32.h:144-249).  The cell-bitmap builder
// (bitmap.cu) sends every edge to its tile in device memory: on R-MAT scale 22 two random
// 64-byte fetches an edge, after zeroing 5.3 GB of tiles.  Here an edge is moved twice in
// near-sequential runs and meets its tile in shared memory, and a tile is written once:
//
//   k_orient      edge -> (row, column) with row > column, range check, self-loops dropped;
//                 counts the edges of each bucket of rows (up to kBuckets buckets).  With a
//                 degree rank the pair is stored, so that the
//                 random rank look-ups happen once.
//   k_bucket_scan bucket starts
//   k_scatter     tiles of 8192 edges sorted by bucket in shared memory, written in runs to
//                 space reserved per bucket (order inside a bucket is free)
//   k_rb_count    edges per row block; scanned into the row blocks' offsets
//   k_rb_scatter  every edge to its row block, as a 32-bit word (row in block << 28 | column)
//   k_count_tiles one CTA per row block: distinct column blocks, by a shared bitmap; a heavy row
//                 block (heavy_edges) is only listed
//   k_heavy_mark  the listed ones, a CTA per slice of their edges: bitmap in device memory, tiles
//   (scan)        tile offsets
//   k_write_tiles one CTA per row block: the bitmap again with a popcount prefix (tile order
//                 is column order), indices, row_indices, tiles ORed in shared memory and
//                 written once, row-occupancy masks
//   k_heavy_emit  the listed ones: prefix, indices, row_indices, tiles and masks zeroed
//   k_heavy_fill  ... and filled, a CTA per slice of their edges
//
// Needs columns below 2^28 and a row block's column bitmap in shared memory (kMaxWords
// words).  Duplicate edges OR the same bit.
#include "common.cuh"

#include <algorithm>
#include <atomic>

namespace btc200 {

int launch_tile_scan(uint32_t* per_tile, uint32_t ntiles, unsigned long long* total, cudaStream_t s);
int launch_scan_u32(uint32_t* v, uint32_t n, uint32_t* bsum, unsigned long long* total, cudaStream_t s);

namespace gp {

constexpr int kBuckets = 2048;
constexpr uint32_t kMaxWords = 4096;
constexpr uint64_t kNone = ~0ull;

// ---- orientation -----------------------------------------------------------------------
constexpr int kOThreads = 512;

__device__ __forceinline__ uint64_t pair_of(int32_t u, int32_t v, int32_t n,
                                            const int32_t* __restrict__ rank, bool& bad)
{
    bad = (u < 0) | (v < 0) | (u >= n) | (v >= n);
    if (bad) return kNone;
    if (rank) {
        u = rank[u];
        v = rank[v];
    }
    if (u == v) return kNone;
    return ((uint64_t)(uint32_t)max(u, v) << 32) | (uint32_t)min(u, v);
}

// pairs (nullable): the oriented pairs, kNone for what is dropped.
__global__ void __launch_bounds__(kOThreads)
k_orient(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t m, int32_t n,
         const int32_t* __restrict__ rank, int shift, uint64_t* __restrict__ pairs,
         uint32_t* __restrict__ hist, unsigned long long* __restrict__ bad_count)
{
    __shared__ uint32_t s_hist[kBuckets];
    for (int i = threadIdx.x; i < kBuckets; i += kOThreads) s_hist[i] = 0;
    __syncthreads();
    constexpr int U = 8;
    uint32_t nbad = 0;
    for (int64_t i0 = (int64_t)blockIdx.x * (U * kOThreads) + threadIdx.x; i0 < m + threadIdx.x;
         i0 += (int64_t)gridDim.x * (U * kOThreads)) {
        int32_t u[U], v[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int64_t i = i0 + k * kOThreads;
            u[k] = i < m ? src[i] : 0;
            v[k] = i < m ? dst[i] : 0;
        }
        uint64_t p[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int64_t i = i0 + k * kOThreads;
            bool bad;
            p[k] = pair_of(u[k], v[k], n, rank, bad);
            if (i >= m) p[k] = kNone;
            else nbad += bad;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int64_t i = i0 + k * kOThreads;
            if (p[k] != kNone) atomicAdd(&s_hist[(uint32_t)(p[k] >> 32) >> shift], 1u);
            if (pairs && i < m) pairs[i] = p[k];
        }
    }
    nbad = __reduce_add_sync(kFull, nbad);
    if ((threadIdx.x & 31) == 0 && nbad) atomicAdd(bad_count, (unsigned long long)nbad);
    __syncthreads();
    for (int i = threadIdx.x; i < kBuckets; i += kOThreads)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// base[b] = edges of buckets below b (base[kBuckets] = all); cursor = the same.  No row block is
// listed as heavy yet.
__global__ void __launch_bounds__(1024)
k_bucket_scan(const uint32_t* __restrict__ hist, uint32_t* __restrict__ base, uint32_t* __restrict__ cursor,
              uint32_t* __restrict__ heavy_count)
{
    __shared__ uint32_t s_warp[32];
    static_assert(kBuckets == 2048, "two buckets per thread");
    const uint32_t a = hist[2 * threadIdx.x], b = hist[2 * threadIdx.x + 1];
    uint32_t total;
    const uint32_t ex = cta_exclusive_scan<1024>(a + b, s_warp, total);
    base[2 * threadIdx.x] = cursor[2 * threadIdx.x] = ex;
    base[2 * threadIdx.x + 1] = cursor[2 * threadIdx.x + 1] = ex + a;
    if (threadIdx.x == 1023) base[kBuckets] = total;
    if (threadIdx.x == 0) *heavy_count = 0;
}

// ---- edges to buckets --------------------------------------------------------------------
constexpr int kSThreads = 512;
constexpr int kSItems = 16;
constexpr int kSTile = kSThreads * kSItems;

struct ScatterSmem {
    uint64_t stage[kSTile];
    uint32_t start[kBuckets];  // first place of a bucket in stage
    uint32_t count[kBuckets];
    uint32_t dest[kBuckets];   // its place in the output less start
    uint32_t scan[kSThreads / kWarp];
};

__global__ void __launch_bounds__(kSThreads, 2)
k_scatter(const uint64_t* __restrict__ pairs, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
          int64_t m, int32_t n, int shift, uint32_t* __restrict__ cursor, uint64_t* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char scatter_smem_raw[];
    ScatterSmem& s = *reinterpret_cast<ScatterSmem*>(scatter_smem_raw);
    const int64_t base = (int64_t)blockIdx.x * kSTile + threadIdx.x;
    for (int i = threadIdx.x; i < kBuckets; i += kSThreads) s.count[i] = 0;
    uint64_t p[kSItems];
    if (pairs) {
#pragma unroll
        for (int k = 0; k < kSItems; ++k) {
            const int64_t i = base + k * kSThreads;
            p[k] = i < m ? pairs[i] : kNone;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kSItems; ++k) {
            const int64_t i = base + k * kSThreads;
            const int32_t u = i < m ? src[i] : 0, v = i < m ? dst[i] : 0;
            bool bad;
            p[k] = pair_of(u, v, n, nullptr, bad);
            if (i >= m) p[k] = kNone;
        }
    }
    __syncthreads();
    uint32_t at[kSItems];
#pragma unroll
    for (int k = 0; k < kSItems; ++k)
        if (p[k] != kNone) at[k] = atomicAdd(&s.count[(uint32_t)(p[k] >> 32) >> shift], 1u);
    __syncthreads();
    constexpr int kPer = kBuckets / kSThreads;
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        c[k] = s.count[kPer * threadIdx.x + k];
        sum += c[k];
    }
    uint32_t total;
    uint32_t run = cta_exclusive_scan<kSThreads>(sum, s.scan, total);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int b = kPer * threadIdx.x + k;
        s.start[b] = run;
        s.dest[b] = c[k] ? atomicAdd(&cursor[b], c[k]) - run : 0u;
        run += c[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSItems; ++k)
        if (p[k] != kNone) s.stage[s.start[(uint32_t)(p[k] >> 32) >> shift] + at[k]] = p[k];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < total; i += kSThreads) {
        const uint64_t q = s.stage[i];
        out[s.dest[(uint32_t)(q >> 32) >> shift] + i] = q;
    }
}

// ---- buckets to row blocks -----------------------------------------------------------------
// Tiles of kSTile consecutive edges of the bucketed list, whatever buckets they lie in, so
// that a heavy bucket keeps many CTAs busy (one CTA per bucket: 1.96 ms on R-MAT scale 22,
// whose buckets differ by a factor of 20; 0.50 ms
// like this).  A tile's row blocks are close together; its
// per-row-block counts go through shared memory when they span at most kSpan.
constexpr uint32_t kSpan = 8192;

// The tile's row blocks: [lo, lo + span).
__device__ __forceinline__ void tile_span(const uint64_t (&p)[kSItems], uint32_t* s_mm, uint32_t& lo, uint32_t& span)
{
    uint32_t mn = 0xffffffffu, mx = 0;
#pragma unroll
    for (int k = 0; k < kSItems; ++k)
        if (p[k] != kNone) {
            const uint32_t rb = (uint32_t)(p[k] >> 36);
            mn = min(mn, rb);
            mx = max(mx, rb);
        }
    mn = __reduce_min_sync(kFull, mn);
    mx = __reduce_max_sync(kFull, mx);
    if (threadIdx.x == 0) {
        s_mm[0] = 0xffffffffu;
        s_mm[1] = 0;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_mm[0], mn);
        atomicMax(&s_mm[1], mx);
    }
    __syncthreads();
    lo = s_mm[0];
    span = s_mm[1] >= lo ? s_mm[1] - lo + 1 : 0u;
}

// Row blocks with so many edges that one CTA each would be the last to end (a clique's): above
// 4,096 edges and a 512th of all, so there are fewer than 512 of them.  They are built by slices of
// kSlice edges through bitmaps in device memory.  Cliques of 2,900 and 6,000 among sparse pairs on
// 200,000 and 1M vertices, in degree order, 16x128: build 0.46 -> 0.36 and 1.45 -> 1.34 ms; where
// there are none the three launches cost 8 us.
constexpr uint32_t kMaxHeavy = 512;
constexpr uint32_t kHeavyLeast = 4096;
constexpr uint32_t kSlice = 2048;
inline uint32_t heavy_edges(int64_t m) { return (uint32_t)std::max<int64_t>(kHeavyLeast, m / kMaxHeavy); }
inline uint32_t heavy_most(int64_t m) { return (uint32_t)std::min<int64_t>(kMaxHeavy, m / kHeavyLeast); }
struct Heavy {
    uint32_t* count;
    uint32_t* list;  // row blocks
    uint32_t* done;  // slices marked
    uint32_t* bm;    // a bitmap of `words` words each
    uint32_t* pre;   // tiles of the row block before each word
    uint32_t limit;  // edges of a row block that is not heavy, at most
    uint32_t most;   // room in the arrays above
};

// cnt[I] += the edges of row block I.  Also zeroes the heavy row blocks' bitmaps.
__global__ void __launch_bounds__(kSThreads)
k_rb_count(const uint64_t* __restrict__ in, const uint32_t* __restrict__ d_m, uint32_t* __restrict__ cnt,
           uint32_t* __restrict__ bitmaps, uint32_t bitmap_words)
{
    for (uint32_t i = blockIdx.x * kSThreads + threadIdx.x; i < bitmap_words; i += gridDim.x * kSThreads)
        bitmaps[i] = 0;
    __shared__ uint32_t s_cnt[kSpan];
    __shared__ uint32_t s_mm[2];
    const uint32_t m = *d_m;
    const uint64_t base = (uint64_t)blockIdx.x * kSTile;
    if (base >= m) return;
    uint64_t p[kSItems];
#pragma unroll
    for (int k = 0; k < kSItems; ++k) {
        const uint64_t i = base + k * kSThreads + threadIdx.x;
        p[k] = i < m ? in[i] : kNone;
    }
    uint32_t lo, span;
    tile_span(p, s_mm, lo, span);
    if (span > kSpan) {
#pragma unroll
        for (int k = 0; k < kSItems; ++k)
            if (p[k] != kNone) atomicAdd(&cnt[(uint32_t)(p[k] >> 36)], 1u);
        return;
    }
    for (uint32_t i = threadIdx.x; i < span; i += kSThreads) s_cnt[i] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSItems; ++k)
        if (p[k] != kNone) atomicAdd(&s_cnt[(uint32_t)(p[k] >> 36) - lo], 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < span; i += kSThreads)
        if (s_cnt[i]) atomicAdd(&cnt[lo + i], s_cnt[i]);
}

// Every edge to its row block: cursor[I] is the next place of row block I (its offset at
// first, the next row block's at the end).
__global__ void __launch_bounds__(kSThreads)
k_rb_scatter(const uint64_t* __restrict__ in, const uint32_t* __restrict__ d_m, uint32_t* __restrict__ cursor,
             uint32_t* __restrict__ out)
{
    __shared__ uint32_t s_cnt[kSpan];
    __shared__ uint32_t s_mm[2];
    const uint32_t m = *d_m;
    const uint64_t base = (uint64_t)blockIdx.x * kSTile;
    if (base >= m) return;
    uint64_t p[kSItems];
#pragma unroll
    for (int k = 0; k < kSItems; ++k) {
        const uint64_t i = base + k * kSThreads + threadIdx.x;
        p[k] = i < m ? in[i] : kNone;
    }
    uint32_t lo, span;
    tile_span(p, s_mm, lo, span);
    auto word = [](uint64_t q) { return ((uint32_t)(q >> 4) & 0xf0000000u) | (uint32_t)q; };
    if (span > kSpan) {
#pragma unroll
        for (int k = 0; k < kSItems; ++k)
            if (p[k] != kNone) out[atomicAdd(&cursor[(uint32_t)(p[k] >> 36)], 1u)] = word(p[k]);
        return;
    }
    for (uint32_t i = threadIdx.x; i < span; i += kSThreads) s_cnt[i] = 0;
    __syncthreads();
    uint32_t at[kSItems];
#pragma unroll
    for (int k = 0; k < kSItems; ++k)
        if (p[k] != kNone) at[k] = atomicAdd(&s_cnt[(uint32_t)(p[k] >> 36) - lo], 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < span; i += kSThreads) {
        const uint32_t c = s_cnt[i];
        if (c) s_cnt[i] = atomicAdd(&cursor[lo + i], c);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSItems; ++k)
        if (p[k] != kNone) out[s_cnt[(uint32_t)(p[k] >> 36) - lo] + at[k]] = word(p[k]);
}

// ---- tiles ---------------------------------------------------------------------------------
constexpr uint32_t kTileBytes = 32768;  // tile buffer, at most
constexpr uint32_t kDirect = 1u << 18;  // looks at an edge from which a row block is written directly

template <int LOG2C, int kTThreads>
__global__ void __launch_bounds__(kTThreads)
k_count_tiles(const uint32_t* __restrict__ edges, const uint32_t* __restrict__ rb_end, uint32_t R,
              uint32_t words, uint32_t* __restrict__ indptr, Heavy hv)
{
    extern __shared__ uint32_t s_bm[];
    __shared__ uint32_t s_red[kTThreads / kWarp];
    for (uint32_t i = threadIdx.x; i < words; i += kTThreads) s_bm[i] = 0;
    __syncthreads();
    for (uint32_t I = blockIdx.x; I < R; I += gridDim.x) {
        const uint32_t e0 = I ? rb_end[I - 1] : 0u, end = rb_end[I];
        const bool heavy = end - e0 > hv.limit;
        const uint32_t e1 = heavy ? e0 : end;
        uint32_t mine = 0;
        for (uint32_t e = e0 + threadIdx.x; e < e1; e += kTThreads) {
            const uint32_t cb = (edges[e] & 0x0fffffffu) >> LOG2C;
            const uint32_t bit = 1u << (cb & 31u);
            // read first: most edges of a dense row block find their bit set
            if (!(*(volatile uint32_t*)&s_bm[cb >> 5] & bit)) mine += !(atomicOr(&s_bm[cb >> 5], bit) & bit);
        }
        mine = __reduce_add_sync(kFull, mine);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (int w = 0; w < kTThreads / kWarp; ++w) t += s_red[w];
            if (!heavy) {
                indptr[I] = t;
            } else {
                const uint32_t at = atomicAdd(hv.count, 1u);
                if (at < hv.most) {
                    hv.list[at] = I;
                    hv.done[at] = 0;
                }
            }
        }
        for (uint32_t e = e0 + threadIdx.x; e < e1; e += kTThreads)
            s_bm[((edges[e] & 0x0fffffffu) >> LOG2C) >> 5] = 0;
        __syncthreads();
    }
}

template <int LOG2C, int kTThreads>
__global__ void __launch_bounds__(kTThreads)
k_write_tiles(const uint32_t* __restrict__ edges, const uint32_t* __restrict__ rb_end, uint32_t R,
              uint32_t words, const uint32_t* __restrict__ indptr, const unsigned long long* __restrict__ d_tiles, uint32_t cap,
              uint32_t* __restrict__ indices, uint32_t* __restrict__ row_indices, uint4* __restrict__ blocks,
              uint32_t* __restrict__ rowmask, uint32_t NT, uint32_t heavy_limit)
{
    if (*d_tiles > cap) return;  // more tiles than the arrays hold: the builder redoes this step
    constexpr int C = 1 << LOG2C;
    constexpr int WPR = C / 32, TW = 16 * WPR;
    extern __shared__ __align__(16) uint32_t s_all[];
    uint32_t* s_tile = s_all;                                      // NT * TW words
    uint32_t* s_bm = s_all + NT * TW;                              // words (whole fours)
    uint32_t* s_pre = s_bm + words;                                // words: tiles before each word
    uint32_t* s_mask = s_pre + words;                              // NT row masks
    __shared__ uint32_t s_scan[kTThreads / kWarp];
    // a tile and its mask
    auto zero = [&](uint32_t n) {
        for (uint32_t i = threadIdx.x; i < n * (TW / 4); i += kTThreads)
            reinterpret_cast<uint4*>(s_tile)[i] = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t i = threadIdx.x; i < n; i += kTThreads) s_mask[i] = 0u;
    };
    for (uint32_t i = threadIdx.x; i < words; i += kTThreads) s_bm[i] = 0;
    __syncthreads();
    // A row block's first kHeld * kTThreads edges are held in registers (for both looks at
    // them), loaded while the row block before is written; so are its bounds one earlier.
    constexpr int kHeld = 2;
    uint32_t I = blockIdx.x;
    uint32_t e0 = 0, e1 = 0, t0 = 0, t1 = 0;
    auto bounds = [&](uint32_t i, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
        a = b = c = d = 0;
        if (i < R) {
            a = i ? rb_end[i - 1] : 0u;
            b = rb_end[i];
            c = indptr[i];
            d = indptr[i + 1];
        }
    };
    uint32_t held[kHeld];
    auto hold = [&](uint32_t a, uint32_t b) {
#pragma unroll
        for (int k = 0; k < kHeld; ++k) {
            const uint32_t e = a + k * kTThreads + threadIdx.x;
            held[k] = e < b ? edges[e] : 0u;
        }
    };
    bounds(I, e0, e1, t0, t1);
    hold(e0, e1);
    uint32_t ne0, ne1, nt0, nt1;
    for (; I < R; I += gridDim.x, e0 = ne0, e1 = ne1, t0 = nt0, t1 = nt1) {
        const uint32_t nt = t1 - t0;
        bounds(I + gridDim.x, ne0, ne1, nt0, nt1);
        if (nt == 0 || e1 - e0 > heavy_limit) {  // uniform for the CTA
            hold(ne0, ne1);
            continue;
        }
        auto each_edge = [&](auto f) {
#pragma unroll
            for (int k = 0; k < kHeld; ++k)
                if (e0 + k * kTThreads + threadIdx.x < e1) f(held[k]);
            for (uint32_t e = e0 + kHeld * kTThreads + threadIdx.x; e < e1; e += kTThreads) f(edges[e]);
        };
        each_edge([&](uint32_t x) {
            const uint32_t cb = (x & 0x0fffffffu) >> LOG2C;
            const uint32_t bit = 1u << (cb & 31u);
            if (!(*(volatile uint32_t*)&s_bm[cb >> 5] & bit)) atomicOr(&s_bm[cb >> 5], bit);
        });
        // the tile buffer, zeroed meanwhile
        zero(min(nt, NT));
        __syncthreads();
        // tile numbers: a popcount prefix over the words that can hold a bit (columns stay
        // below the row block's last row), a run of words per thread
        const uint32_t used = min(words, ((16u * I + 15u) >> LOG2C) / 32u + 1u);
        const uint32_t per = (used + 4 * kTThreads - 1) / (4 * kTThreads);  // in fours
        uint4* bm4 = reinterpret_cast<uint4*>(s_bm);
        uint4* pre4 = reinterpret_cast<uint4*>(s_pre);
        uint32_t cnt = 0;
        for (uint32_t q = threadIdx.x * per; q < (threadIdx.x + 1) * per && 4 * q < used; ++q) {
            const uint4 w = bm4[q];
            cnt += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
        }
        uint32_t total;
        uint32_t run = cta_exclusive_scan<kTThreads>(cnt, s_scan, total);
        for (uint32_t q = threadIdx.x * per; q < (threadIdx.x + 1) * per && 4 * q < used; ++q) {
            const uint4 w = bm4[q];
            uint4 p;
            p.x = run;
            p.y = p.x + __popc(w.x);
            p.z = p.y + __popc(w.y);
            p.w = p.z + __popc(w.z);
            run = p.w + __popc(w.w);
            pre4[q] = p;
        }
        __syncthreads();
        // One edge: its tile's number, the tile's word (ORed where `tile` says) and mask.
        auto place = [&](uint32_t x, uint32_t tb, uint32_t nb, uint32_t* tile, uint32_t* mask) {
            const uint32_t c = x & 0x0fffffffu;
            const uint32_t cb = c >> LOG2C;
            const uint32_t t = s_pre[cb >> 5] + __popc(s_bm[cb >> 5] & ((1u << (cb & 31u)) - 1u)) - tb;
            if (t >= nb) return;
            const uint32_t cl = c & (C - 1), r = x >> 28;
            // the edge that finds its word empty marks the row (16x128: its half), and the one
            // that finds the tile's mask empty names the tile
            if (atomicOr(&tile[(size_t)t * TW + r * WPR + (cl >> 5)], 1u << (cl & 31u)) == 0u &&
                atomicOr(&mask[t], 1u << (r + (C == 128 ? (cl & 64u) / 4u : 0u))) == 0u) {
                indices[t0 + tb + t] = cb;
                row_indices[t0 + tb + t] = I;
            }
        };
        // A hub row block (its edges would be looked at once per buffer of tiles) goes straight
        // to device memory.
        const bool direct = (uint64_t)(e1 - e0) * nt > (uint64_t)kDirect * NT;
        if (direct) {
            for (uint32_t i = threadIdx.x; i < nt * (TW / 4); i += kTThreads)
                blocks[(size_t)t0 * (TW / 4) + i] = make_uint4(0u, 0u, 0u, 0u);
            for (uint32_t i = threadIdx.x; i < nt; i += kTThreads) rowmask[t0 + i] = 0u;
            __threadfence();
            __syncthreads();
            uint32_t* tile = reinterpret_cast<uint32_t*>(blocks) + (size_t)t0 * TW;
            each_edge([&](uint32_t x) { place(x, 0, nt, tile, rowmask + t0); });
            hold(ne0, ne1);
            __syncthreads();
            for (uint32_t w = threadIdx.x; w < used; w += kTThreads) s_bm[w] = 0;
            __syncthreads();
        }
        for (uint32_t tb = 0; tb < nt && !direct; tb += NT) {
            const uint32_t nb = min(NT, nt - tb);
            if (tb) {
                zero(nb);
                __syncthreads();
            }
            each_edge([&](uint32_t x) { place(x, tb, nb, s_tile, s_mask); });
            if (tb + NT >= nt) hold(ne0, ne1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the bulk copy reads s_tile
            __syncthreads();
            // write them: the tiles by one bulk copy (whole 64- or 256-byte tiles, 16-byte
            // aligned on both sides), the masks by the threads
            if (threadIdx.x == 0) {
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                                 (uint64_t)__cvta_generic_to_global(blocks + (size_t)(t0 + tb) * (TW / 4))),
                             "r"((uint32_t)__cvta_generic_to_shared(s_tile)), "r"(nb * TW * 4u)
                             : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            for (uint32_t i = threadIdx.x; i < nb; i += kTThreads) rowmask[t0 + tb + i] = s_mask[i];
            if (tb + NT >= nt)
                for (uint32_t w = threadIdx.x; w < used; w += kTThreads) s_bm[w] = 0;
            // the copy has read the buffer before anyone writes it again
            if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- heavy row blocks ------------------------------------------------------------------------
constexpr int kHThreads = 512;

// The slices of the listed row blocks: f(h, I, first edge, end, slices of h) for this CTA's.
template <class F>
__device__ __forceinline__ void each_slice(const Heavy& hv, const uint32_t* __restrict__ rb_end, F f)
{
    static_assert(kMaxHeavy == kHThreads, "a row block per thread");
    __shared__ uint32_t s_first[kMaxHeavy];  // slices of the row blocks before
    __shared__ uint32_t s_scan[kHThreads / kWarp];
    const uint32_t n = min(*hv.count, hv.most);
    if (n == 0) return;
    auto slices = [&](uint32_t h) -> uint32_t {
        if (h >= n) return 0u;
        const uint32_t I = hv.list[h];
        return (rb_end[I] - (I ? rb_end[I - 1] : 0u) + kSlice - 1) / kSlice;
    };
    uint32_t total;
    s_first[threadIdx.x] = cta_exclusive_scan<kHThreads>(slices(threadIdx.x), s_scan, total);
    __syncthreads();
    for (uint32_t s = blockIdx.x; s < total; s += gridDim.x) {
        uint32_t h = 0, end = n;  // the last row block with s_first <= s
        while (end - h > 1) {
            const uint32_t mid = (h + end) >> 1;
            if (s_first[mid] <= s) h = mid;
            else end = mid;
        }
        const uint32_t I = hv.list[h];
        const uint32_t e = (I ? rb_end[I - 1] : 0u) + (s - s_first[h]) * kSlice;
        f(h, I, e, min(e + kSlice, rb_end[I]), (h + 1 < n ? s_first[h + 1] : total) - s_first[h]);
    }
}

// The bitmaps of the row blocks' column blocks; a row block's last slice counts its tiles.
template <int LOG2C>
__global__ void __launch_bounds__(kHThreads)
k_heavy_mark(const uint32_t* __restrict__ edges, const uint32_t* __restrict__ rb_end, uint32_t words, Heavy hv,
             uint32_t* __restrict__ indptr)
{
    extern __shared__ uint32_t s_bm[];
    __shared__ uint32_t s_red[kHThreads / kWarp];
    __shared__ int s_last;
    each_slice(hv, rb_end, [&](uint32_t h, uint32_t I, uint32_t e0, uint32_t e1, uint32_t slices) {
        uint32_t* bm = hv.bm + (size_t)h * words;
        for (uint32_t w = threadIdx.x; w < words; w += kHThreads) s_bm[w] = 0;
        __syncthreads();
        for (uint32_t e = e0 + threadIdx.x; e < e1; e += kHThreads) {
            const uint32_t cb = (edges[e] & 0x0fffffffu) >> LOG2C;
            const uint32_t bit = 1u << (cb & 31u);
            if (!(*(volatile uint32_t*)&s_bm[cb >> 5] & bit)) atomicOr(&s_bm[cb >> 5], bit);
        }
        __syncthreads();
        for (uint32_t w = threadIdx.x; w < words; w += kHThreads)
            if (s_bm[w]) atomicOr(&bm[w], s_bm[w]);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(&hv.done[h], 1u) == slices - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            uint32_t sum = 0;
            for (uint32_t w = threadIdx.x; w < words; w += kHThreads) sum += __popc(__ldcg(&bm[w]));
            uint32_t total;
            cta_exclusive_scan<kHThreads>(sum, s_red, total);
            if (threadIdx.x == 0) indptr[I] = total;
        }
        __syncthreads();
    });
}

constexpr int kEThreads = 256;
constexpr uint32_t kSegWords = 128;  // words a CTA of k_heavy_emit takes

// Tile numbers before each word, indices and row_indices; tiles and masks zeroed.
__global__ void __launch_bounds__(kEThreads)
k_heavy_emit(uint32_t words, Heavy hv, const uint32_t* __restrict__ indptr,
             const unsigned long long* __restrict__ d_tiles, uint32_t cap, uint32_t vec4,
             uint32_t* __restrict__ indices, uint32_t* __restrict__ row_indices, uint4* __restrict__ blocks,
             uint32_t* __restrict__ rowmask)
{
    if (*d_tiles > cap) return;
    __shared__ uint32_t s_scan[kEThreads / kWarp];
    const uint32_t segs = (words + kSegWords - 1) / kSegWords;
    const uint32_t n = min(*hv.count, hv.most);
    for (uint32_t u = blockIdx.x; u < n * segs; u += gridDim.x) {
        const uint32_t h = u / segs, w0 = (u % segs) * kSegWords;
        const uint32_t I = hv.list[h];
        const uint32_t* bm = hv.bm + (size_t)h * words;
        uint32_t sum = 0;
        for (uint32_t w = threadIdx.x; w < w0; w += kEThreads) sum += __popc(bm[w]);
        uint32_t base, total;
        cta_exclusive_scan<kEThreads>(sum, s_scan, base);
        const uint32_t w = w0 + threadIdx.x;
        uint32_t x = threadIdx.x < kSegWords && w < words ? bm[w] : 0u;
        uint32_t t = base + cta_exclusive_scan<kEThreads>(__popc(x), s_scan, total);
        if (threadIdx.x < kSegWords && w < words) hv.pre[(size_t)h * words + w] = t;
        const size_t t0 = indptr[I];
        for (; x; x &= x - 1, ++t) {
            indices[t0 + t] = w * 32 + (__ffs(x) - 1);
            row_indices[t0 + t] = I;
        }
        for (uint32_t i = threadIdx.x; i < total; i += kEThreads) rowmask[t0 + base + i] = 0u;
        for (size_t i = threadIdx.x; i < (size_t)total * vec4; i += kEThreads)
            blocks[(t0 + base) * vec4 + i] = make_uint4(0u, 0u, 0u, 0u);
    }
}

template <int LOG2C>
__global__ void __launch_bounds__(kHThreads)
k_heavy_fill(const uint32_t* __restrict__ edges, const uint32_t* __restrict__ rb_end, uint32_t words, Heavy hv,
             const uint32_t* __restrict__ indptr, const unsigned long long* __restrict__ d_tiles, uint32_t cap,
             uint32_t* __restrict__ blocks, uint32_t* __restrict__ rowmask)
{
    if (*d_tiles > cap) return;
    constexpr int C = 1 << LOG2C, WPR = C / 32, TW = 16 * WPR, U = 4;
    each_slice(hv, rb_end, [&](uint32_t h, uint32_t I, uint32_t e0, uint32_t e1, uint32_t) {
        const uint32_t* bm = hv.bm + (size_t)h * words;
        const uint32_t* pre = hv.pre + (size_t)h * words;
        const size_t t0 = indptr[I];
        for (uint32_t e = e0 + threadIdx.x; e < e1; e += U * kHThreads) {
            uint32_t x[U], old[U];
            size_t t[U];
#pragma unroll
            for (int k = 0; k < U; ++k) x[k] = e + k * kHThreads < e1 ? edges[e + k * kHThreads] : 0u;
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const uint32_t cb = (x[k] & 0x0fffffffu) >> LOG2C;
                t[k] = t0 + pre[cb >> 5] + __popc(bm[cb >> 5] & ((1u << (cb & 31u)) - 1u));
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const uint32_t cl = x[k] & (C - 1), r = x[k] >> 28;
                old[k] = 1u;
                if (e + k * kHThreads < e1) old[k] = atomicOr(&blocks[t[k] * TW + r * WPR + (cl >> 5)], 1u << (cl & 31u));
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const uint32_t cl = x[k] & (C - 1), r = x[k] >> 28;
                if (old[k] == 0u) atomicOr(&rowmask[t[k]], 1u << (r + (C == 128 ? (cl & 64u) / 4u : 0u)));
            }
        }
    });
}

}  // namespace gp

// Row bits below a bucket: at most kBuckets buckets of whole row blocks.
static int bucket_shift(int64_t rows)
{
    int s = 4;
    while (((rows - 1) >> s) >= gp::kBuckets) ++s;
    return s;
}

// Threads of a row block's CTA: one warp where the row blocks average at most 96 edges (a grid
// of 7 points per vertex, 48 edges a row block: k_write_tiles 273 us with four warps, 190 with
// one, k_count_tiles 93 / 65), four above (R-MAT scale 22 in degree order averages 256).
static int row_block_threads(int64_t m, uint32_t R) { return m <= 96ll * R ? 32 : 128; }

// Whether the grouped builder takes a matrix of n columns in col_blocks column blocks.
bool group_possible(int64_t n, uint64_t col_blocks)
{
    return n > 0 && n <= (1ll << 28) && (col_blocks + 31) / 32 <= gp::kMaxWords;
}

// Buckets, row-block ends, a sum; then the heavy row blocks' lists and bitmaps.
static size_t group_front_words(uint32_t R) { return 3 * (size_t)gp::kBuckets + 1 + (size_t)R + 3; }
static uint32_t bitmap_row_words(uint64_t col_blocks) { return (uint32_t)((col_blocks + 31) / 32); }

size_t group_scratch_words(uint32_t R, int64_t m, uint64_t col_blocks)
{
    return group_front_words(R) + 1 + 2 * (size_t)gp::kMaxHeavy +
           2 * (size_t)gp::heavy_most(m) * bitmap_row_words(col_blocks);
}

// balanced: no row block has a share of the edges that is worth slices; none is heavy.
static gp::Heavy heavy_of(uint32_t* scratch, uint32_t R, int64_t m, uint64_t col_blocks, bool balanced)
{
    uint32_t* at = scratch + group_front_words(R);
    gp::Heavy h{};
    h.count = at;
    h.list = at + 1;
    h.done = h.list + gp::kMaxHeavy;
    h.bm = h.done + gp::kMaxHeavy;
    h.most = balanced ? 0u : gp::heavy_most(m);
    h.pre = h.bm + (size_t)h.most * bitmap_row_words(col_blocks);
    h.limit = balanced ? 0xffffffffu : gp::heavy_edges(m);
    return h;
}

// The edges grouped by row block and the row blocks' tile counts scanned into indptr.
// pairs: m uint64 (only written with rank); grouped: m uint64 of scratch whose
// contents end up in `edges` (m words, may share memory with pairs); balanced: see heavy_of; scratch:
// group_scratch_words(R, m, col_blocks); bsum: scan scratch of R words.  Writes meta[kMetaBad] and
// meta[kMetaTiles].
int group_edges(const int32_t* src, const int32_t* dst, int64_t m, int32_t n,
                const int32_t* rank, bool balanced, int tile_cols, uint64_t col_blocks, uint64_t* pairs,
                uint64_t* grouped, uint32_t* edges, uint32_t* scratch, uint32_t* indptr, uint32_t* bsum,
                unsigned long long* meta, cudaStream_t s)
{
    const uint32_t R = (uint32_t)(((int64_t)n + 15) / 16);
    uint32_t* hist = scratch;
    uint32_t* cursor = scratch + gp::kBuckets;
    uint32_t* base = cursor + gp::kBuckets;
    uint32_t* rb_end = base + gp::kBuckets + 1;  // offsets at first, then (moved on) ends
    unsigned long long* sum = reinterpret_cast<unsigned long long*>(scratch + (group_front_words(R) - 2) / 2 * 2);
    const gp::Heavy hv = heavy_of(scratch, R, m, col_blocks, balanced);
    const int shift = bucket_shift(n);
    if (cudaMemsetAsync(hist, 0, sizeof(uint32_t) * gp::kBuckets, s) != cudaSuccess) return BTC_E_CUDA;
    const bool store = rank != nullptr;
    const int ogrid = (int)std::min<int64_t>((m + 8 * gp::kOThreads - 1) / (8 * gp::kOThreads),
                                             4 * (int64_t)device_sm_count());
    if (m > 0)
        gp::k_orient<<<ogrid, gp::kOThreads, 0, s>>>(src, dst, m, n, rank, shift,
                                                     store ? pairs : nullptr, hist, meta + kMetaBad);
    gp::k_bucket_scan<<<1, 1024, 0, s>>>(hist, base, cursor, hv.count);
    static std::atomic<unsigned long long> scatter_ok[kMaxDevices];
    if (!allow_dynamic_smem(reinterpret_cast<const void*>(&gp::k_scatter), sizeof(gp::ScatterSmem), scatter_ok))
        return BTC_E_CUDA;
    if (m > 0)
        gp::k_scatter<<<(unsigned)((m + gp::kSTile - 1) / gp::kSTile), gp::kSThreads, sizeof(gp::ScatterSmem), s>>>(
            store ? pairs : nullptr, src, dst, m, n, shift, cursor, grouped);
    if (cudaMemsetAsync(rb_end, 0, sizeof(uint32_t) * (size_t)R, s) != cudaSuccess) return BTC_E_CUDA;
    const unsigned stiles = (unsigned)((m + gp::kSTile - 1) / gp::kSTile);
    const uint32_t* d_m = base + gp::kBuckets;
    if (m > 0)
        gp::k_rb_count<<<stiles, gp::kSThreads, 0, s>>>(grouped, d_m, rb_end, hv.bm,
                                                        hv.most * bitmap_row_words(col_blocks));
    BTC_TRY(launch_scan_u32(rb_end, R, bsum, sum, s));
    if (m > 0) gp::k_rb_scatter<<<stiles, gp::kSThreads, 0, s>>>(grouped, d_m, rb_end, edges);
    const uint32_t words = bitmap_row_words(col_blocks);
    const int threads = row_block_threads(m, R);
    const uint32_t grid = std::min<uint32_t>(R, 32u * device_sm_count() * (128 / threads));
    auto count = [&](auto kernel, auto mark) {
        kernel<<<grid, threads, 4 * words, s>>>(edges, rb_end, R, words, indptr, hv);
        if (hv.most)
            mark<<<2 * device_sm_count(), gp::kHThreads, 4 * words, s>>>(edges, rb_end, words, hv, indptr);
    };
    if (tile_cols == 128)
        count(threads == 32 ? gp::k_count_tiles<7, 32> : gp::k_count_tiles<7, 128>, gp::k_heavy_mark<7>);
    else
        count(threads == 32 ? gp::k_count_tiles<5, 32> : gp::k_count_tiles<5, 128>, gp::k_heavy_mark<5>);
    return launch_scan_u32(indptr, R, bsum, meta + kMetaTiles, s);
}

// Tiles, indices, row_indices and row masks from the grouped edges (indptr[R] set), against
// `cap` tiles: nothing when meta[kMetaTiles] is above it.
int group_write(int tile_cols, uint64_t col_blocks, int64_t m, uint32_t R, bool balanced,
                const uint32_t* edges, uint32_t* scratch, const uint32_t* indptr,
                const unsigned long long* meta, uint32_t cap, uint32_t* indices, uint32_t* row_indices,
                uint32_t* blocks, uint32_t* rowmask, uint32_t tiles_hint, cudaStream_t s)
{
    const uint32_t* rb_end = scratch + 3 * (size_t)gp::kBuckets + 1;
    const uint32_t words = (uint32_t)((col_blocks + 127) / 128 * 4);  // whole fours
    // tiles built at once: one and a half times the average row block's, in 4 KB (a mesh's
    // row blocks: more CTAs) up to 16 KB (16x128) or 32 KB (16x32); 8 KB cost R-MAT scale 22
    // 15%, 32 KB 20%
    const uint32_t tile_bytes = 2u * (uint32_t)tile_cols;
    uint32_t buf = 4096;
    const uint32_t buf_most = tile_cols == 128 ? gp::kTileBytes / 2 : gp::kTileBytes;
    while (buf < buf_most && (uint64_t)buf * R * 2 < 3ull * tiles_hint * tile_bytes) buf *= 2;
    const uint32_t NT = buf / tile_bytes;
    const size_t smem = buf + 4 * (size_t)NT + 8 * (size_t)words;
    const size_t most = gp::kTileBytes + 4 * (gp::kTileBytes / 64) + 8 * (size_t)gp::kMaxWords;
    static std::atomic<unsigned long long> ok[4][kMaxDevices];
    const int threads = row_block_threads(m, R);
    const uint32_t grid = std::min<uint32_t>(R, 32u * device_sm_count() * (128 / threads));
    const gp::Heavy hv = heavy_of(scratch, R, m, col_blocks, balanced);
    const uint32_t hwords = bitmap_row_words(col_blocks);
    auto write = [&](auto kernel, int which, auto fill) {
        if (!allow_dynamic_smem(reinterpret_cast<const void*>(kernel), most, ok[which])) return BTC_E_CUDA;
        kernel<<<grid, threads, smem, s>>>(edges, rb_end, R, words, indptr, meta + kMetaTiles, cap,
                                           indices, row_indices, reinterpret_cast<uint4*>(blocks), rowmask, NT,
                                           hv.limit);
        if (hv.most) {
            gp::k_heavy_emit<<<4 * device_sm_count(), gp::kEThreads, 0, s>>>(
                hwords, hv, indptr, meta + kMetaTiles, cap, tile_bytes / 16, indices, row_indices,
                reinterpret_cast<uint4*>(blocks), rowmask);
            fill<<<2 * device_sm_count(), gp::kHThreads, 0, s>>>(edges, rb_end, hwords, hv, indptr, meta + kMetaTiles,
                                                                 cap, blocks, rowmask);
        }
        return cudaGetLastError() == cudaSuccess ? BTC_OK : BTC_E_CUDA;
    };
    if (tile_cols == 128)
        return threads == 32 ? write(gp::k_write_tiles<7, 32>, 0, gp::k_heavy_fill<7>)
                             : write(gp::k_write_tiles<7, 128>, 1, gp::k_heavy_fill<7>);
    return threads == 32 ? write(gp::k_write_tiles<5, 32>, 2, gp::k_heavy_fill<5>)
                         : write(gp::k_write_tiles<5, 128>, 3, gp::k_heavy_fill<5>);
}

}  // namespace btc200
