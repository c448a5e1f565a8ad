// common.cuh -- shared definitions for the engine's CUDA sources (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <atomic>
#include <cstddef>
#include <cstdint>

#include "btc_c.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "this engine is written for sm_100a (B200) only"
#endif

namespace btc200 {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

// Status propagation for host code: evaluate a CUDA call, map failure to BTC_E_CUDA
// (or BTC_E_NOMEM for allocation failures) and return from the enclosing function.
#define BTC_CUDA_TRY(expr)                                                      \
    do {                                                                        \
        cudaError_t _e = (expr);                                                \
        if (_e != cudaSuccess) {                                                \
            ::btc200::note_cuda_error(_e, #expr, __FILE__, __LINE__);           \
            return _e == cudaErrorMemoryAllocation ? BTC_E_NOMEM : BTC_E_CUDA;  \
        }                                                                       \
    } while (0)

#define BTC_TRY(expr)                 \
    do {                              \
        int _s = (expr);              \
        if (_s != BTC_OK) return _s;  \
    } while (0)

void note_cuda_error(cudaError_t e, const char* what, const char* file, int line);

__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__host__ __device__ __forceinline__ int bit_length_u64(uint64_t x)
{
#ifdef __CUDA_ARCH__
    return x ? 64 - __clzll((long long)x) : 0;
#else
    return x ? 64 - __builtin_clzll(x) : 0;
#endif
}

__host__ __device__ __forceinline__ int log2_exact(int x)
{
    int k = 0;
    while ((1 << k) < x) ++k;
    return k;
}

// Device memory for handles and workspaces, from a pool the library keeps per device
// (devmem.cu): a cudaMalloc and cudaFree pair of a fresh allocation cost 0.1 to 2 ms here, a
// pair from the pool a few microseconds (a one-off build, count and free of an R-MAT scale
// 16 graph, 17 buffers: 5.3-8.6 ms before).  The memory can be used on any stream once the
// call returns.  dev_free does not wait: nothing may be using the memory any more.
cudaError_t dev_alloc(void** p, size_t bytes);
void dev_free(void* p);
// Waits for device `dev` (the current one when it is negative); the current device stays.  The
// owner of memory on one device may be destroyed while another is current (a finaliser runs on
// any thread), so a wait before a free names the memory's device.
cudaError_t wait_device(int dev);
// Waits for the device of the arrays (all on one, null ones among them) and frees them; a failed
// wait gives the memory up: something may still use it.
void free_arrays(void* const* arrays, int n);

// A zeroed slot of kHostSlotWords uint64 in pinned, mapped, portable host memory (nullptr
// without memory) of the current context, whose id is given with it, and its return: nothing may
// be writing to it any more.
constexpr size_t kHostSlotWords = 16;
unsigned long long* host_slot_alloc(unsigned long long* context);
void host_slot_free(unsigned long long* s, unsigned long long context);

// A grow-only device buffer.  reserve() keeps contents only when no reallocation
// happens; callers treat it as scratch.
struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
    // Stream-ordered allocation, for an owner that uses the buffer on one stream only:
    // with `pool` and `stream` set, a growth frees and allocates in that stream's order
    // (cudaFreeAsync / cudaMallocFromPoolAsync) instead of waiting for the whole device.
    // `pooled` and `device` record how and where the current allocation was made.
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    bool pooled = false;
    int device = -1;
    int reserve(size_t need)
    {
        if (need <= bytes && ptr) return BTC_OK;
        release();
        if (need == 0) return BTC_OK;
        size_t want = need + need / 8;  // headroom for slowly growing rebuilds
        if (allocate(want) != cudaSuccess) {
            cudaGetLastError();
            if (allocate(need) != cudaSuccess) {
                cudaGetLastError();
                ptr = nullptr;
                return BTC_E_NOMEM;
            }
            want = need;
        }
        bytes = want;
        return BTC_OK;
    }
    cudaError_t allocate(size_t b)
    {
        pooled = pool != nullptr && stream != nullptr;
        if (cudaGetDevice(&device) != cudaSuccess) device = -1;
        return pooled ? cudaMallocFromPoolAsync(&ptr, b, pool, stream) : dev_alloc(&ptr, b);
    }
    void release()
    {
        if (ptr && !pooled && wait_device(device) != cudaSuccess) {
            cudaGetLastError();  // something may still use it: the memory is given up
            ptr = nullptr;
        }
        release_idle();
    }
    // the same when nothing uses the buffer any more (the owner has waited)
    void release_idle()
    {
        if (ptr) {
            if (pooled) cudaFreeAsync(ptr, stream);
            else dev_free(ptr);
        }
        ptr = nullptr;
        bytes = 0;
    }
    // zeroes the first n bytes, ordered with the buffer's stream when it has one
    cudaError_t zero(size_t n) const
    {
        return pooled ? cudaMemsetAsync(ptr, 0, n, stream) : cudaMemset(ptr, 0, n);
    }
    template <class T>
    T* as() const { return static_cast<T*>(ptr); }
};

// Exclusive prefix of one value per thread over a CTA of kThreads (s_warp: a word per warp);
// `total` is the sum.  Every thread of the CTA calls it.
template <int kThreads>
__device__ __forceinline__ uint32_t cta_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t wbase = 0;
    total = 0;
    for (int w = 0; w < kThreads / kWarp; ++w) {
        const uint32_t x = s_warp[w];
        if (w < warp) wbase += x;
        total += x;
    }
    __syncthreads();
    return wbase + incl - v;
}

// ---------------------------------------------------------------------------
// Sort (radix.cu)
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096 keys per CTA tile
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;

inline size_t sort_tiles(size_t n) { return (n + kSortTile - 1) / kSortTile; }

// Scratch words needed by radix_sort_u64 for up to n keys.
size_t radix_scratch_words(size_t n);

// Stable LSD sort of keys[0, *d_count) by bits [lo_bit, hi_bit).  d_count lives in
// device memory (at most max_n); alt is a second buffer of max_n keys.  Returns the
// buffer holding the sorted keys (keys or alt).
uint64_t* radix_sort_u64(uint64_t* keys, uint64_t* alt, size_t max_n,
                         const unsigned long long* d_count, int lo_bit, int hi_bit,
                         uint32_t* scratch, cudaStream_t s, int* status);

// ---------------------------------------------------------------------------
// Build (build.cu)
// ---------------------------------------------------------------------------
struct BuildGeom {
    int32_t n;
    int tile_cols;      // C
    int log2c;          // log2(C)
    int payload_bits;   // 4 + log2(C): (row in tile, column in tile)
    int cb_bits;        // bits of the column-block id
    int t_bits;         // bits of the tile key (row block, column block)
    int32_t n_row_blocks;
    int64_t n_col_blocks;
};
BuildGeom make_geom(int32_t n, int tile_cols);

// ---------------------------------------------------------------------------
// Count (count.cu)
// ---------------------------------------------------------------------------
// One graph of a batch union: its rows, vertex ids and the part of the cell bitmap (and
// of the (cell word, tile prefix) pairs) that covers it.  The cell of union row block J and
// union column block K is word bm_off + (J - row_off) * wpr + ((K - cb_lo) >> 5), bit
// (K - cb_lo) & 31; a single graph is the one segment {0, n, 0, 0, words per row, 0, 0}.
struct GraphSeg {
    uint32_t row_off;  // first global row block
    int32_t n;         // vertices (local ids are in [0, n))
    uint32_t vbase;    // first global vertex id (16 * row_off)
    uint32_t cb_lo;    // first global column block of the graph's vertex range
    uint32_t wpr;      // bitmap words per row block
    uint32_t pad;
    uint64_t bm_off;   // first bitmap word of the graph
};

struct CountScratch {
    unsigned long long* partials;  // one per CTA of the persistent grid
    unsigned int* done;            // CTAs finished (reset to 0 by the last one)
    unsigned long long* work;      // tile queue head (reset to 0 by the last CTA)
    unsigned long long* result;    // where the final count lands
    unsigned long long* result2;   // optional second destination (nullable)
    // optional device alias of mapped pinned host memory that also receives the count
    // (written by the last CTA, no copy-engine hop)
    unsigned long long* result_host = nullptr;
    // A count behind an enqueued build (build_meta) whose tiles the host cannot guess is launched for
    // few and for many: the launch whose bounds the tiles are outside of leaves everything as it is.
    unsigned long long tiles_from = 0, tiles_below = ~0ull;
};

int count_grid_size(int tile_cols);
// graph_rows / graph_counts (nullable): per-graph attribution for batches; graph g
// owns row blocks [graph_rows[g], graph_rows[g+1]) and its count is added to
// graph_counts[g] (which the caller zeroes).
int launch_count(int tile_cols, const uint32_t* indptr, const uint32_t* indices,
                 const uint32_t* row_indices, const uint32_t* blocks, uint32_t num_tiles,
                 int32_t n_row_blocks, int tau, CountScratch scr, cudaStream_t s,
                 const uint32_t* graph_rows = nullptr, uint32_t num_graphs = 0,
                 unsigned long long* graph_counts = nullptr, const uint32_t* rowmask = nullptr,
                 const uint2* cellpp = nullptr,
                 uint64_t cell_wpr = 0, const unsigned long long* row_max = nullptr,
                 uint32_t tile_begin = 0, uint32_t tile_end = 0xffffffffu,
                 const unsigned long long* build_meta = nullptr, uint32_t tiles_hint = 0,
                 const uint32_t* row_off = nullptr, const uint2* row_ent = nullptr,
                 bool dense_tiles = false, const GraphSeg* segs = nullptr);

// rowmask[t] bit r = tile t's row r has a bit -- in 16x128 tiles in its first 64 columns,
// and bit 16 + r in its last 64 (fold_rows joins them) -- for t < T = *d_tiles (T = cap when d_tiles
// is null) when T >= 8 * n_row_blocks (the heavy count variant's condition), and
// *row_max = max(*row_max, the most tiles in one row block), which picks the count
// kernel's schedule (the caller zeroes it).  Runs after the tiles are filled.  Writes
// nothing when T > cap (the tile arrays overflowed).
// masks = false: only *row_max (the bitmap builder's fill pass sets the masks itself);
// always = true: masks whatever T is (the row store reads them).
__host__ __device__ __forceinline__ uint32_t fold_rows(uint32_t m) { return (m | (m >> 16)) & 0xFFFFu; }
int launch_rowmask(int tile_cols, const uint32_t* blocks, uint32_t cap,
                   const unsigned long long* d_tiles, const uint32_t* indptr, int32_t n_row_blocks,
                   uint32_t* rowmask, unsigned long long* row_max, cudaStream_t s, bool masks = true,
                   bool always = false);

// The rows of L in 64-column words (rowstore.cu), the streaming count kernel's operand.
constexpr uint32_t kRowChunk = 16;  // entries per chunk: a row is whole chunks
constexpr uint32_t kRowLanes = 8;   // words per chunk: entry i is in word i % 8, half i / 8
constexpr uint32_t kRowRun = 4;     // chunks per first_row entry
struct RowStore {
    uint32_t* off;        // 17 R: row r of row block I has chunks [off[17 I + r], off[17 I + r + 1])
    void* key;            // word: the two entries' column blocks (64 columns), 16 bits each,
                          // or 32 when the graph has more of them (row_store_wide)
    uint4* bits;          // word: the two entries' 64 bits each
    uint32_t* first_row;  // the row that holds chunk kRowRun b; row blocks hold whole runs, from
                          // chunk kRowRun on; chunk 0 is empty
};
// Whether column block ids need more than 16 bits: 16 n_row_blocks / 64 of them.
inline bool row_store_wide(int64_t n_row_blocks) { return (n_row_blocks + 3) / 4 > 0x10000; }
// Chunks that hold `entries` entries of a graph of R row blocks, at most.
inline uint64_t row_store_chunks(uint64_t entries, uint64_t R)
{
    const uint64_t rows = 16 * R < entries ? 16 * R : entries;  // rows with an entry
    const uint64_t blocks = R < entries ? R : entries;
    return kRowRun + (entries + rows * (kRowChunk - 1)) / kRowChunk + blocks * (kRowRun - 1);
}

// Sets *bad and *d_host (a mapped host word) when a Bit-BSR that the engine did not build is not
// one the row store and its count take: they are sized by 16 R columns (the count's table, the
// 16-bit keys) and need ascending column blocks.  A tile whose first column is at or past 16 R
// (a slab of rows of a wider matrix) is for the tile-wise kernel.
int launch_rowstore_check(int tile_cols, const uint32_t* indices, const uint32_t* row_indices, uint32_t T,
                          int32_t n_row_blocks, unsigned long long* bad, unsigned long long* d_host,
                          cudaStream_t s);
// *out += the set bits of mask[0, n).
int launch_mask_popcount(const uint32_t* mask, uint32_t n, unsigned long long* out, cudaStream_t s);
// Enqueues the row store of a Bit-BSR whose row masks exist (T = *d_tiles tiles, bounded by
// cap, or cap when d_tiles is null; nothing when T > cap or *d_tiles < least).  by_degree: the ids are in
// descending-degree order.  meta: the build's metadata slots (kMetaRowChunks zero: it counts the
// chunks handed out); also raises meta[kMetaRowMax] to the most tiles and meta[kMetaRowLong] to the
// most chunks in one row block.
int launch_rowstore(int tile_cols, const uint32_t* indptr, const uint32_t* indices, const uint32_t* blocks,
                    int32_t n_row_blocks, const uint32_t* rowmask, const unsigned long long* d_tiles,
                    uint32_t cap, bool by_degree, unsigned long long* meta, const RowStore& out,
                    cudaStream_t s, unsigned long long least = 0);

// The streaming count (count_stream.cu) of the sample tiles [tile_begin, tile_end), or of
// all of them with `whole`.  rs_chunks: the store's meta[kMetaRowChunks], with meta[kMetaRowLong]
// behind it.  max_col_blocks: the most 64-column blocks a row's columns can span.  lower: the
// matrix is a lower triangle (every handle's is; a caller's Bit-BSR need not be).  grid: the CTAs
// scr.partials has room for.
int stream_blocks_per_sm_max();
int launch_count_stream(const RowStore& rs, const unsigned long long* rs_chunks, int tile_cols,
                        int32_t n_row_blocks, uint32_t max_col_blocks, CountScratch scr,
                        const uint32_t* graph_rows, uint32_t num_graphs, unsigned long long* graph_counts,
                        const uint32_t* row_indices, const uint32_t* indices, uint32_t tile_begin, uint32_t tile_end, bool whole,
                        bool lower, const unsigned long long* build_meta, int grid, cudaStream_t s);

// Row index of the row-wise count kernel (rowindex.cu): for vertex u, ent[off[u],
// off[u+1]) lists (column block, tile) of the tiles whose row u % 16 holds a bit, in tile
// order.  Built when the row masks are (T >= 8 * n_row_blocks, T = *d_tiles or cap);
// tot: n_row_blocks words, bsum: ri_scan_blocks(n_row_blocks) words, total: one uint64 of
// scratch; off: 16 * n_row_blocks + 1 words; ent: ent_cap entries (>= the unique edges).
uint32_t ri_scan_blocks(uint32_t n_row_blocks);
int launch_rowindex(const uint32_t* indptr, const uint32_t* indices, int32_t n_row_blocks,
                    const uint32_t* rowmask, const unsigned long long* d_tiles, uint32_t cap,
                    uint32_t* tot, uint32_t* bsum, unsigned long long* total, uint32_t* off,
                    uint2* ent, uint64_t ent_cap, cudaStream_t s);

// The grouped builder (group.cu).  Degree-ordered edge lists from this length on are grouped by row
// block instead of marked and filled edge by edge: the tiles of a power-law graph this large do not
// stay in L2 between zeroing and filling (R-MAT scale 18, 4.2M draws: 0.71 ms against 0.73 a
// step; scale 19: 1.29 / 1.43; scale 22: build 8.7 -> 5.2 ms; scale 17: the same).  In
// natural order the bitmap stays: meshes and communities have small tile arrays (27-point
// mesh 100^3 0.61 ms against 0.69 grouped, 8 communities on 60,000 vertices 4.0 / 4.5) and hubs
// unbalance the row blocks (scale 18: 2.1 / 2.4); uniform graphs of
// more than 3M edges would gain (800,000 vertices, 6.4M edges: 1.9 / 1.35 ms), but nothing
// at hand tells them from a power-law graph.
constexpr int64_t kGroupEdges = 1 << 22;
bool group_possible(int64_t n, uint64_t col_blocks);
size_t group_scratch_words(uint32_t R, int64_t m, uint64_t col_blocks);
int group_edges(const int32_t* src, const int32_t* dst, int64_t m, int32_t n,
                const int32_t* rank, bool balanced, int tile_cols, uint64_t col_blocks, uint64_t* pairs,
                uint64_t* grouped, uint32_t* edges, uint32_t* scratch, uint32_t* indptr, uint32_t* bsum,
                unsigned long long* meta, cudaStream_t s);
int group_write(int tile_cols, uint64_t col_blocks, int64_t m, uint32_t R, bool balanced,
                const uint32_t* edges, uint32_t* scratch, const uint32_t* indptr,
                const unsigned long long* meta, uint32_t cap, uint32_t* indices, uint32_t* row_indices,
                uint32_t* blocks, uint32_t* rowmask, uint32_t tiles_hint, cudaStream_t s);
// indptr[R] = the tile count, the overflow flag and the host's status slots (bitmap.cu).
int launch_finish_tiles(uint32_t* indptr, int32_t R, unsigned long long* meta, uint32_t cap,
                        unsigned long long* host_meta, cudaStream_t s);
// Bits and number of up to 4,096 evenly spaced tiles (T > 0), to two words of mapped host memory.
int launch_sample_bits(int tile_cols, const uint32_t* blocks, uint32_t T, unsigned long long* d_host, cudaStream_t s);
// The (cell word, tile prefix) pairs of `words` words from the tiles, for a count that wants
// them after a build that made none.
int launch_cells(const uint32_t* indptr, const uint32_t* indices, const uint32_t* row_indices, uint32_t cap,
                 const unsigned long long* d_tiles, uint64_t words, uint64_t wpr, uint2* cellpp,
                 cudaStream_t s);

// Id locality of an edge list for the tile policy (policy.cu): sampled share of edges
// with |u - v| < 128 over the share uniform ids would give.  e_off / nv (nullable): the
// batch layout, each edge measured against its own graph's vertex count.  skewed (nullable): whether
// one row block of 16 vertices has about a 1,024th of the oriented edges or more, by the same sample.
constexpr uint32_t kPolicySamples = 1u << 16;
constexpr int32_t kPolicyNear = 128;  // |u - v| below this counts as local
// One sampled edge: is it local, and the chance that two uniform ids are (2^20 = 1).
__device__ __forceinline__ void policy_sample(int32_t u, int32_t v, int32_t n, unsigned long long& local,
                                              unsigned long long& expect)
{
    if (u == v || u < 0 || v < 0 || u >= n || v >= n) return;
    local += (u > v ? u - v : v - u) < kPolicyNear ? (1ull << 20) : 0ull;
    expect += n > 2 * kPolicyNear ? ((2ull * kPolicyNear - 1ull) << 20) / (unsigned long long)n : (1ull << 20);
}
// A locality of at least 16, as btc_tile_policy_from_features decides it (the sums stay below
// 2^37, so the quotient there rounds to 16 only where it is 16).
__device__ __forceinline__ bool policy_is_local(unsigned long long local, unsigned long long expect)
{
    return expect != 0 && local >= 16 * expect;
}
// Whether the average degree alone decides for 16x32 tiles.
bool policy_dense(int64_t m, int32_t n);

// The one-launch builder of small graphs (small.cu).
constexpr int kHostTileCols = 9;  // host slot: the width the policy picked
struct SmallBuild {
    const int32_t* src;
    const int32_t* dst;
    int64_t m;
    int32_t n;
    int tile_cols;       // 0: the policy's
    uint32_t* words;     // cell words (of 16x32 tiles where the width is open)
    uint32_t* counts;    // two per SM
    uint2* cellpp;
    uint32_t* indices;
    uint32_t* row_indices;
    uint32_t* indptr;
    uint32_t* blocks;
    uint32_t* rowmask;
    uint32_t cap128, cap32;
    unsigned long long* meta;
    unsigned long long* host;  // the device's address of the status slots
    unsigned long long* policy_sums;
    unsigned int* bar;
    int64_t step;
    uint32_t samples;
    uint32_t max_spins = 1u << 22;  // of a wait of one CTA for the others: seconds
};
// kNotLaunched: the device does not run that many CTAs together for this program (an SM limit, as
// a multi-process service sets it); nothing was enqueued.
constexpr int kNotLaunched = 1;
constexpr unsigned long long kGaveUp = 2;  // meta[kMetaOverflow] of a build whose wait ran out
int launch_build_small(const SmallBuild& b, cudaStream_t s);

struct PolicyWords {
    DevBuf dev;                          // two sums and a ticket
    DevBuf skew;                         // counters of the samples' row blocks, and the most
    unsigned long long* host = nullptr;  // a host slot
    unsigned long long host_context = 0;
    bool dirty = false;                  // a call did not come to its end
    void release()
    {
        if (host && wait_device(dev.ptr ? dev.device : skew.device) != cudaSuccess) {
            cudaGetLastError();
            host = nullptr;  // (something may still write to it)
            dev.release();
            skew.release();
        }
        dev.release_idle();
        skew.release_idle();
        host_slot_free(host, host_context);
        host = nullptr;
    }
};
int policy_locality(const int32_t* src, const int32_t* dst, int64_t m, int32_t n, bool on_host,
                    const int64_t* e_off, const int32_t* nv, uint32_t G, cudaStream_t s, PolicyWords& w,
                    double* L, bool* skewed = nullptr);
// btc_select_tile_policy with the caller's words.
// skewed (nullable): set where the sample is taken, else unchanged.
int policy_select(const int32_t* src, const int32_t* dst, int64_t m, int32_t n, uint32_t flags, cudaStream_t s,
                  PolicyWords& w, int* tile_cols, int* tau, int* skewed = nullptr);

// Device metadata slots of a build (uint64 each): valid keys, out-of-range flag, tile
// count, unique edges, sort length, longest row-block list, tile-capacity overflow flag,
// the chunk-scan ticket (CTAs of the chunk popcount that have finished), and of the row store the
// chunks handed out and the most that one row block has.
enum {
    kMetaValid = 0,
    kMetaBad = 1,
    kMetaTiles = 2,
    kMetaUniq = 3,
    kMetaN = 4,
    kMetaRowMax = 5,
    kMetaOverflow = 6,
    kMetaTicket = 7,
    kMetaRowChunks = 8,
    kMetaRowLong = 9,
    kMetaSlots = 10
};
static_assert(kMetaSlots <= kHostSlotWords, "a host slot holds the metadata");

__device__ __forceinline__ bool count_is_another(const CountScratch& scr, const unsigned long long* build_meta)
{
    return build_meta && (build_meta[kMetaTiles] < scr.tiles_from || build_meta[kMetaTiles] >= scr.tiles_below);
}

// Queue/completion words of the count kernel: done (u32) at byte 0, work (u64) at 8.
constexpr size_t kCountCtlBytes = 16;

int device_sm_count();
constexpr int kMaxDevices = 64;
// Lets a kernel take `bytes` of dynamic shared memory on the current device: an opt-in that is
// made once per device and context (done: the context it was made in, per device).
bool allow_dynamic_smem(const void* kernel, size_t bytes, std::atomic<unsigned long long>* done);
// Id of the calling thread's current context (0 when it cannot be read): a device reset
// gives the device a new one.
unsigned long long current_context_id();

}  // namespace btc200
