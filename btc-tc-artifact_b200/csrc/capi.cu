// capi.cu -- the C ABI (include/btc_c.h): handles, build pipeline, count calls and
// the reference-shaped struct surface.  Host code only; the builders' kernels live in bitmap.cu,
// group.cu, small.cu, build.cu and radix.cu, the counts' in count.cu, count_rows.cu and
// count_stream.cu.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>

#include "common.cuh"
#include "handle.cuh"

#include <algorithm>

namespace btc200 {

int launch_degree(const int32_t*, const int32_t*, int64_t, int32_t, uint32_t*, cudaStream_t);
int launch_rank_keys(const uint32_t*, int32_t, uint32_t, uint64_t*, cudaStream_t);
int launch_rank_scatter(const uint64_t*, int32_t, int32_t*, cudaStream_t);
int launch_make_keys(const BuildGeom&, const int32_t*, const int32_t*, int64_t, const int32_t*,
                     uint64_t*, unsigned long long*, cudaStream_t);
int launch_segment(const BuildGeom&, const uint64_t*, size_t, const unsigned long long*, uint32_t*,
                   unsigned long long*, cudaStream_t);
int launch_fill(const BuildGeom&, const uint64_t*, size_t, const unsigned long long*,
                const uint32_t*, uint32_t*, uint32_t*, uint32_t*, cudaStream_t);
uint64_t bitmap_words_per_row(const BuildGeom&);
size_t bitmap_chunks(uint64_t W);
int bitmap_mark_and_count(const BuildGeom&, const int32_t*, const int32_t*, int64_t, const int32_t*,
                          uint32_t*, uint32_t*, unsigned long long*, unsigned long long*, cudaStream_t);
int bitmap_emit_and_fill(const BuildGeom&, const int32_t*, const int32_t*, int64_t, const int32_t*,
                         const uint32_t*, const uint32_t*, uint2*, uint32_t*, uint32_t*, uint32_t*,
                         uint32_t*, unsigned long long*, uint32_t, unsigned long long*,
                         cudaStream_t, uint32_t*, bool, bool);
int launch_popcount_sum(int, const uint32_t*, uint64_t, unsigned long long*, cudaStream_t);
int launch_indptr(const uint32_t*, uint32_t, int32_t, uint32_t*, cudaStream_t);
int launch_density(int, const uint32_t*, uint32_t, unsigned long long*, cudaStream_t);
int launch_set_u64(unsigned long long* p, unsigned long long v, cudaStream_t s);

void note_cuda_error(cudaError_t e, const char* what, const char* file, int line)
{
    static const bool verbose = std::getenv("BTC_DEBUG") != nullptr;
    if (verbose)
        std::fprintf(stderr, "[btc] CUDA error %s (%s) at %s:%d: %s\n", cudaGetErrorName(e),
                     cudaGetErrorString(e), file, line, what);
}

int device_sm_count()
{
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cache[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        cache[dev] = v;
    }
    return cache[dev];
}

}  // namespace btc200

using namespace btc200;

// Engine's default dense/sparse switch.  A tile takes the binary tensor-core path
// when its popcount exceeds tau.
// Measured on sm_100a (policy.cu, the tau sweep): 16x128 tiles switch to the binary
// tensor core above 1024 bits (half full), 16x32 tiles above 64 (the reference's value).
int default_tau(int tile_cols) { return tile_cols == 128 ? 1024 : 64; }

// A row's walk costs the streaming count its neighbours' entries, however full they are; the
// row-wise kernel's tensor cores take a dense tile's 16 rows at once.  Measured on communities
// of 512 to 8,192 vertices, density 0.05 to 1, with and without edges between them (count
// only, streaming / row-wise, by edges per tile and tiles per row block).  16x32: 149 and 16.5
// 32 / 25 us, 99 and 16.5 44 / 46; 200 and 82 474 / 429, 160 and 82 376 / 429; 508 and 64 1.87 /
// 1.16 ms, 305 and 65 1.10 / 1.18; 56 and 117 0.47 / 1.64 ms, 12 and 212 0.24 / 1.68: the line
// is below every pair where the row-wise kernel wins.  16x128: 866 and 8.5 196 / 336 us, 1,156
// and 8.5 256 / 219, 596 and 16.5 0.58 / 1.51 ms, 1,191 and 16.5 1.10 / 1.05.
bool dense_graph(int tile_cols, int64_t m, uint32_t T, int64_t R)
{
    if (T == 0 || R <= 0) return false;
    const double per_tile = (double)m / (double)T;
    return tile_cols == 128 ? per_tile > 896.0 : per_tile > 64.0 + (double)T / (double)R;
}

// The streaming count takes a warp some 2 us a row however short it is (0.55 ns over the GPU); the
// row-wise kernel takes the 16 rows of a tile together.  Where a row block's tiles are few and
// shared, or its graph so small that no row block's list is long, the latter wins (count only,
// streaming / row-wise, 400,000 vertices in all): 16x32, graphs
// of 512 vertices and average degree 4 / 8 / 16 / 48 205 / 96, 253 / 115, 286 / 171, 371 / 336 us; of
// 1,024 247 / 143 (8), 281 / 226 (16), communities 309 / 207, R-MAT 279 / 227; of 2,048 245 / 184
// (8) but 281 / 308 (16) and R-MAT 288 / 354; 16x128, of 2,048 195 / 111 (4), 243 / 154 (8), 278 / 267
// (16), 402 / 706 (48).  A 27-point mesh 51^3 in degree order, 16x32: 142 / 61 us, 102^3 896 / 282.
// Nearly a tile an edge and at most five edges a vertex: uniform pairs, in whose lists nothing is
// long (131,072 vertices, average degree 4 97 / 58, 8 119 / 95, 16 146 / 188; R-MAT scale 20, edge
// factor 2, whose tiles hold 1.3 edges and up, 1.2 / 5.0 ms in natural order).
// widest: 64-column blocks of the widest graph; cells: the build makes the cell pairs, without which
// the tiles are searched for.  Below 1,024 row blocks both counts are launches.
static bool short_rows(int tile_cols, int64_t m, uint64_t T, int64_t R, uint32_t widest, bool cells)
{
    if (R < 1024) return false;
    const uint64_t r = (uint64_t)R, e = (uint64_t)m;
    const bool few = T < 16 * r;
    if (tile_cols == 32 && few && e >= 12 * T) return true;
    if (cells && R >= 4096 && 10 * e <= 11 * T && e <= 80 * r) return true;
    if (widest > 33) return false;  // 2,048 vertices
    return tile_cols == 32 ? few || e <= 80 * r : few && e <= 128 * r;
}

bool tiles_win(int tile_cols, int64_t m, uint32_t T, int64_t R, uint32_t widest, bool cells)
{
    return dense_graph(tile_cols, m, T, R) || short_rows(tile_cols, m, T, R, widest, cells);
}

static constexpr uint64_t kMaxEdges = (1ull << 32) - (uint64_t)kSortTile;

int ensure_count_scratch(btc_bitbsr* g)
{
    const int grid = count_grid_size(128) > count_grid_size(32) ? count_grid_size(128)
                                                                 : count_grid_size(32);
    const size_t need = sizeof(unsigned long long) * (size_t)grid;
    if (g->partials.bytes < need) BTC_TRY(g->partials.reserve(need));
    if (!g->done.ptr) {
        BTC_TRY(g->done.reserve(kCountCtlBytes));
        BTC_CUDA_TRY(g->done.zero(kCountCtlBytes));
    }
    if (!g->result.ptr) {
        BTC_TRY(g->result.reserve(sizeof(unsigned long long)));
        BTC_CUDA_TRY(g->result.zero(sizeof(unsigned long long)));
    }
    return BTC_OK;
}

// Pinned host slots the device writes directly (mapped): build status, tile count and
// the count result reach the host without a copy-engine hop.
int ensure_host_meta(btc_bitbsr* g)
{
    if (g->h_meta) return BTC_OK;
    unsigned long long* p = host_slot_alloc(&g->h_context);
    if (!p) return BTC_E_NOMEM;
    void* d = nullptr;
    if (cudaHostGetDevicePointer(&d, p, 0) != cudaSuccess) {
        cudaGetLastError();
        host_slot_free(p, g->h_context);
        return BTC_E_CUDA;
    }
    g->h_meta = p;
    g->d_hmeta = static_cast<unsigned long long*>(d);
    return BTC_OK;
}

// What one build enqueues, fixed before anything is enqueued (every buffer reserved).
struct BuildPlan {
    BuildGeom geom;
    const int32_t* src;  // caller's arrays (host with BTC_INPUT_ON_HOST)
    const int32_t* dst;
    const int32_t* d_src;  // device arrays the kernels read
    const int32_t* d_dst;
    int64_t m;
    int32_t n;
    uint32_t flags;
    bool use_bitmap;
    bool use_group;  // the grouped builder (group.cu)
    bool small;      // the one-launch builder (small.cu)
    bool open_width; // ... which picks the tile width
    uint32_t cap32, cap128;  // ... and the tiles the arrays hold at either
    uint64_t col_blocks;
    bool degree;
    uint64_t bm_words;
    uint32_t cap;  // > 0: the post-count steps run against this tile capacity
    bool heavy = false;      // the graph can average 8 tiles per row block: make its row masks
    bool row_store = false;  // ... and the streaming count's row store (rowstore.cu)
    bool open = false;       // ... both only if it does (by the device's tile count)
    bool row_index = false;  // ... or the row-wise kernel's index
};

// Graphs the one-launch builder takes, when the call waits: it saves about 17 us of launches
// and waits whatever the size (Erdos-Renyi, a step: 1,000 vertices 83 -> 66 us, 16,384 / 16
// 112 -> 91, 40,000 / 26, 520,000 draws 184 -> 168), which from 2^19 edges on is a few percent
// and on a mesh of 1.5M edges nothing.  An enqueued rebuild replays a graph, whose launches
// cost less than the barriers (16,384 / 16: 66 us, 71 by one launch).
static constexpr int64_t kSmallEdges = 1 << 19;
static constexpr size_t kSmallFirstBytes = 32ull << 20;
static bool small_possible(int64_t m, int32_t n)
{
    if (m <= 0 || m > kSmallEdges || n <= 0) return false;
    const BuildGeom g = make_geom(n, 32);
    return bitmap_words_per_row(g) * (uint64_t)g.n_row_blocks <= (1ull << 20);
}

// Only a graph with at least 8 edges per row block can average 8 tiles per row block (every
// tile holds an edge).
static bool row_store_possible(int64_t m, int32_t n_row_blocks)
{
    return n_row_blocks > 0 && m >= 8 * (int64_t)n_row_blocks && m < (int64_t)0xffffffffll;
}

RowStore row_store_of(const btc_bitbsr* g)
{
    return RowStore{g->rs_off.as<uint32_t>(), g->rs_key.ptr, g->rs_bits.as<uint4>(),
                    g->rs_first.as<uint32_t>()};
}

int reserve_row_store(btc_bitbsr* g, uint64_t entries)
{
    const uint64_t R = (uint64_t)g->n_row_blocks;
    BTC_TRY(g->rs_off.reserve(sizeof(uint32_t) * (17 * R + 1)));
    const uint64_t chunks = row_store_chunks(entries, R);
    if (chunks * kRowChunk > 0xffffffffull) return BTC_E_NOMEM;  // entries are numbered in 32 bits
    BTC_TRY(g->rs_key.reserve((row_store_wide(g->n_row_blocks) ? sizeof(uint2) : sizeof(uint32_t)) * kRowLanes * chunks));
    BTC_TRY(g->rs_bits.reserve(sizeof(uint4) * kRowLanes * chunks));
    return g->rs_first.reserve(sizeof(uint32_t) * (chunks / kRowRun + 1));
}

// The row store after the tiles and row masks (T = *d_tiles bounded by cap, or cap itself).
static int enqueue_row_store(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap,
                             bool by_degree, cudaStream_t s, bool open = false)
{
    return launch_rowstore(g->tile_cols, g->indptr.as<uint32_t>(), g->indices.as<uint32_t>(),
                           g->blocks.as<uint32_t>(), g->n_row_blocks, g->rowmask.as<uint32_t>(), d_tiles,
                           cap, by_degree, g->meta.as<unsigned long long>(), row_store_of(g), s,
                           open ? 8ull * (uint64_t)g->n_row_blocks : 0ull);
}

bool stream_capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
        cudaGetLastError();
        return true;  // (the legacy stream beside a global capture: allocate nothing)
    }
    return st != cudaStreamCaptureStatusNone;
}

// A buffer of at least `bytes`, without an allocation while a stream is capturing.
static bool room(DevBuf& b, size_t bytes, bool capturing)
{
    return capturing ? b.ptr && b.bytes >= bytes : b.reserve(bytes) == BTC_OK;
}

bool ensure_cells(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap, uint64_t words, uint64_t wpr,
                  cudaStream_t s)
{
    const bool capturing = stream_capturing(s), keep = !capturing && !d_tiles && !g->captured;
    if (g->cells && (keep || !g->cells_lazy)) return true;
    if (4 * words > 32ull * (uint64_t)g->input_edges + (64ull << 20) ||
        !room(g->prefix, sizeof(uint2) * (words ? words : 1), capturing))
        return false;
    const bool made = launch_cells(g->indptr.as<uint32_t>(), g->indices.as<uint32_t>(), g->row_indices.as<uint32_t>(),
                                   cap, d_tiles, words, wpr, g->prefix.as<uint2>(), s) == BTC_OK;
    if (keep) g->cells = g->cells_lazy = made;
    return made;
}

// The row index's buffers for up to `cap` tiles.
static bool row_index_room(btc_bitbsr* g, uint32_t cap, bool capturing)
{
    const uint64_t R = (uint64_t)g->n_row_blocks;
    const uint64_t ent = std::min<uint64_t>((uint64_t)g->input_edges, 16ull * cap);
    return row_store_possible(g->input_edges, g->n_row_blocks) &&
           room(g->row_off, sizeof(uint32_t) * (16 * R + 1), capturing) &&
           room(g->row_ent, sizeof(uint2) * (size_t)ent, capturing) &&
           room(g->row_tot, sizeof(uint32_t) * R, capturing) &&
           room(g->row_bsum, sizeof(unsigned long long) + sizeof(uint32_t) * ((size_t)ri_scan_blocks((uint32_t)R) + 1),
                capturing);
}

bool reserve_row_index(btc_bitbsr* g, uint32_t cap) { return row_index_room(g, cap, false); }

int enqueue_row_index(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap, cudaStream_t s)
{
    unsigned long long* total = g->row_bsum.as<unsigned long long>();
    return launch_rowindex(g->indptr.as<uint32_t>(), g->indices.as<uint32_t>(), g->n_row_blocks,
                           g->rowmask.as<uint32_t>(), d_tiles, cap, g->row_tot.as<uint32_t>(),
                           reinterpret_cast<uint32_t*>(total + 1), total, g->row_off.as<uint32_t>(),
                           g->row_ent.as<uint2>(), g->row_ent.bytes / sizeof(uint2), s);
}

bool ensure_row_index(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap, cudaStream_t s)
{
    if (g->index_built) return true;
    const bool capturing = stream_capturing(s), keep = !capturing && !d_tiles && !g->captured;
    if (g->row_index && keep) return true;
    if (!row_index_room(g, cap, capturing)) return false;
    const bool made = enqueue_row_index(g, d_tiles, cap, s) == BTC_OK;
    if (keep) g->row_index = made;
    return made;
}

// Tiles the handle's arrays hold room for at its width.  What a build reserves beside them follows
// this, not its own tiles: the next rebuild is enqueued against it, and is not to allocate then.
static uint32_t tile_capacity(const btc_bitbsr* g)
{
    const uint64_t c = std::min<uint64_t>(std::min<uint64_t>(g->indices.bytes, g->row_indices.bytes),
                                          g->rowmask.bytes) / 4;
    return (uint32_t)std::min<uint64_t>(std::min<uint64_t>(c, g->blocks.bytes / (2 * (size_t)g->tile_cols)), 0xffffffffull);
}

static int enqueue_group_write(btc_bitbsr* g, const BuildPlan& P, uint32_t cap, cudaStream_t s)
{
    return group_write(P.geom.tile_cols, P.col_blocks, P.m, (uint32_t)P.geom.n_row_blocks, !P.degree,
                       g->keys0.as<uint32_t>(), g->tile_base.as<uint32_t>(), g->indptr.as<uint32_t>(),
                       g->meta.as<unsigned long long>(), cap, g->indices.as<uint32_t>(),
                       g->row_indices.as<uint32_t>(), g->blocks.as<uint32_t>(), g->rowmask.as<uint32_t>(),
                       g->num_tiles, s);
}

// Enqueues the build up to the tile count (bitmap path) or up to the tile segmentation
// (radix path), and with plan.cap > 0 the whole bitmap build.  No waits, no allocation:
// this sequence is what a cached CUDA graph replays.
static int enqueue_build(btc_bitbsr* g, const BuildPlan& P, uint64_t** sorted_out, cudaStream_t s)
{
    const BuildGeom& geom = P.geom;
    unsigned long long* meta = g->meta.as<unsigned long long>();
    if (!P.small) BTC_CUDA_TRY(cudaMemsetAsync(meta, 0, sizeof(unsigned long long) * kMetaSlots, s));
    if ((P.flags & BTC_INPUT_ON_HOST) && P.m > 0) {
        BTC_CUDA_TRY(cudaMemcpyAsync(g->in_src.ptr, P.src, sizeof(int32_t) * (size_t)P.m,
                                     cudaMemcpyHostToDevice, s));
        BTC_CUDA_TRY(cudaMemcpyAsync(g->in_dst.ptr, P.dst, sizeof(int32_t) * (size_t)P.m,
                                     cudaMemcpyHostToDevice, s));
    }
    uint64_t* k0 = g->keys0.as<uint64_t>();
    uint64_t* k1 = g->keys1.as<uint64_t>();
    int st = BTC_OK;

    // ---- optional descending-degree relabel ---------------------------------
    const int32_t* rank = nullptr;
    if (P.degree) {
        const int32_t n = P.n;
        BTC_CUDA_TRY(cudaMemsetAsync(g->deg.ptr, 0, sizeof(uint32_t) * (size_t)n, s));
        BTC_TRY(launch_degree(P.d_src, P.d_dst, P.m, n, g->deg.as<uint32_t>(), s));
        int db = bit_length_u64(2ull * (uint64_t)P.m);  // degrees fit in db bits
        if (db > 32) db = 32;
        const uint32_t dmax = db >= 32 ? 0xffffffffu : ((1u << db) - 1u);
        BTC_TRY(launch_rank_keys(g->deg.as<uint32_t>(), n, dmax, k0, s));
        BTC_TRY(launch_set_u64(meta + kMetaN, (unsigned long long)n, s));
        uint64_t* sorted = radix_sort_u64(k0, k1, (size_t)n, meta + kMetaN, 32, 32 + (db ? db : 1),
                                          g->sort_scratch.as<uint32_t>(), s, &st);
        BTC_TRY(st);
        BTC_TRY(launch_rank_scatter(sorted, n, g->rank.as<int32_t>(), s));
        rank = g->rank.as<int32_t>();
    }

    if (P.small) {
        unsigned long long* w = g->small.as<unsigned long long>();
        SmallBuild b{P.d_src, P.d_dst, P.m, P.n, P.open_width ? 0 : geom.tile_cols, g->bitmap.as<uint32_t>(),
                     g->tile_base.as<uint32_t>(), g->prefix.as<uint2>(), g->indices.as<uint32_t>(),
                     g->row_indices.as<uint32_t>(), g->indptr.as<uint32_t>(), g->blocks.as<uint32_t>(),
                     g->rowmask.as<uint32_t>(), P.cap128, P.cap32, meta, g->d_hmeta, w,
                     reinterpret_cast<unsigned int*>(w + 2),
                     std::max<int64_t>(P.m / (int64_t)kPolicySamples, 1),
                     (uint32_t)std::min<int64_t>(P.m, (int64_t)kPolicySamples)};
        BTC_TRY(launch_build_small(b, s));
    } else if (P.use_bitmap) {
        BTC_TRY(bitmap_mark_and_count(geom, P.d_src, P.d_dst, P.m, rank, g->bitmap.as<uint32_t>(),
                                      g->tile_base.as<uint32_t>(), meta + kMetaBad,
                                      meta + kMetaTiles, s));
        if (P.cap) {
            BTC_TRY(bitmap_emit_and_fill(geom, P.d_src, P.d_dst, P.m, rank,
                                         g->bitmap.as<uint32_t>(), g->tile_base.as<uint32_t>(),
                                         g->prefix.as<uint2>(), g->indices.as<uint32_t>(),
                                         g->row_indices.as<uint32_t>(), g->indptr.as<uint32_t>(),
                                         g->blocks.as<uint32_t>(), meta, P.cap, g->d_hmeta, s,
                                         g->rowmask.as<uint32_t>(), P.heavy && !P.open,
                                         P.row_store && !P.open));
            // (the fill pass set the row masks, or found the longest row-block list)
            if (P.row_store) BTC_TRY(enqueue_row_store(g, meta + kMetaTiles, P.cap, P.degree, s, P.open));
            if (P.row_index) BTC_TRY(enqueue_row_index(g, meta + kMetaTiles, P.cap, s));
        }
    } else if (P.use_group) {
        const uint32_t R = (uint32_t)geom.n_row_blocks;
        uint32_t* scratch = g->tile_base.as<uint32_t>();
        BTC_TRY(group_edges(P.d_src, P.d_dst, P.m, P.n, rank, !P.degree, geom.tile_cols, P.col_blocks,
                            k0, k1, g->keys0.as<uint32_t>(), scratch, g->indptr.as<uint32_t>(),
                            scratch + group_scratch_words(R, P.m, P.col_blocks), meta, s));
        if (P.cap) {
            BTC_TRY(launch_finish_tiles(g->indptr.as<uint32_t>(), geom.n_row_blocks, meta, P.cap, g->d_hmeta, s));
            BTC_TRY(enqueue_group_write(g, P, P.cap, s));
            if (P.row_store) BTC_TRY(enqueue_row_store(g, meta + kMetaTiles, P.cap, P.degree, s, P.open));
            if (!P.row_store || P.open)
                BTC_TRY(launch_rowmask(geom.tile_cols, g->blocks.as<uint32_t>(), P.cap,
                                       meta + kMetaTiles, g->indptr.as<uint32_t>(), geom.n_row_blocks,
                                       g->rowmask.as<uint32_t>(), meta + kMetaRowMax, s, false));
        }
    } else {
        // ---- keys, sort, segmentation ---------------------------------------
        BTC_TRY(launch_make_keys(geom, P.d_src, P.d_dst, P.m, rank, k0, meta, s));
        uint64_t* sorted = radix_sort_u64(k0, k1, (size_t)P.m, meta + kMetaValid,
                                          geom.payload_bits, geom.payload_bits + geom.t_bits,
                                          g->sort_scratch.as<uint32_t>(), s, &st);
        BTC_TRY(st);
        BTC_TRY(launch_segment(geom, sorted, (size_t)P.m, meta + kMetaValid,
                               g->tile_base.as<uint32_t>(), meta + kMetaTiles, s));
        *sorted_out = sorted;
    }
    return BTC_OK;
}

// Everything an enqueued build reads or writes, plus its arguments: a graph captured
// from enqueue_build replays only under the same key.
static void build_key(const btc_bitbsr* g, const BuildPlan& P, BuildGraphKey* k)
{
    std::memset(k, 0, sizeof(*k));
    const void* w[] = {P.src, P.dst, g->meta.ptr, g->in_src.ptr, g->in_dst.ptr, g->keys0.ptr,
                       g->keys1.ptr, g->sort_scratch.ptr, g->deg.ptr, g->rank.ptr, g->bitmap.ptr,
                       g->prefix.ptr, g->tile_base.ptr, g->indices.ptr, g->row_indices.ptr,
                       g->indptr.ptr, g->blocks.ptr, g->rowmask.ptr, g->d_hmeta, g->rs_off.ptr,
                       g->rs_key.ptr, g->rs_bits.ptr, g->rs_first.ptr, g->row_off.ptr, g->row_ent.ptr,
                       g->row_tot.ptr, g->row_bsum.ptr};
    static_assert(sizeof(w) / sizeof(w[0]) == kBuildKeyPtrs, "key layout");
    for (int i = 0; i < kBuildKeyPtrs; ++i) k->ptr[i] = w[i];
    k->m = P.m;
    k->n = P.n;
    k->tile_cols = P.geom.tile_cols;
    k->flags = P.flags | (P.row_store ? 0x80000000u : 0u) | (P.use_group ? 0x40000000u : 0u) |
               (P.heavy ? 0x20000000u : 0u) | (P.row_index ? 0x10000000u : 0u) | (P.open ? 0x08000000u : 0u);
    k->cap = P.cap;
}

// Replays (or, on the second identical call, captures) the enqueued build as a CUDA
// graph: one launch instead of about a dozen.  Returns false when it did not enqueue.
static bool launch_build_graph(btc_bitbsr* g, const BuildPlan& P, cudaStream_t s)
{
    BuildGraphKey key;
    build_key(g, P, &key);
    if (g->graph_exec && std::memcmp(&key, &g->graph_key, sizeof(key)) == 0)
        return cudaGraphLaunch(g->graph_exec, s) == cudaSuccess;
    const bool repeat = std::memcmp(&key, &g->last_key, sizeof(key)) == 0;
    g->last_key = key;
    if (!repeat) return false;
    if (!g->capture_stream &&
        cudaStreamCreateWithFlags(&g->capture_stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(g->capture_stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    uint64_t* unused = nullptr;
    const int st = enqueue_build(g, P, &unused, g->capture_stream);
    const cudaError_t e = cudaStreamEndCapture(g->capture_stream, &graph);
    cudaGraphExec_t exec = nullptr;
    const bool ok = st == BTC_OK && e == cudaSuccess && graph &&
                    cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    if (!ok) {
        cudaGetLastError();
        if (exec) cudaGraphExecDestroy(exec);
        return false;
    }
    if (g->graph_exec) cudaGraphExecDestroy(g->graph_exec);
    g->graph_exec = exec;
    g->graph_key = key;
    return cudaGraphLaunch(g->graph_exec, s) == cudaSuccess;
}

// The cell bitmap (one bit per (row block, column block)) replaces the sort when it is small next
// to the edge list.
static bool bitmap_takes(const BuildGeom& geom, int64_t m)
{
    const uint64_t bytes = 4 * bitmap_words_per_row(geom) * (uint64_t)geom.n_row_blocks;
    return bytes <= (4ull << 30) && bytes <= 32ull * (uint64_t)m + (64ull << 20);
}

static int mark_tail(btc_bitbsr* g, cudaStream_t s)
{
    if (!g->meta_event)
        BTC_CUDA_TRY(cudaEventCreateWithFlags(&g->meta_event, cudaEventDisableTiming));
    BTC_CUDA_TRY(cudaEventRecord(g->meta_event, s));
    g->tail = true;
    return BTC_OK;
}

// (inside a capture the event is one from outside it)
static int wait_tail(btc_bitbsr* g, cudaStream_t s)
{
    if (g->tail)
        BTC_CUDA_TRY(cudaStreamWaitEvent(s, g->meta_event,
                                         stream_capturing(s) ? cudaEventWaitExternal : cudaEventWaitDefault));
    return BTC_OK;
}

// After a build whose tiles the host knows (row masks made where they average 8 per row block): the
// row store, or the row-wise kernel's index, or neither.
static int finish_known(btc_bitbsr* g, const BuildPlan& P, uint32_t widest, bool tiles_only, cudaStream_t s)
{
    const int64_t R = P.geom.n_row_blocks;
    const uint32_t T = g->num_tiles;
    g->heavy = !tiles_only && row_store_possible(P.m, P.geom.n_row_blocks) && (uint64_t)T >= 8ull * (uint64_t)R;
    g->row_store = g->heavy && !tiles_win(g->tile_cols, P.m, T, R, widest, P.use_bitmap) &&
                   reserve_row_store(g, std::min<uint64_t>((uint64_t)P.m, 32ull * tile_capacity(g))) == BTC_OK;
    if (g->row_store) BTC_TRY(enqueue_row_store(g, nullptr, T, P.degree, s));
    g->index_built = g->heavy && !g->row_store && P.use_bitmap && reserve_row_index(g, tile_capacity(g));
    if (g->index_built) BTC_TRY(enqueue_row_index(g, nullptr, T, s));
    return g->row_store || g->index_built ? mark_tail(g, s) : BTC_OK;
}

// tiles_only: the caller keeps the reference-shaped arrays alone, so no row store is made.
static int build_into(btc_bitbsr* g, const int32_t* src, const int32_t* dst, int64_t m, int32_t n,
                      int tile_cols, uint32_t flags, cudaStream_t s, bool tiles_only = false,
                      bool allow_small = true)
{
    if (n < 0 || m < 0 || (uint64_t)m > kMaxEdges) return BTC_E_INVAL;
    if (m > 0 && (!src || !dst)) return BTC_E_INVAL;
    if (flags & ~(BTC_INPUT_ON_HOST | BTC_ORIENT_DEGREE | BTC_BUILD_RADIX | BTC_BUILD_ASYNC))
        return BTC_E_INVAL;
    if (g->pending) resolve_build(g);  // an enqueued build still owns the buffers
    BTC_TRY(wait_tail(g, s));
    g->tail = false;
    // A small graph in natural order is built by one launch (small.cu), which also picks the
    // tile width where it is open: device input, and not the degree's to decide.
    bool small = allow_small && !(flags & (BTC_ORIENT_DEGREE | BTC_BUILD_RADIX | BTC_BUILD_ASYNC)) &&
                 small_possible(m, n);
    const bool open_width = small && tile_cols == 0 && !(flags & BTC_INPUT_ON_HOST) && !policy_dense(m, n);
    int skewed = -1;  // of the row blocks, where the policy's sample has told
    if (open_width) {
        tile_cols = 32;  // the larger cell grid, for the sizes below
    } else if (tile_cols == 0) {
        // the engine's tile policy (policy.cu).  With degree ordering it needs only m and
        // n; otherwise it samples the edges (a wait), which an enqueued rebuild skips by
        // keeping the handle's width.
        if (flags & BTC_ORIENT_DEGREE)
            BTC_TRY(btc_tile_policy_from_features(m, n, BTC_ORIENT_DEGREE, 0.0, &tile_cols, nullptr));
        else if ((flags & BTC_BUILD_ASYNC) && (g->tile_cols == 32 || g->tile_cols == 128))
            tile_cols = g->tile_cols;
        else
            BTC_TRY(policy_select(src, dst, m, n, flags & BTC_INPUT_ON_HOST, s, g->policy, &tile_cols, nullptr,
                                  bitmap_takes(make_geom(n, 32), m) ? nullptr : &skewed));
    }
    if (tile_cols != 32 && tile_cols != 128) return BTC_E_INVAL;
    BTC_CUDA_TRY(cudaGetDevice(&g->device));

    BuildPlan P{};
    P.geom = make_geom(n, tile_cols);
    const BuildGeom& geom = P.geom;
    // What an enqueued build cannot know: the previous graph of this handle, when it had the same
    // geometry, predicts whether this one averages 8 or more tiles per row block (the row store's
    // condition) and, with its tiles, whether the tile kernels count it faster than a row store does
    const uint32_t widest = ((uint32_t)n + 63) / 64;
    const bool prev_same = g->tile_cols == tile_cols && g->n_row_blocks == geom.n_row_blocks;
    const bool prev_light = g->num_tiles > 0 && (uint64_t)g->num_tiles < 8ull * (uint64_t)g->n_row_blocks;
    const uint32_t prev_tiles = g->num_tiles;
    g->tile_cols = tile_cols;
    g->n = n;
    g->n_row_blocks = geom.n_row_blocks;
    g->input_edges = m;
    g->edges_known = false;
    g->num_edges = 0;

    // ---- reserve every buffer the enqueued steps use ---------------------------
    BTC_TRY(ensure_host_meta(g));
    BTC_TRY(g->meta.reserve(sizeof(unsigned long long) * kMetaSlots));
    unsigned long long* meta = g->meta.as<unsigned long long>();
    P.src = src;
    P.dst = dst;
    P.d_src = src;
    P.d_dst = dst;
    P.m = m;
    P.n = n;
    P.flags = flags;
    if ((flags & BTC_INPUT_ON_HOST) && m > 0) {
        BTC_TRY(g->in_src.reserve(sizeof(int32_t) * (size_t)m));
        BTC_TRY(g->in_dst.reserve(sizeof(int32_t) * (size_t)m));
        P.d_src = g->in_src.as<int32_t>();
        P.d_dst = g->in_dst.as<int32_t>();
    }
    P.bm_words = bitmap_words_per_row(geom) * (uint64_t)geom.n_row_blocks;
    P.use_bitmap = !(flags & BTC_BUILD_RADIX) && bitmap_takes(geom, m);
    small = small && P.use_bitmap;
    // An enqueued build is one that the bitmap takes, whichever builder then runs; on any other
    // graph the call waits, and grows the arrays where they are too small.
    const bool enqueued = (flags & BTC_BUILD_ASYNC) && P.use_bitmap;
    // Large edge lists are grouped by row block instead of marked and filled edge by edge
    // (see kGroupEdges), and so is what the bitmap does not take.
    P.col_blocks = (uint64_t)geom.n_col_blocks;
    P.degree = (flags & BTC_ORIENT_DEGREE) && n > 0;
    // (the first of the large buffers: the time of the degree count's atomics differs by up to a
    // fifth with where its words lie, which is not to follow from the others' sizes)
    if (P.degree) {
        BTC_TRY(g->deg.reserve(sizeof(uint32_t) * (size_t)n));
        BTC_TRY(g->rank.reserve(sizeof(int32_t) * (size_t)n));
    }
    P.use_group = !(flags & BTC_BUILD_RADIX) && group_possible(n, P.col_blocks) &&
                  (!P.use_bitmap || (P.degree && m >= kGroupEdges));
    // In natural order a hub's row block may have any share of the edges, and its tiles are too much
    // for a CTA: such a list is sorted.
    if (P.use_group && !P.degree) {
        if (skewed < 0) {
            bool is = false;
            double unused = 0.0;
            BTC_TRY(policy_locality(src, dst, m, n, (flags & BTC_INPUT_ON_HOST) != 0, nullptr, nullptr, 0, s,
                                    g->policy, &unused, &is));
            skewed = is;
        }
        if (skewed) P.use_group = false;
    }
    if (P.use_group) {
        const uint64_t R = (uint64_t)geom.n_row_blocks;
        if (g->keys0.reserve(sizeof(uint64_t) * (size_t)(m ? m : 1)) != BTC_OK ||
            g->keys1.reserve(sizeof(uint64_t) * (size_t)(m ? m : 1)) != BTC_OK ||
            g->tile_base.reserve(sizeof(uint32_t) * (group_scratch_words((uint32_t)R, m, P.col_blocks) +
                                                     ri_scan_blocks((uint32_t)R) + 1)) != BTC_OK) {
            if (!P.use_bitmap) return BTC_E_NOMEM;
            P.use_group = false;  // the bitmap may still fit
        }
        if (P.use_group) P.use_bitmap = false;
    }
    g->cells = P.use_bitmap;
    g->heavy = g->row_store = g->row_index = g->cells_lazy = g->index_built = false;
    if ((flags & BTC_BUILD_ASYNC) && stream_capturing(s)) g->captured = true;
    size_t key_cap = P.use_bitmap || P.use_group ? 0 : (size_t)m;
    if (P.degree && (size_t)n > key_cap) key_cap = (size_t)n;
    if (key_cap) {
        BTC_TRY(g->keys0.reserve(sizeof(uint64_t) * key_cap));
        BTC_TRY(g->keys1.reserve(sizeof(uint64_t) * key_cap));
        BTC_TRY(g->sort_scratch.reserve(sizeof(uint32_t) * radix_scratch_words(key_cap)));
    }
    if (!P.use_group) {
        const size_t chunk_slots = P.use_bitmap ? bitmap_chunks(P.bm_words) : sort_tiles((size_t)m);
        BTC_TRY(g->tile_base.reserve(sizeof(uint32_t) * (chunk_slots + 1)));
    }
    if (P.use_bitmap) {
        BTC_TRY(g->bitmap.reserve(sizeof(uint32_t) * (P.bm_words ? P.bm_words : 1)));
        BTC_TRY(g->prefix.reserve(sizeof(uint2) * (P.bm_words ? P.bm_words : 1)));
    }
    BTC_TRY(g->indptr.reserve(sizeof(uint32_t) * ((size_t)geom.n_row_blocks + 1)));
    BTC_TRY(ensure_count_scratch(g));

    const size_t TW = (size_t)16 * (tile_cols / 32);
    if (small) {
        // a first build reserves a tile per edge (or per cell) instead of waiting for the count
        if (!g->indices.ptr || !g->row_indices.ptr || !g->blocks.ptr || !g->rowmask.ptr) {
            const uint64_t cells = (uint64_t)geom.n_row_blocks * (uint64_t)geom.n_col_blocks;
            const uint64_t most = std::min<uint64_t>((uint64_t)m, cells);
            const size_t bytes = (size_t)(open_width ? 256 : 4 * TW) * most;
            if (bytes <= kSmallFirstBytes) {
                BTC_TRY(g->indices.reserve(sizeof(uint32_t) * most));
                BTC_TRY(g->row_indices.reserve(sizeof(uint32_t) * most));
                BTC_TRY(g->rowmask.reserve(sizeof(uint32_t) * most));
                BTC_TRY(g->blocks.reserve(bytes));
            } else {
                small = false;
            }
        }
        if (small) {
            const bool fresh = !g->small.ptr;
            BTC_TRY(g->small.reserve(4 * sizeof(unsigned long long)));
            BTC_TRY(g->tile_base.reserve(sizeof(uint32_t) * 2 * (size_t)device_sm_count()));
            if (fresh || g->small_dirty)
                BTC_CUDA_TRY(cudaMemsetAsync(g->small.ptr, 0, 4 * sizeof(unsigned long long), s));
            g->small_dirty = true;  // until a wait has seen the build's end
        } else if (open_width) {
            return build_into(g, src, dst, m, n, 0, flags, s, tiles_only, false);
        }
    }
    P.small = small;
    P.open_width = open_width;
    // Tiles the arrays already hold room for (a rebuild): the bitmap path then enqueues
    // the whole build against that capacity, with every post-count kernel checking the
    // device tile count, and waits once at the end (or not at all with BTC_BUILD_ASYNC);
    // a count above the capacity is redone below at the right size.  A first build
    // waits for the count in between.
    if ((P.use_bitmap || P.use_group) && g->indices.ptr && g->row_indices.ptr && g->blocks.ptr && g->rowmask.ptr) {
        P.cap = tile_capacity(g);
        const uint64_t rows = std::min<uint64_t>(g->indices.bytes / 4,
                                                 std::min<uint64_t>(g->row_indices.bytes / 4, g->rowmask.bytes / 4));
        P.cap32 = (uint32_t)std::min<uint64_t>(rows, g->blocks.bytes / 64);
        P.cap128 = (uint32_t)std::min<uint64_t>(rows, g->blocks.bytes / 256);
        // The row store of the streaming count.  A build that waits decides when it knows the tiles
        // (the store is then enqueued after the wait, where the count would have been).  An enqueued
        // one whose previous graph of the same geometry averaged fewer than 8 tiles per row block
        // makes none (a mesh counts faster tile-wise); should this graph average more after all,
        // the count takes the tile-wise kernel, which needs no store.  So does a graph without
        // the memory for it.  After such a graph of another geometry, of whose size nothing follows
        // for this one, the device decides: two launches that may find nothing to do.
        P.heavy = enqueued && !tiles_only && P.cap && row_store_possible(m, geom.n_row_blocks) &&
                  !(prev_same && prev_light);
        P.row_store = P.heavy &&
                      !(prev_same && tiles_win(tile_cols, m, prev_tiles, geom.n_row_blocks, widest, P.use_bitmap)) &&
                      reserve_row_store(g, std::min<uint64_t>((uint64_t)m, 32ull * P.cap)) == BTC_OK;
        P.open = P.row_store && prev_light;
        // (the index needs the cell pairs beside it, which the bitmap builder makes)
        P.row_index = P.heavy && !P.row_store && P.use_bitmap && reserve_row_index(g, P.cap);
        g->heavy = P.heavy;
        g->row_store = P.row_store;
        g->index_built = P.row_index;
        g->open = P.open;
    }

    uint64_t* sorted = nullptr;
    if (P.cap) {
        // repeated identical asynchronous rebuilds of device input replay a CUDA graph
        const bool graphed = enqueued && !(flags & BTC_INPUT_ON_HOST) &&
                             launch_build_graph(g, P, s);
        if (!graphed) {
            const int st = enqueue_build(g, P, &sorted, s);
            if (st == kNotLaunched)
                return build_into(g, src, dst, m, n, open_width ? 0 : tile_cols, flags, s, tiles_only, false);
            BTC_TRY(st);
        }
        // the build's status and tile count are in h_meta once the stream has run it
        // (k_set_last writes them through the mapping)
        if (!g->meta_event)
            BTC_CUDA_TRY(cudaEventCreateWithFlags(&g->meta_event, cudaEventDisableTiming));
        BTC_CUDA_TRY(cudaEventRecord(g->meta_event, s));
        g->pending = true;
        g->pending_cap = P.cap;
        if (enqueued) return BTC_OK;  // resolved by the next wait
        const int st2 = resolve_build(g);
        if (small) {
            if (st2 == BTC_E_CUDA) {
                if (g->h_meta[kMetaOverflow] != kGaveUp) return st2;
                return build_into(g, src, dst, m, n, open_width ? 0 : tile_cols, flags, s, tiles_only, false);
            }
            if (open_width) {
                tile_cols = (int)g->h_meta[kHostTileCols];
                if (tile_cols != 32 && tile_cols != 128) return BTC_E_CUDA;
                g->tile_cols = tile_cols;
            }
            if (st2 == BTC_E_CAPACITY)
                return build_into(g, src, dst, m, n, tile_cols, flags, s, tiles_only, false);
        }
        if (st2 == BTC_OK) return finish_known(g, P, widest, tiles_only, s);
        if (st2 != BTC_E_CAPACITY) return st2;
        // more tiles than the arrays hold: redo the post-count steps at the right size
        BTC_CUDA_TRY(cudaMemsetAsync(meta + kMetaOverflow, 0, sizeof(unsigned long long), s));
    } else {
        BTC_TRY(enqueue_build(g, P, &sorted, s));
    }
    BTC_CUDA_TRY(cudaMemcpyAsync(g->h_meta, meta, sizeof(unsigned long long) * 3,
                                 cudaMemcpyDeviceToHost, s));
    BTC_CUDA_TRY(cudaStreamSynchronize(s));
    if (g->h_meta[kMetaBad] != 0) return BTC_E_RANGE;
    const unsigned long long tiles = g->h_meta[kMetaTiles];
    if (tiles > 0xffffffffull) return BTC_E_INVAL;
    g->num_tiles = (uint32_t)tiles;

    // ---- tile arrays ----------------------------------------------------------
    BTC_TRY(g->indices.reserve(sizeof(uint32_t) * (tiles ? tiles : 1)));
    BTC_TRY(g->row_indices.reserve(sizeof(uint32_t) * (tiles ? tiles : 1)));
    BTC_TRY(g->blocks.reserve(sizeof(uint32_t) * TW * (tiles ? tiles : 1)));
    BTC_TRY(g->rowmask.reserve(sizeof(uint32_t) * (tiles ? tiles : 1)));
    // the tile count is known here: row masks exactly when the graph averages 8 or more tiles
    // per row block, the row store when it is not dense besides
    P.heavy = !tiles_only && row_store_possible(m, geom.n_row_blocks) &&
              (uint64_t)g->num_tiles >= 8ull * (uint64_t)geom.n_row_blocks;
    P.row_store = P.heavy && !tiles_win(tile_cols, m, g->num_tiles, geom.n_row_blocks, widest, P.use_bitmap) &&
                  reserve_row_store(g, std::min<uint64_t>((uint64_t)m, 32ull * tile_capacity(g))) == BTC_OK;
    if (P.use_bitmap) {
        BTC_TRY(bitmap_emit_and_fill(geom, P.d_src, P.d_dst, m, P.degree ? g->rank.as<int32_t>() : nullptr,
                                     g->bitmap.as<uint32_t>(), g->tile_base.as<uint32_t>(),
                                     g->prefix.as<uint2>(), g->indices.as<uint32_t>(),
                                     g->row_indices.as<uint32_t>(), g->indptr.as<uint32_t>(),
                                     g->blocks.as<uint32_t>(), meta, (uint32_t)tiles, nullptr, s,
                                     g->rowmask.as<uint32_t>(), P.heavy, P.row_store));
    } else if (P.use_group) {
        BTC_TRY(launch_finish_tiles(g->indptr.as<uint32_t>(), geom.n_row_blocks, meta, (uint32_t)tiles, nullptr, s));
        BTC_TRY(enqueue_group_write(g, P, (uint32_t)tiles, s));
    } else {
        if (tiles)
            BTC_CUDA_TRY(cudaMemsetAsync(g->blocks.ptr, 0, sizeof(uint32_t) * TW * tiles, s));
        BTC_TRY(launch_fill(geom, sorted, (size_t)m, meta + kMetaValid, g->tile_base.as<uint32_t>(),
                            g->indices.as<uint32_t>(), g->row_indices.as<uint32_t>(),
                            g->blocks.as<uint32_t>(), s));
        BTC_TRY(launch_indptr(g->row_indices.as<uint32_t>(), g->num_tiles, geom.n_row_blocks,
                              g->indptr.as<uint32_t>(), s));
    }
    // the bitmap and grouped builders set the row masks; the radix path's are computed here
    const bool have_masks = P.use_bitmap || P.use_group;
    if (!have_masks || (P.use_group && !P.row_store))
        BTC_TRY(launch_rowmask(tile_cols, g->blocks.as<uint32_t>(), g->num_tiles, nullptr,
                               g->indptr.as<uint32_t>(), g->n_row_blocks, g->rowmask.as<uint32_t>(),
                               meta + kMetaRowMax, s, !have_masks));
    if (P.row_store) BTC_TRY(enqueue_row_store(g, nullptr, g->num_tiles, P.degree, s));
    P.row_index = P.heavy && !P.row_store && reserve_row_index(g, tile_capacity(g)) && P.use_bitmap;
    if (P.row_index) BTC_TRY(enqueue_row_index(g, nullptr, g->num_tiles, s));
    g->heavy = P.heavy;
    g->row_store = P.row_store;
    g->index_built = P.row_index;
    return mark_tail(g, s);
}

int count_handle(btc_bitbsr* g, int tau, cudaStream_t s, unsigned long long* d_out2,
                 uint32_t tile_begin, uint32_t tile_end, bool to_host)
{
    if (!g) return BTC_E_INVAL;
    if (tau == BTC_TAU_DEFAULT) tau = default_tau(g->tile_cols);
    if (tau < 0) return BTC_E_INVAL;
    if (!g->pending && g->failed != BTC_OK) return g->failed;
    BTC_TRY(ensure_count_scratch(g));
    BTC_TRY(wait_tail(g, s));
    CountScratch scr{g->partials.as<unsigned long long>(), g->done.as<unsigned int>(),
                     reinterpret_cast<unsigned long long*>(g->done.as<char>() + 8),
                     g->result.as<unsigned long long>(), d_out2};
    if (to_host) {
        BTC_TRY(ensure_host_meta(g));
        scr.result_host = g->d_hmeta + 7;
    }
    // after an enqueued build the kernel reads the tile count (and the build's status)
    // from the device; the capacity bounds it
    const unsigned long long* build_meta = g->pending ? g->meta.as<unsigned long long>() : nullptr;
    const uint32_t cap = g->pending ? g->pending_cap : g->num_tiles;
    // tiles averaging more than half of tau's bits: the tensor-core path's graphs
    const bool dense = (uint64_t)g->input_edges * 2 > (uint64_t)tau * (uint64_t)g->num_tiles;
    const bool whole = tile_begin == 0 && tile_end == 0xffffffffu;
    // A caller's lower tau asks for the tensor cores, which only the tile kernels use.  While an
    // enqueued build is pending its tiles are not known (num_tiles is the graph's before it, of
    // whatever size): the store it has made is used.
    // Once they are known, a mesh and a dense graph take the tile kernels all the same.
    const bool open = g->pending && g->open;
    const uint64_t many = 8ull * (uint64_t)g->n_row_blocks;
    const bool streams = g->pending || ((uint64_t)g->num_tiles >= many &&
                                        !dense_graph(g->tile_cols, g->input_edges, g->num_tiles, g->n_row_blocks));
    const uint64_t wpr = bitmap_words_per_row(make_geom(g->n, g->tile_cols));
    auto tiles_count = [&](const uint32_t* rowmask, const uint2* cellpp, bool index, uint32_t hint) {
        return launch_count(g->tile_cols, g->indptr.as<uint32_t>(), g->indices.as<uint32_t>(),
                            g->row_indices.as<uint32_t>(), g->blocks.as<uint32_t>(),
                            cap, g->n_row_blocks, tau, scr, s, nullptr, 0, nullptr, rowmask, cellpp, wpr,
                            g->meta.as<unsigned long long>() + kMetaRowMax, tile_begin, tile_end,
                            build_meta, hint, index ? g->row_off.as<uint32_t>() : nullptr,
                            index ? g->row_ent.as<uint2>() : nullptr, dense);
    };
    if (open) {
        scr.tiles_below = many;
        BTC_TRY(tiles_count(nullptr, nullptr, false, g->num_tiles));
        scr.tiles_below = ~0ull;
        scr.tiles_from = many;
    }
    if (g->row_store && tau >= default_tau(g->tile_cols) && streams)
        return launch_count_stream(row_store_of(g), g->meta.as<unsigned long long>() + kMetaRowChunks,
                                   g->tile_cols, g->n_row_blocks, ((uint32_t)g->n + 63) / 64, scr, nullptr, 0,
                                   nullptr, g->row_indices.as<uint32_t>(), g->indices.as<uint32_t>(), tile_begin,
                                   std::min(tile_end, cap), whole, true, build_meta,
                                   count_grid_size(g->tile_cols), s);
    bool cells = g->cells && !g->cells_lazy, index = false;
    if (g->heavy && (g->pending || g->num_tiles >= many)) {
        const unsigned long long* d_tiles = build_meta ? build_meta + kMetaTiles : nullptr;
        cells = ensure_cells(g, d_tiles, cap, wpr * (uint64_t)g->n_row_blocks, wpr, s);
        index = cells && ensure_row_index(g, d_tiles, cap, s);
    }
    return tiles_count(g->rowmask.as<uint32_t>(), cells ? g->prefix.as<uint2>() : nullptr, index,
                       open ? (uint32_t)std::max<uint64_t>(g->num_tiles, many) : g->num_tiles);
}

int resolve_build(btc_bitbsr* g)
{
    if (!g->pending) return g->failed;
    g->pending = false;
    if (cudaEventSynchronize(g->meta_event) != cudaSuccess) {
        cudaGetLastError();
        return g->failed = BTC_E_CUDA;
    }
    const unsigned long long* h = g->h_meta;
    g->small_dirty = g->small_dirty && h[kMetaOverflow] == kGaveUp;
    if (h[kMetaOverflow] == kGaveUp) {
        g->failed = BTC_E_CUDA;
    } else if (h[kMetaBad] != 0) {
        g->failed = BTC_E_RANGE;
    } else if (h[kMetaOverflow] != 0 || h[kMetaTiles] > g->pending_cap) {
        g->failed = BTC_E_CAPACITY;
    } else {
        g->num_tiles = (uint32_t)h[kMetaTiles];
        g->failed = BTC_OK;
    }
    return g->failed;
}

// ===========================================================================
// C ABI
// ===========================================================================
namespace btc200 {
// An empty handle whose allocations are all stream-ordered on `s` from `pool`, for an
// owner that uses it on `s` only (a server slot); its first (re)build sizes it.
btc_bitbsr* bitbsr_new_pooled(cudaMemPool_t pool, cudaStream_t s)
{
    btc_bitbsr* g = new (std::nothrow) btc_bitbsr();
    if (g) g->set_pool(pool, s);
    return g;
}
}  // namespace btc200

extern "C" {

int btc_abi_version(void) { return (1 << 16) | 1; }

int btc_default_tau(int tile_cols) { return default_tau(tile_cols); }

const char* btc_strerror(int status)
{
    switch (status) {
    case BTC_OK: return "ok";
    case BTC_E_INVAL: return "invalid argument";
    case BTC_E_NOMEM: return "out of memory";
    case BTC_E_CUDA: return "CUDA error";
    case BTC_E_TIMEOUT: return "device wait timed out";
    case BTC_E_RANGE: return "vertex id out of range";
    case BTC_E_CAPACITY: return "an enqueued rebuild needed more tiles than the handle held";
    default: return "unknown status";
    }
}

int btc_lite_select_tile_cols(int64_t nnz, int32_t num_rows, int mode)
{
    if (mode == 1) return 32;
    if (mode == 2) return 128;
    const float avg = num_rows > 0 ? (float)nnz / (float)num_rows : 0.0f;
    return (avg < 15.0f || num_rows < 50000) ? 32 : 128;
}

int btc_build_bitbsr(const int32_t* src, const int32_t* dst, int64_t m, int32_t n, int tile_cols,
                     uint32_t flags, btc_stream_t stream, btc_bitbsr** out)
{
    if (!out) return BTC_E_INVAL;
    *out = nullptr;
    btc_bitbsr* g = new (std::nothrow) btc_bitbsr();
    if (!g) return BTC_E_NOMEM;
    const int st = build_into(g, src, dst, m, n, tile_cols, flags, stream);
    if (st != BTC_OK) {
        g->release_all();
        delete g;
        return st;
    }
    *out = g;
    return BTC_OK;
}

int btc_rebuild_bitbsr(btc_bitbsr* g, const int32_t* src, const int32_t* dst, int64_t m, int32_t n,
                       int tile_cols, uint32_t flags, btc_stream_t stream)
{
    if (!g) return BTC_E_INVAL;
    const int st = build_into(g, src, dst, m, n, tile_cols, flags, stream);
    if (!g->pending) g->failed = st;  // an enqueued build's status comes with resolve_build
    return st;
}

int btc_count_async(btc_bitbsr* g, int tau, btc_stream_t stream, unsigned long long* d_out)
{
    return count_handle(g, tau, stream, d_out);
}

int btc_count(btc_bitbsr* g, int tau, btc_stream_t stream, unsigned long long* out_count,
              float* kernel_ms)
{
    if (!g || !out_count) return BTC_E_INVAL;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (kernel_ms) {
        BTC_CUDA_TRY(cudaEventCreate(&e0));
        BTC_CUDA_TRY(cudaEventCreate(&e1));
        BTC_CUDA_TRY(cudaEventRecord(e0, stream));
    }
    // the count kernel's last CTA writes the result into h_meta[7] through the mapping
    int st = count_handle(g, tau, stream, nullptr, 0, 0xffffffffu, true);
    if (st == BTC_OK && kernel_ms && cudaEventRecord(e1, stream) != cudaSuccess) st = BTC_E_CUDA;
    if (st == BTC_OK && cudaStreamSynchronize(stream) != cudaSuccess) st = BTC_E_CUDA;
    if (st == BTC_OK) st = resolve_build(g);
    if (st == BTC_OK) {
        *out_count = g->h_meta[7];
        if (kernel_ms) cudaEventElapsedTime(kernel_ms, e0, e1);
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    return st;
}

int btc_bitbsr_info(const btc_bitbsr* gc, btc_bitbsr_view* v)
{
    if (!gc || !v) return BTC_E_INVAL;
    btc_bitbsr* g = const_cast<btc_bitbsr*>(gc);
    BTC_TRY(resolve_build(g));
    if (!g->edges_known) {
        // unique lower edges = bits set in the tiles (duplicates OR the same bit); the
        // build may have run on any stream, so wait for the device first
        BTC_CUDA_TRY(cudaDeviceSynchronize());
        unsigned long long u = 0;
        unsigned long long* d = g->meta.as<unsigned long long>() + kMetaUniq;
        BTC_TRY(launch_popcount_sum(g->tile_cols, g->blocks.as<uint32_t>(), g->num_tiles, d, nullptr));
        BTC_CUDA_TRY(cudaMemcpy(&u, d, sizeof(u), cudaMemcpyDeviceToHost));
        g->num_edges = (int64_t)u;
        g->edges_known = true;
    }
    std::memset(v, 0, sizeof(*v));
    v->bcsr.indptr = g->indptr.as<uint32_t>();
    v->bcsr.indices = g->indices.as<uint32_t>();
    v->bcsr.blocks = g->blocks.as<uint32_t>();
    v->bcsr.row_indices = g->row_indices.as<uint32_t>();
    v->bcsr.result = g->result.as<unsigned long long>();
    v->bcsr.n = g->n;
    v->bcsr.n_row_blocks = g->n_row_blocks;
    v->bcsr.num_blocks = g->num_tiles;
    v->tile_cols = g->tile_cols;
    v->device = g->device;
    v->num_edges = g->num_edges;
    v->input_edges = g->input_edges;
    v->device_bytes = g->device_bytes();
    return BTC_OK;
}

int btc_density_hist(btc_bitbsr* g, btc_stream_t stream, uint64_t* hist)
{
    if (!g || !hist) return BTC_E_INVAL;
    BTC_TRY(resolve_build(g));
    const size_t nb = (size_t)16 * g->tile_cols + 1;
    DevBuf d;
    BTC_TRY(d.reserve(sizeof(unsigned long long) * nb));
    int st = BTC_OK;
    if (cudaMemsetAsync(d.ptr, 0, sizeof(unsigned long long) * nb, stream) != cudaSuccess) st = BTC_E_CUDA;
    if (st == BTC_OK)
        st = launch_density(g->tile_cols, g->blocks.as<uint32_t>(), g->num_tiles,
                            d.as<unsigned long long>(), stream);
    if (st == BTC_OK && cudaMemcpyAsync(hist, d.ptr, sizeof(unsigned long long) * nb,
                                        cudaMemcpyDeviceToHost, stream) != cudaSuccess)
        st = BTC_E_CUDA;
    if (st == BTC_OK && cudaStreamSynchronize(stream) != cudaSuccess) st = BTC_E_CUDA;
    if (st == BTC_OK) d.release_idle();
    else d.release();
    return st;
}

void btc_free(btc_bitbsr* g)
{
    if (!g) return;
    g->release_all();
    delete g;
}

// ---------------------------------------------------------------------------
// reference-shaped struct surface
// ---------------------------------------------------------------------------
static int convert_struct(btc_bcsr_device* b, const int32_t* d_rows, const int32_t* d_cols,
                          int64_t nnz, int32_t num_rows, int tile_cols)
{
    if (!b) return BTC_E_INVAL;
    std::memset(b, 0, sizeof(*b));
    btc_bitbsr* g = nullptr;
    g = new (std::nothrow) btc_bitbsr();
    if (!g) return BTC_E_NOMEM;
    const int st = build_into(g, d_rows, d_cols, nnz, num_rows, tile_cols, 0, nullptr, true);
    if (st != BTC_OK) {
        btc_free(g);
        return st;
    }
    // hand the arrays to the struct; it frees them one by one (btc_bcsr_free)
    b->indptr = g->indptr.as<uint32_t>();
    b->indices = g->indices.as<uint32_t>();
    b->blocks = g->blocks.as<uint32_t>();
    b->row_indices = g->row_indices.as<uint32_t>();
    b->result = g->result.as<unsigned long long>();
    b->n = g->n;
    b->n_row_blocks = g->n_row_blocks;
    b->num_blocks = g->num_tiles;
    g->indptr.ptr = g->indices.ptr = g->blocks.ptr = g->row_indices.ptr = g->result.ptr = nullptr;
    g->indptr.bytes = g->indices.bytes = g->blocks.bytes = g->row_indices.bytes = g->result.bytes = 0;
    btc_free(g);
    return BTC_OK;
}

int btc_convert_coo_to_bcsr_16x128_gpu(btc_bcsr_device* b, const int32_t* d_rows,
                                       const int32_t* d_cols, int64_t nnz, int32_t num_rows)
{
    return convert_struct(b, d_rows, d_cols, nnz, num_rows, 128);
}

int btc_convert_coo_to_bcsr_16x32_gpu(btc_bcsr_device* b, const int32_t* d_rows,
                                      const int32_t* d_cols, int64_t nnz, int32_t num_rows)
{
    return convert_struct(b, d_rows, d_cols, nnz, num_rows, 32);
}

void btc_bcsr_free(btc_bcsr_device* b)
{
    if (!b) return;
    void* const arrays[] = {b->indptr, b->indices, b->blocks, b->row_indices, b->result};
    free_arrays(arrays, 5);
    b->indptr = b->indices = b->blocks = b->row_indices = nullptr;
    b->result = nullptr;
}

int btc_bcsr_reset_result(btc_bcsr_device* b)
{
    if (!b || !b->result) return BTC_E_INVAL;
    BTC_CUDA_TRY(cudaMemset(b->result, 0, sizeof(unsigned long long)));
    return BTC_OK;
}

int btc_bcsr_get_result(const btc_bcsr_device* b, unsigned long long* out)
{
    if (!b || !b->result || !out) return BTC_E_INVAL;
    BTC_CUDA_TRY(cudaMemcpy(out, b->result, sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    return BTC_OK;
}

}  // extern "C"

// Per-device count scratch for the struct surface, whose calls are blocking; a mutex
// serialises them.
namespace {
struct StructScratch {
    std::mutex mu;
    DevBuf partials[64];
    DevBuf done[64];
};
StructScratch& struct_scratch()
{
    static StructScratch s;
    return s;
}
}  // namespace

// Device time of the kernels a struct count enqueues on the legacy stream, without the allocations
// and waits between them: the sum over its spans.
struct KernelTime {
    static constexpr int kMost = 8;
    cudaEvent_t at[kMost] = {};
    int n = 0;
    bool on;
    explicit KernelTime(bool wanted) : on(wanted) {}
    KernelTime(const KernelTime&) = delete;
    KernelTime& operator=(const KernelTime&) = delete;
    ~KernelTime()
    {
        for (int i = 0; i < n; ++i) cudaEventDestroy(at[i]);
    }
    // begins a span, or ends the one begun before
    int mark()
    {
        if (!on || n == kMost) return BTC_OK;
        BTC_CUDA_TRY(cudaEventCreate(&at[n]));
        ++n;
        BTC_CUDA_TRY(cudaEventRecord(at[n - 1], nullptr));
        return BTC_OK;
    }
    // after the last span's work is done
    float ms() const
    {
        float sum = 0.f;
        for (int i = 0; i + 1 < n; i += 2) {
            float t = 0.f;
            if (cudaEventElapsedTime(&t, at[i], at[i + 1]) == cudaSuccess) sum += t;
        }
        return sum;
    }
};

// The streaming count of a struct whose row blocks average 8 or more tiles: the row masks
// and the row store are made for this call, which costs a pass over the tiles (R-MAT scale
// 18 in natural order, 16x128: 0.3 ms) and saves the tile-wise kernel's searches (22 ms).
// BTC_E_NOMEM where there is no memory for them, or the tiles are not what they take
// (launch_rowstore_check): the caller takes the tile-wise kernel.
static int count_struct_stream(const btc_bcsr_device* b, int tile_cols, CountScratch scr, KernelTime& kt)
{
    struct Scratch {
        DevBuf rowmask, off, key, bits, first, meta;
        unsigned long long* host = nullptr;
        unsigned long long context = 0;
        bool idle = false;
        ~Scratch()
        {
            if (!idle && cudaDeviceSynchronize() != cudaSuccess) return;  // (given up: see DevBuf)
            for (DevBuf* d : {&rowmask, &off, &key, &bits, &first, &meta}) d->release_idle();
            host_slot_free(host, context);
        }
    } w;
    const uint32_t T = b->num_blocks;
    const uint64_t R = (uint64_t)b->n_row_blocks;
    BTC_TRY(w.rowmask.reserve(sizeof(uint32_t) * (size_t)T));
    BTC_TRY(w.meta.reserve(sizeof(unsigned long long) * kMetaSlots));
    unsigned long long* meta = w.meta.as<unsigned long long>();
    BTC_CUDA_TRY(cudaMemsetAsync(meta, 0, sizeof(unsigned long long) * kMetaSlots, nullptr));
    // a struct that the store is not made for is found out beside the counting: the count kernel
    // then does nothing (as after a failed build), and the host learns it from the wait it has
    if (!(w.host = host_slot_alloc(&w.context))) return BTC_E_NOMEM;
    void* d_host = nullptr;
    BTC_CUDA_TRY(cudaHostGetDevicePointer(&d_host, w.host, 0));
    BTC_TRY(kt.mark());
    BTC_TRY(launch_rowstore_check(tile_cols, b->indices, b->row_indices, T, b->n_row_blocks, meta + kMetaOverflow,
                                  static_cast<unsigned long long*>(d_host), nullptr));
    BTC_TRY(launch_rowmask(tile_cols, b->blocks, T, nullptr, b->indptr, b->n_row_blocks,
                           w.rowmask.as<uint32_t>(), meta + kMetaRowMax, nullptr));
    // one entry per mask bit at most; counted (a wait) where 16 or 32 per tile is too much
    uint64_t entries = (uint64_t)T * (tile_cols == 128 ? 32 : 16);
    const bool counted = entries > (16ull << 20);
    if (counted) BTC_TRY(launch_mask_popcount(w.rowmask.as<uint32_t>(), T, meta + kMetaUniq, nullptr));
    BTC_TRY(kt.mark());
    if (counted) {
        unsigned long long bits = 0;
        BTC_CUDA_TRY(cudaMemcpy(&bits, meta + kMetaUniq, sizeof(bits), cudaMemcpyDeviceToHost));
        entries = bits;
    }
    const uint64_t chunks = row_store_chunks(entries, R);
    if (chunks * kRowChunk > 0xffffffffull) return BTC_E_NOMEM;
    const bool wide = row_store_wide(b->n_row_blocks);
    BTC_TRY(w.off.reserve(sizeof(uint32_t) * (17 * R + 1)));
    BTC_TRY(w.key.reserve((wide ? sizeof(uint2) : sizeof(uint32_t)) * kRowLanes * chunks));
    BTC_TRY(w.bits.reserve(sizeof(uint4) * kRowLanes * chunks));
    BTC_TRY(w.first.reserve(sizeof(uint32_t) * (chunks / kRowRun + 1)));
    BTC_TRY(kt.mark());
    const RowStore rs{w.off.as<uint32_t>(), w.key.ptr, w.bits.as<uint4>(), w.first.as<uint32_t>()};
    BTC_TRY(launch_rowstore(tile_cols, b->indptr, b->indices, b->blocks, b->n_row_blocks,
                            w.rowmask.as<uint32_t>(), nullptr, T, false, meta, rs, nullptr));
    BTC_TRY(launch_count_stream(rs, meta + kMetaRowChunks, tile_cols, b->n_row_blocks,
                                ((uint32_t)b->n_row_blocks * 16u + 63) / 64, scr, nullptr, 0, nullptr,
                                b->row_indices, b->indices, 0, T, true, false, meta,
                                count_grid_size(tile_cols), nullptr));
    BTC_TRY(kt.mark());
    BTC_CUDA_TRY(cudaStreamSynchronize(nullptr));
    w.idle = true;
    return *static_cast<volatile unsigned long long*>(w.host) ? BTC_E_NOMEM : BTC_OK;
}

// Whether the tile-wise kernel's tensor cores count a struct faster: dense 16x32 tiles, told
// from a sample (a struct does not know its edges).  At 16x128 streaming wins at any density
// (the complete graph on 4,096 vertices: 0.43 ms against 1.18).
static bool struct_dense(const btc_bcsr_device* b, int tile_cols, KernelTime& kt)
{
    if (tile_cols != 32) return false;
    unsigned long long context = 0;
    unsigned long long* h = host_slot_alloc(&context);
    void* d = nullptr;
    bool dense = false;
    bool sampled = h && cudaHostGetDevicePointer(&d, h, 0) == cudaSuccess;
    if (sampled) {
        kt.mark();
        sampled = launch_sample_bits(tile_cols, b->blocks, b->num_blocks, static_cast<unsigned long long*>(d),
                                     nullptr) == BTC_OK;
        kt.mark();
    }
    if (sampled) {
        if (cudaStreamSynchronize(nullptr) != cudaSuccess) return false;  // (the slot is given up)
        dense = h[1] && dense_graph(tile_cols, (int64_t)((double)h[0] / (double)h[1] * (double)b->num_blocks), b->num_blocks,
                                    b->n_row_blocks);
    } else {
        cudaGetLastError();
    }
    host_slot_free(h, context);
    return dense;
}

static int count_struct(btc_bcsr_device* b, int tile_cols, float* kernel_ms,
                        unsigned long long* out)
{
    if (!b || !b->result || !out) return BTC_E_INVAL;
    if (b->num_blocks && (!b->indptr || !b->indices || !b->blocks || !b->row_indices))
        return BTC_E_INVAL;
    int dev = 0;
    BTC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return BTC_E_INVAL;
    StructScratch& ss = struct_scratch();
    std::lock_guard<std::mutex> lock(ss.mu);
    const size_t need = sizeof(unsigned long long) * (size_t)count_grid_size(tile_cols);
    if (ss.partials[dev].bytes < need) BTC_TRY(ss.partials[dev].reserve(need));
    if (!ss.done[dev].ptr) {
        BTC_TRY(ss.done[dev].reserve(kCountCtlBytes));
        BTC_CUDA_TRY(cudaMemset(ss.done[dev].ptr, 0, kCountCtlBytes));
    }
    KernelTime kt(kernel_ms != nullptr);
    CountScratch scr{ss.partials[dev].as<unsigned long long>(), ss.done[dev].as<unsigned int>(),
                     reinterpret_cast<unsigned long long*>(ss.done[dev].as<char>() + 8), b->result,
                     nullptr};
    int st = BTC_E_NOMEM;
    if (b->n_row_blocks > 0 && (uint64_t)b->num_blocks >= 8ull * (uint64_t)b->n_row_blocks &&
        !struct_dense(b, tile_cols, kt))
        st = count_struct_stream(b, tile_cols, scr, kt);
    if (st == BTC_E_NOMEM) {
        BTC_TRY(kt.mark());
        st = launch_count(tile_cols, b->indptr, b->indices, b->row_indices, b->blocks, b->num_blocks,
                          b->n_row_blocks, default_tau(tile_cols), scr, nullptr);
        if (st == BTC_OK) st = kt.mark();
    }
    if (st == BTC_OK && cudaMemcpy(out, b->result, sizeof(unsigned long long),
                                   cudaMemcpyDeviceToHost) != cudaSuccess)
        st = BTC_E_CUDA;
    if (st == BTC_OK && kernel_ms) *kernel_ms = kt.ms();
    return st;
}

extern "C" int btc_count_triangles_16x128_adaptive(btc_bcsr_device* b, int threshold_blocks,
                                                   float* kernel_ms, unsigned long long* out)
{
    (void)threshold_blocks;
    return count_struct(b, 128, kernel_ms, out);
}

extern "C" int btc_count_triangles_16x32_adaptive(btc_bcsr_device* b, int threshold_blocks,
                                                  float* kernel_ms, unsigned long long* out)
{
    (void)threshold_blocks;
    return count_struct(b, 32, kernel_ms, out);
}
