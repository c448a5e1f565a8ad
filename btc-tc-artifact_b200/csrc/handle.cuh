// handle.cuh -- the engine's device-resident handle (private to the library).
#pragma once

#include "common.cuh"

// Arguments and buffers of an enqueued build (a cached build graph replays only when
// they are unchanged).
constexpr int kBuildKeyPtrs = 27;
struct BuildGraphKey {
    const void* ptr[kBuildKeyPtrs];
    int64_t m;
    int32_t n;
    int32_t tile_cols;
    uint32_t flags;
    uint32_t cap;
};

struct btc_bitbsr {
    int device = 0;
    int tile_cols = 0;
    int32_t n = 0;
    int32_t n_row_blocks = 0;
    uint32_t num_tiles = 0;
    int64_t input_edges = 0;
    // Bit-BSR arrays (reference layout)
    btc200::DevBuf indptr, indices, row_indices, blocks, result, rowmask;
    // row store of the streaming count (rowstore.cu): row starts, column blocks, bits and
    // the row of every run of chunks
    btc200::DevBuf rs_off, rs_key, rs_bits, rs_first;
    // row index of the row-wise count kernel (rowindex.cu), made by the build of a graph that takes
    // it, else by the first count that does: per-vertex list offsets and (column block, tile)
    // entries, plus the scan's scratch
    btc200::DevBuf row_off, row_ent, row_tot, row_bsum;
    // build workspace
    btc200::DevBuf in_src, in_dst, keys0, keys1, sort_scratch, tile_base, meta, deg, rank, bitmap, prefix;
    bool cells = false;      // prefix holds the (cell word, tile prefix) pairs of the last build
    bool heavy = false;      // the last build's graph can average 8 tiles per row block: it has row masks
    bool row_store = false;  // ... and the last build made the row store
    bool row_index = false;  // the row index of the last build's graph has been made
    bool index_built = false; // ... by the build itself, and so by each of its replays
    bool cells_lazy = false; // ... and the pairs by a count, not by the build
    bool captured = false;   // a caller's CUDA graph holds a rebuild, whose replays this handle does not see
    // count scratch
    btc200::DevBuf partials, done;
    btc200::PolicyWords policy;
    btc200::DevBuf small;     // the one-launch builder's sums and barrier (small.cu), zero between launches
    bool small_dirty = false; // a launch may have left something in them
    unsigned long long* h_meta = nullptr;  // pinned and mapped, kHostSlotWords words
    unsigned long long h_context = 0;      // ... of this context
    unsigned long long* d_hmeta = nullptr; // the device's address of h_meta
    bool edges_known = false;
    int64_t num_edges = 0;
    // BTC_BUILD_ASYNC: the build is enqueued and its metadata copy to h_meta is marked
    // by meta_event; num_tiles is the previous build's until resolve_build() has waited.
    bool pending = false;
    uint32_t pending_cap = 0;  // tile capacity the enqueued build ran against
    int failed = 0;  // status of the last build (BTC_OK once resolved without error)
    cudaEvent_t meta_event = nullptr;
    // A build that has waited may enqueue more after its wait (the row store, its index, the
    // tiles themselves where the arrays grew); meta_event then marks the end, which a count or
    // a rebuild on any stream waits for.
    bool tail = false;
    // An enqueued build whose row store is made only if the graph averages 8 tiles per row block:
    // the count behind it is launched for either case.
    bool open = false;
    // CUDA graph of a repeated asynchronous rebuild (captured on the second identical call)
    cudaGraphExec_t graph_exec = nullptr;
    BuildGraphKey graph_key{};
    BuildGraphKey last_key{};
    cudaStream_t capture_stream = nullptr;

    template <class F>
    void for_each_buf(F f)
    {
        btc200::DevBuf* all[] = {&indptr, &indices, &row_indices, &blocks, &result, &in_src, &in_dst,
                                 &keys0, &keys1, &sort_scratch, &tile_base, &meta, &deg, &rank,
                                 &bitmap, &prefix, &partials, &done, &rowmask, &row_off, &row_ent,
                                 &row_tot, &row_bsum, &rs_off, &rs_key, &rs_bits, &rs_first, &small};
        for (btc200::DevBuf* b : all) f(*b);
    }
    size_t device_bytes() const
    {
        size_t s = 0;
        const_cast<btc_bitbsr*>(this)->for_each_buf([&](btc200::DevBuf& b) { s += b.bytes; });
        return s;
    }
    // every later allocation of this handle is stream-ordered on `s` from `pool` (the
    // handle is then used on `s` only)
    void set_pool(cudaMemPool_t pool, cudaStream_t s)
    {
        for_each_buf([&](btc200::DevBuf& b) {
            b.pool = pool;
            b.stream = s;
        });
        for (btc200::DevBuf* b : {&policy.dev, &policy.skew}) {
            b->pool = pool;
            b->stream = s;
        }
    }
    void release_all()
    {
        // one wait per device for all the buffers that are not stream-ordered, and for the host
        // slot, which the kernels on the handle's device write
        constexpr int kNone = -2;
        int waited = kNone;
        bool idle = true;
        auto wait = [&](int dev) {
            if (dev == waited) return;
            waited = dev;
            if (btc200::wait_device(dev) == cudaSuccess) return;
            cudaGetLastError();
            idle = false;
        };
        if (h_meta) wait(device);
        for_each_buf([&](btc200::DevBuf& b) {
            if (b.ptr && !b.pooled) wait(b.device);
        });
        if (!idle) {
            for_each_buf([](btc200::DevBuf& b) { b.release(); });
            h_meta = nullptr;  // (given up: something may still write to it)
        }
        policy.release();
        for_each_buf([](btc200::DevBuf& b) { b.release_idle(); });
        btc200::host_slot_free(h_meta, h_context);
        h_meta = nullptr;
        d_hmeta = nullptr;
        if (meta_event) cudaEventDestroy(meta_event);
        meta_event = nullptr;
        pending = false;
        if (graph_exec) cudaGraphExecDestroy(graph_exec);
        graph_exec = nullptr;
        if (capture_stream) cudaStreamDestroy(capture_stream);
        capture_stream = nullptr;
        graph_key = BuildGraphKey{};
        last_key = BuildGraphKey{};
    }
};

// Waits for an enqueued (BTC_BUILD_ASYNC) build's metadata if one is pending, sets
// num_tiles and returns the build's status (BTC_E_RANGE, BTC_E_CAPACITY or BTC_OK).
int resolve_build(btc_bitbsr* g);


btc200::RowStore row_store_of(const btc_bitbsr* g);
// Reserves the row store of a graph with at most `entries` entries (BTC_E_NOMEM: the caller
// goes on without one); no allocation when the buffers already hold it.
int reserve_row_store(btc_bitbsr* g, uint64_t entries);
// What the row-wise count kernel reads beside the tiles, enqueued on s where the last build
// and the counts since have not made it: the cell pairs (`words` of them) and the row index.
// True when this count may use them; without the memory for the pairs it goes tile-wise, and
// without the index the kernel walks whole row blocks.  While s is capturing nothing is
// allocated; and what a replay may find changed (a capturing s, a build still pending, a
// captured rebuild) is made again by every count.
bool ensure_cells(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap, uint64_t words, uint64_t wpr,
                  cudaStream_t s);
bool ensure_row_index(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap, cudaStream_t s);
bool stream_capturing(cudaStream_t s);

int default_tau(int tile_cols);
// Whether a graph of m edges in T tiles and R row blocks is dense enough for the row-wise
// kernel's tensor cores to count it faster than the streaming count.
bool dense_graph(int tile_cols, int64_t m, uint32_t T, int64_t R);
// Whether the row-wise kernel counts it faster than the streaming one: dense, or of short rows
// (widest: 64-column blocks of the widest graph; cells: the build makes the cell pairs).  Such a
// graph gets no row store.
bool tiles_win(int tile_cols, int64_t m, uint32_t T, int64_t R, uint32_t widest, bool cells);
// Reserves the row-wise kernel's index for up to `cap` tiles (false without the memory), and
// enqueues it after the tiles and row masks.
bool reserve_row_index(btc_bitbsr* g, uint32_t cap);
int enqueue_row_index(btc_bitbsr* g, const unsigned long long* d_tiles, uint32_t cap, cudaStream_t s);
int ensure_count_scratch(btc_bitbsr* g);
// Counts tiles [tile_begin, tile_end) (clamped to the tile count) into g->result and,
// when d_out2 is given, *d_out2.
int count_handle(btc_bitbsr* g, int tau, cudaStream_t s, unsigned long long* d_out2,
                 uint32_t tile_begin = 0, uint32_t tile_end = 0xffffffffu, bool to_host = false);
// Allocates the handle's mapped pinned metadata slots (h_meta, d_hmeta) once.
int ensure_host_meta(btc_bitbsr* g);
