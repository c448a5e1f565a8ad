// rowstore.cu -- per-vertex rows of L in 64-column words, the operand of the streaming count
// kernel (count_stream.cu; no counterpart in the reference).
//
// Vertex u's row lists, in column order, one entry per 64-column block K that holds a
// neighbour of u: K and the 64 bits.  Rows are whole chunks of 16 entries -- the last one
// padded with entries without bits that repeat the row's last K -- and a chunk is eight
// words, entry i in word i % 8, half i / 8: one aligned 128-byte read of bits and one of 32
// (64 when K needs 32 bits) of keys, and eight lanes that take the first halves of their
// words take consecutive entries.  All rows sit in one array in vertex order: u's chunks
// are [off[u], off[u + 1]); chunk 0 is empty.  first_row[b] is the row that holds chunk 4 b
// (where a count warp starts a run).  64 columns: on R-MAT scale 20 in degree order the rows
// the count walks take 462 bytes an edge, against 598 in 128-column entries and 553 in
// 32-column ones with 32-bit keys, and the whole store 0.6 times the 128-column one.
//
// 16x128 tiles give up to two entries per (tile, occupied row), 16x32 tiles are joined two
// at a time, so the store and the kernel that reads it are the same for both widths.
// Entries number at most the unique edges and at most 32 per tile.
//
// One pass over the row blocks, a team of warps each: the team counts its rows' entries
// from the tiles' row-occupancy masks (byte-packed warp adds), takes the chunks it needs
// from a counter (whole runs of kRowRun, so that a run lies in one row block), and writes
// the entries, 32 tiles per warp a round: a round's entries are listed in row order in
// shared memory, then copied one per lane, so that a row's entries are written together
// and all reads are independent.  Row blocks come to lie in the order their teams arrive;
// inside one, rows are in vertex order.
#include "common.cuh"

#include <algorithm>
#include <type_traits>

namespace btc200 {
namespace rs {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / kWarp;

// What tile t of row block [a, b) adds to the rows.  16x128: its rows' first and last 64
// columns (m0, m1).  16x32: the rows of the 64-column block that starts at it (m0; 0 unless
// it is the block's first tile), `pair` when the next tile is in the block too.
template <int C>
__device__ __forceinline__ void block_rows(const uint32_t* __restrict__ indices,
                                           const uint32_t* __restrict__ rowmask, uint32_t a, uint32_t b,
                                           uint32_t t, uint32_t& K, uint32_t& m0, uint32_t& m1, bool& pair)
{
    K = m0 = m1 = 0;
    pair = false;
    if (t >= b) return;
    K = indices[t];
    const uint32_t m = rowmask[t];
    m0 = m & 0xFFFFu;
    if constexpr (C == 128) {
        m1 = m >> 16;
    } else {
        // column blocks ascend, so 2 k and 2 k + 1 are neighbours in the list
        const uint32_t before = t > a ? indices[t - 1] : 0xffffffffu;
        const uint32_t after = t + 1 < b ? indices[t + 1] : 0xffffffffu;
        pair = (K & 1u) == 0u && after == K + 1u;
        const uint32_t m_after = rowmask[t + 1 < b ? t + 1 : t];
        if (pair) m0 |= m_after;
        if ((K & 1u) && before == K - 1u) m0 = 0u;
    }
}

// Rows 4k .. 4k+3 of a 16-bit mask, one row per byte (a nibble times 0x00204081 puts its
// bit j at bit 8 j).
__device__ __forceinline__ uint32_t spread_rows(uint32_t m, int k)
{
    return (((m >> (4 * k)) & 0xFu) * 0x00204081u) & 0x01010101u;
}

// Byte of row r in four words of four rows each (0 from row 16 on).
__device__ __forceinline__ uint32_t row_byte(const uint32_t (&q)[4], uint32_t r)
{
    const uint32_t g = r >> 2;
    const uint32_t w = g == 0 ? q[0] : g == 1 ? q[1] : g == 2 ? q[2] : g == 3 ? q[3] : 0u;
    return (w >> (8 * (r & 3))) & 0xFFu;
}

// Barrier of a team of kTeam warps (teams of a CTA run independently).
template <int kTeam>
__device__ __forceinline__ void team_sync(int team)
{
    if constexpr (kTeam == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeam * kWarp) : "memory");
}

// kWide: 32-bit keys.  kTeam: warps per row block.
template <int C, bool kWide, int kTeam>
__global__ void __launch_bounds__(kThreads)
k_rs_fill(const uint32_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
          const uint32_t* __restrict__ blocks, uint32_t R, const uint32_t* __restrict__ rowmask,
          const unsigned long long* __restrict__ d_tiles, uint32_t cap,
          unsigned long long* __restrict__ meta, uint32_t* __restrict__ off, void* __restrict__ key_words,
          uint4* __restrict__ bit_words, uint32_t* __restrict__ first_row, uint32_t len_lo, uint32_t len_hi,
          unsigned long long least)
{
    constexpr int TW = 16 * (C / 32);
    constexpr int kPerTile = C == 128 ? 32 : 16;
    constexpr int kTeams = kWarps / kTeam;
    constexpr uint32_t kStep = kWarp * kTeam;  // tiles a team takes per round
    using Key = typename std::conditional<kWide, uint32_t, uint16_t>::type;
    Key* __restrict__ key = static_cast<Key*>(key_words);
    uint2* __restrict__ bits = reinterpret_cast<uint2*>(bit_words);
    // where entry i (of the whole store) sits, in halves of words
    auto place_of = [](uint32_t i) {
        return i / kRowChunk * kRowChunk + (i % kRowLanes) * 2 + (i / kRowLanes) % 2;
    };
    struct Warp {
        uint16_t code[kPerTile * kWarp];  // the round's entries in row order: half, row, lane
        uint32_t K[kWarp];                // the lanes' tile columns (16x32: bit 31 marks a pair)
        uint32_t base[16];                // the rows' next entries less their first place in code
    };
    struct Team {
        uint32_t cnt[2][kTeam][16];  // entries per row and warp (rounds alternate)
        uint32_t end[16];            // the rows' ends, in entries
        uint32_t last[16];           // the rows' last keys
        uint32_t chunk;              // the row block's first chunk
    };
    __shared__ Warp s_all[kWarps];
    __shared__ Team s_team[kTeams];
    // overflowed tile arrays: nothing was built; fewer tiles than asked for: no store is wanted
    if (d_tiles && (*d_tiles > cap || *d_tiles < least)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int team = warp / kTeam, w = warp % kTeam;
    Warp& s = s_all[warp];
    Team& tm = s_team[team];
    if (blockIdx.x == 0 && threadIdx.x < kRowChunk) {  // chunk 0: empty
        key[threadIdx.x] = 0;
        bits[threadIdx.x] = make_uint2(0u, 0u);
    }
    uint32_t longest = 0, most_chunks = 0;
    auto row_block = [&](uint64_t I, uint32_t a, uint32_t b) {
        // ---- the rows' entries (lane r < 16: row r's) -----------------------------------
        uint32_t K = 0, m0 = 0, m1 = 0;
        bool pair = false;
        uint32_t cnt = 0;
        for (uint32_t t0 = a + kWarp * w; t0 < b; t0 += kStep) {
            block_rows<C>(indices, rowmask, a, b, t0 + lane, K, m0, m1, pair);
            // the lanes' masks, four rows to a word, added by one warp add per word (at most
            // 64 per byte)
            uint32_t q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                q[k] = __reduce_add_sync(kFull, spread_rows(m0, k) + (C == 128 ? spread_rows(m1, k) : 0u));
            cnt += row_byte(q, lane);
        }
        if constexpr (kTeam > 1) {
            if (lane < 16) tm.cnt[1][w][lane] = cnt;
            team_sync<kTeam>(team);
            cnt = 0;
            if (lane < 16)
                for (int x = 0; x < kTeam; ++x) cnt += tm.cnt[1][x][lane];
        }
        // ---- chunks: every row whole ones, the row block whole runs ------------------------
        const uint32_t chunks = (cnt + kRowChunk - 1) / kRowChunk;  // 0 from lane 16 on
        uint32_t incl = chunks;
#pragma unroll
        for (int d = 1; d < 16; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, incl, d);
            if (lane >= d) incl += y;
        }
        const uint32_t total = __shfl_sync(kFull, incl, 15);
        most_chunks = max(most_chunks, total);
        if (w == 0 && lane == 0) {
            const uint32_t want = (total + kRowRun - 1) / kRowRun * kRowRun;
            tm.chunk = kRowRun + (want ? (uint32_t)atomicAdd(&meta[kMetaRowChunks], (unsigned long long)want) : 0u);
        }
        team_sync<kTeam>(team);
        const uint32_t start = tm.chunk + incl - chunks;
        if (w == 0) {
            if (lane < 16) {
                off[17 * I + lane] = start;
                tm.end[lane] = start * kRowChunk + cnt;
                tm.last[lane] = 0u;
                for (uint32_t x = (start + kRowRun - 1) / kRowRun; x * kRowRun < start + chunks; ++x)
                    first_row[x] = 16 * (uint32_t)I + lane;
            } else if (lane == 16) {
                off[17 * I + 16] = tm.chunk + total;
            }
        }
        uint32_t next = start * kRowChunk;  // lane r: row r's next entry (the same in every warp)
        // ---- the entries --------------------------------------------------------------------
        int flip = 0;
        for (uint32_t t0 = a; t0 < b; t0 += kStep, flip ^= 1) {
            const uint32_t tw = t0 + kWarp * w;  // this warp's tiles
            if (b - a > kStep) block_rows<C>(indices, rowmask, a, b, tw + lane, K, m0, m1, pair);
            s.K[lane] = K | (pair ? 0x80000000u : 0u);
            // per row: entries of lower lanes (pre) and of all lanes (all), one byte per row
            uint32_t pre[4], all[4], own[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                pre[k] = own[k] = spread_rows(m0, k) + (C == 128 ? spread_rows(m1, k) : 0u);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t y = __shfl_up_sync(kFull, pre[k], d);
                    if (lane >= d) pre[k] += y;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                all[k] = __shfl_sync(kFull, pre[k], 31);
                pre[k] -= own[k];
            }
            // lane r: row r's entries this round and their first place in the list
            const uint32_t rc = row_byte(all, lane);
            uint32_t first = rc;
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, first, d);
                if (lane >= d) first += y;
            }
            const uint32_t n = __shfl_sync(kFull, first, 15);
            first -= rc;
            if constexpr (kTeam > 1) {
                if (lane < 16) tm.cnt[flip][w][lane] = rc;
                team_sync<kTeam>(team);  // (also: the ends and last keys above)
                if (lane < 16) {
                    uint32_t before = 0, sum = 0;
                    for (int x = 0; x < kTeam; ++x) {
                        const uint32_t c = tm.cnt[flip][x][lane];
                        before += x < w ? c : 0u;
                        sum += c;
                    }
                    s.base[lane] = next + before - first;
                    next += sum;
                }
            } else if (lane < 16) {
                s.base[lane] = next - first;
                next += rc;
            }
            uint32_t rows = __reduce_or_sync(kFull, m0 | m1);  // (the shuffle has every lane)
            while (rows) {
                const uint32_t r = __ffs(rows) - 1;
                rows &= rows - 1;
                uint32_t at = __shfl_sync(kFull, first, r) + row_byte(pre, r);
                if ((m0 >> r) & 1u) s.code[at++] = (uint16_t)((r << 5) | lane);
                if (C == 128 && ((m1 >> r) & 1u)) s.code[at] = (uint16_t)(512u | (r << 5) | lane);
            }
            __syncwarp();
#pragma unroll 2
            for (uint32_t i = lane; i < n; i += kWarp) {
                const uint32_t code = s.code[i], r = (code >> 5) & 15u, l = code & 31u;
                const uint32_t* tile = blocks + (size_t)(tw + l) * TW;
                uint32_t kk = s.K[l];
                uint2 v;
                if constexpr (C == 128) {
                    const uint32_t h = code >> 9;
                    v = *reinterpret_cast<const uint2*>(tile + 4 * r + 2 * h);
                    kk = 2u * kk + h;
                } else {
                    const uint32_t x = tile[r];
                    v = (kk & 1u) ? make_uint2(0u, x) : make_uint2(x, (kk >> 31) ? tile[TW + r] : 0u);
                    kk = (kk & 0x7fffffffu) >> 1;
                }
                const uint32_t at = s.base[r] + i;
                const uint32_t p = place_of(at);
                key[p] = (Key)kk;
                bits[p] = v;
                if (at + 1 == tm.end[r]) tm.last[r] = kk;
            }
            __syncwarp();
        }
        team_sync<kTeam>(team);
        // pad the rows' last chunks
#pragma unroll
        for (int i = w * kWarp + lane; i < 16 * (int)kRowChunk; i += kTeam * kWarp) {
            const uint32_t r = i / kRowChunk;
            const uint32_t end = tm.end[r], at = end + i % kRowChunk;
            if (end % kRowChunk != 0 && at / kRowChunk == end / kRowChunk) {
                const uint32_t p = place_of(at);
                key[p] = (Key)tm.last[r];
                bits[p] = make_uint2(0u, 0u);
            }
        }
        team_sync<kTeam>(team);
    };
    // Row blocks of more than len_lo tiles (0: all) and at most len_hi.
    for (uint64_t I = (uint64_t)blockIdx.x * kTeams + team; I < R; I += (uint64_t)gridDim.x * kTeams) {
        const uint32_t a = indptr[I], b = indptr[I + 1];
        longest = max(longest, b - a);
        if (b - a <= len_hi && (len_lo == 0 || b - a > len_lo)) row_block(I, a, b);
    }
    // the CTA's longest: one atomic each (a team's own were 12 us of R-MAT scale 22's rows)
    __shared__ uint32_t s_long[2];
    if (threadIdx.x < 2) s_long[threadIdx.x] = 0;
    __syncthreads();
    if (w == 0 && lane == 0) {
        atomicMax(&s_long[0], longest);
        atomicMax(&s_long[1], most_chunks);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_long[0]) atomicMax(&meta[kMetaRowMax], (unsigned long long)s_long[0]);
    if (threadIdx.x == 0 && s_long[1]) atomicMax(&meta[kMetaRowLong], (unsigned long long)s_long[1]);
}

// Raises *bad (and the host's word) where a caller's tiles are not what the store and its count
// are sized by: column blocks ascending within a row block and below `limit`.
__global__ void k_rs_check(const uint32_t* __restrict__ indices, const uint32_t* __restrict__ row_indices,
                           uint32_t T, uint32_t limit, unsigned long long* __restrict__ bad,
                           volatile unsigned long long* __restrict__ host_bad)
{
    bool ok = true;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < T;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t K = indices[t];
        ok &= K < limit;
        if (t > 0 && row_indices[t] == row_indices[t - 1]) ok &= indices[t - 1] < K;
    }
    if (!ok) {
        *bad = 1ull;
        *host_bad = 1ull;
    }
}

__global__ void k_mask_popcount(const uint32_t* __restrict__ mask, uint32_t n,
                                unsigned long long* __restrict__ out)
{
    uint32_t sum = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        sum += __popc(mask[i]);
    sum = __reduce_add_sync(kFull, sum);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(out, (unsigned long long)sum);
}

}  // namespace rs

int launch_rowstore_check(int tile_cols, const uint32_t* indices, const uint32_t* row_indices, uint32_t T,
                          int32_t n_row_blocks, unsigned long long* bad, unsigned long long* d_host,
                          cudaStream_t s)
{
    const uint64_t limit = (16ull * (uint64_t)n_row_blocks + tile_cols - 1) / tile_cols;
    if (T)
        rs::k_rs_check<<<std::min<uint32_t>((T + 255) / 256, 4u * device_sm_count()), 256, 0, s>>>(
            indices, row_indices, T, (uint32_t)limit, bad, d_host);
    return cudaGetLastError() == cudaSuccess ? BTC_OK : BTC_E_CUDA;
}

int launch_mask_popcount(const uint32_t* mask, uint32_t n, unsigned long long* out, cudaStream_t s)
{
    if (n) rs::k_mask_popcount<<<std::min<uint32_t>((n + 255) / 256, 4u * device_sm_count()), 256, 0, s>>>(mask, n, out);
    return cudaGetLastError() == cudaSuccess ? BTC_OK : BTC_E_CUDA;
}

int launch_rowstore(int tile_cols, const uint32_t* indptr, const uint32_t* indices, const uint32_t* blocks,
                    int32_t n_row_blocks, const uint32_t* rowmask, const unsigned long long* d_tiles,
                    uint32_t cap, bool by_degree, unsigned long long* meta, const RowStore& out,
                    cudaStream_t s, unsigned long long least)
{
    const uint32_t R = n_row_blocks > 0 ? (uint32_t)n_row_blocks : 0u;
    if (R == 0) return BTC_OK;
    // Few row blocks leave the GPU idle, so eight warps share one (Erdos-Renyi 16384 / 16: 1,024
    // row blocks, 26 us with one warp, 19 with two, 13 with four, 9.7 with eight; R-MAT scale
    // 16: 107, 57, 40 us); from four row blocks per resident warp on, a team's barriers cost
    // more than they save (R-MAT scale 22: 0.98 ms with one warp, 1.10 with two, 1.40 with
    // eight; 256 mixed graphs: 0.31, 0.41 ms, 0.54 with four).
    // In natural order the long row blocks among many (a hub's: 8,192 tiles at R-MAT scale 18,
    // 256 rounds of one warp) get a team in a second launch: 0.51 -> 0.22 ms there.  Degree
    // order has none that long, and the second launch costs more than it gives (scale 22:
    // 0.99 ms without it, 1.15 with).
    constexpr uint32_t kLong = 512, kAny = 0xffffffffu;
    const bool few = R <= 32u * (uint32_t)device_sm_count();
    const uint32_t sms = (uint32_t)device_sm_count();
    auto launch = [&](auto kernel, uint32_t per_cta, uint32_t len_lo, uint32_t len_hi) {
        const uint32_t grid = std::min((R + per_cta - 1) / per_cta, sms * 16);
        kernel<<<grid, rs::kThreads, 0, s>>>(indptr, indices, blocks, R, rowmask, d_tiles, cap, meta, out.off,
                                             out.key, out.bits, out.first_row, len_lo, len_hi, least);
    };
    auto fill = [&](auto one, auto team) {
        if (!few) launch(one, rs::kWarps, 0, by_degree ? kAny : kLong);
        if (few || !by_degree) launch(team, 1, few ? 0 : kLong, kAny);
    };
    if (row_store_wide(n_row_blocks)) {
        if (tile_cols == 128)
            fill(rs::k_rs_fill<128, true, 1>, rs::k_rs_fill<128, true, 8>);
        else
            fill(rs::k_rs_fill<32, true, 1>, rs::k_rs_fill<32, true, 8>);
    } else {
        if (tile_cols == 128)
            fill(rs::k_rs_fill<128, false, 1>, rs::k_rs_fill<128, false, 8>);
        else
            fill(rs::k_rs_fill<32, false, 1>, rs::k_rs_fill<32, false, 8>);
    }
    return cudaGetLastError() == cudaSuccess ? BTC_OK : BTC_E_CUDA;
}

}  // namespace btc200
