// count_stream.cu -- the count kernel over the row store (rowstore.cu): one warp stages a
// vertex's row in shared memory and streams its neighbours' rows past it.
//
// Computes what btc/operations/tc_16x128_mma_v5.h:9-211 and tc_16x32_mma_v6.h:9-238
// compute -- for every edge (u, v), u > v, the size of the intersection of u's and v's
// lower neighbours -- from per-vertex rows of 64-column words instead of from tiles:
//
//  * u's row (its entries: 64-column block K and 64 bits) is scattered into a warp's table
//    of W slots, slot K - K0 with K0 the row's first column block; slots without an entry
//    hold zeros.  Entries past the table (K - K0 >= W) stay in the store and are found by a
//    bitmap of their column blocks with ranks; on degree-ordered power-law graphs W = 1024
//    covers 99.9% of the look-ups (R-MAT scale 20).
//  * u's neighbours v are picked out of its entries' bits one per lane, and the 16-entry
//    chunks of their rows are listed in shared memory.  Four groups of eight lanes take
//    four chunks each per round: a chunk is one 32-byte (64 with 32-bit keys) and one
//    128-byte aligned read, and each lane AND-popcounts its two entries with their table
//    slots.  K alone decides the slot and a row's last chunk is padded with empty entries,
//    so a round needs no search, no branch and no bounds, and its 16 chunks' reads are all
//    in flight together.
//
// Bound by the L1: each look-up's 32 random 8-byte table reads take 3.5 shared-memory
// wavefronts.  One full ncu capture each: R-MAT scale 20 in degree order L1 73%, issue 56%, DRAM
// 4%, L2 hits 92%, 876M warp instructions in 1.38 ms (2.85 ms by the row-wise kernel over the
// tiles); 8 communities on 32,768 vertices L1 95%, issue 53%, 0.65 ms (3.18).  R-MAT scale 22:
// 21.6 GB of DRAM traffic at 2.0 TB/s, issue 47%, 10.8 ms (77.8 GB, 20.8 ms).
#include "count_common.cuh"

#include <atomic>

namespace btc200 {
namespace {

constexpr int kSThreads = 256;
constexpr int kSWarps = kSThreads / kWarp;
constexpr int kIdCap = 240;    // chunks listed per walk
constexpr int kGroup = kRowLanes;  // lanes that read a chunk
constexpr int kGroups = kWarp / kGroup;
constexpr int kBatch = 4;      // chunks a group has in flight
constexpr int kPastWords = 64;
static_assert(kPastWords == 2 * kWarp, "a lane ranks two words");
static_assert(kGroup == 8 && kIdCap % (kGroups * kBatch) == 0, "a walk's rounds are whole");

// Tables of fewer than 1,024 slots are for graphs whose rows they always hold (the engine's own
// builds, and structs that launch_rowstore_check has passed).
template <int W>
constexpr bool kPastTable = W >= 1024;

template <int W>
struct __align__(16) StreamSmem {
    uint2 tab[W + 2];          // u's row by K - K0; slot W stays zero
    uint32_t past[kPastWords]; // column blocks of u's entries past the table, modulo 32 kPastWords
    uint16_t rank[kPastWords]; // set bits of `past` before each word
    uint32_t ids[kIdCap];      // chunks of the neighbours' rows, read four at a time
};
static_assert(sizeof(uint2) * 2 % 16 == 0 && kPastWords % 4 == 0, "ids keep the 16-byte alignment");
static_assert(sizeof(StreamSmem<1024>) * kSWarps + 1184 <= 233472 / 3, "three CTAs per SM");

template <int W>
constexpr size_t stream_smem_bytes() { return sizeof(StreamSmem<W>) * kSWarps; }

// The two column blocks of a lane's key word: 16 bits each, or 32 with kWide.
template <bool kWide>
struct RowKey;
template <>
struct RowKey<false> {
    using Word = uint32_t;
    static __device__ __forceinline__ uint32_t lo(uint32_t k) { return k & 0xFFFFu; }
    static __device__ __forceinline__ uint32_t hi(uint32_t k) { return k >> 16; }
    static __device__ __forceinline__ uint32_t shfl(uint32_t k, int l) { return __shfl_sync(kFull, k, l); }
};
template <>
struct RowKey<true> {
    using Word = uint2;
    static __device__ __forceinline__ uint32_t lo(uint2 k) { return k.x; }
    static __device__ __forceinline__ uint32_t hi(uint2 k) { return k.y; }
    static __device__ __forceinline__ uint2 shfl(uint2 k, int l)
    {
        return make_uint2(__shfl_sync(kFull, k.x, l), __shfl_sync(kFull, k.y, l));
    }
};

// Position of the r-th (from 0) set bit of w, which has more than r.
__device__ __forceinline__ uint32_t select_bit(uint32_t w, uint32_t r)
{
    uint32_t p = 0;
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
        const uint32_t c = __popc(w & ((1u << h) - 1u));
        if (r >= c) {
            r -= c;
            w >>= h;
            p += h;
        }
    }
    return p;
}

// kGraphs: per-graph counts (graph_rows, graph_counts).  kRange: the tiles [tile_begin, tile_end).
template <int W, int kMinBlocks, bool kGraphs, bool kWide, bool kRange>
__global__ void __launch_bounds__(kSThreads, kMinBlocks)
k_count_stream(const uint32_t* __restrict__ off, const void* __restrict__ key_words,
               const uint4* __restrict__ bits, const uint32_t* __restrict__ first_row,
               const unsigned long long* __restrict__ rs_chunks, uint32_t n_row_blocks,
               CountScratch scr, const uint32_t* __restrict__ graph_rows, uint32_t num_graphs,
               unsigned long long* __restrict__ graph_counts, const uint32_t* __restrict__ row_indices,
               const uint32_t* __restrict__ indices, int log2c, uint32_t tile_begin, uint32_t tile_end,
               bool lower, const unsigned long long* __restrict__ build_meta)
{
    using Key = RowKey<kWide>;
    using KeyWord = typename Key::Word;
    const KeyWord* __restrict__ key = static_cast<const KeyWord*>(key_words);
    extern __shared__ __align__(16) unsigned char stream_smem_raw[];
    __shared__ unsigned long long s_red[kSWarps];
    __shared__ int s_last;
    if (count_is_another(scr, build_meta)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane / kGroup, sub = lane % kGroup;
    StreamSmem<W>& s = reinterpret_cast<StreamSmem<W>*>(stream_smem_raw)[warp];
    for (int i = lane; i <= W; i += kWarp) s.tab[i] = make_uint2(0u, 0u);
    for (int i = lane; i < kPastWords; i += kWarp) s.past[i] = 0u;

    // The chunks to take as samples, [kRowRun, e_hi), or with a tile range the row blocks
    // [I_lo, I_hi), the first and last of them cut by column.
    bool build_failed = false;
    uint32_t e_hi = 0, I_lo = 0, I_hi = 0;
    uint32_t cut_lo_u = 0, cut_lo_c = 0, cut_hi_u = 0xffffffffu, cut_hi_c = 0xffffffffu;
    if (build_meta) build_failed = (build_meta[kMetaBad] | build_meta[kMetaOverflow]) != 0ull;
    if (!build_failed) {
        if constexpr (!kRange) {
            e_hi = n_row_blocks ? kRowRun + (uint32_t)*rs_chunks : 0u;
        } else {
            if (build_meta) tile_end = (uint32_t)min((unsigned long long)tile_end, build_meta[kMetaTiles]);
            if (tile_begin < tile_end) {
                I_lo = row_indices[tile_begin];
                I_hi = row_indices[tile_end - 1] + 1;
                cut_lo_u = 16 * I_lo + 16;  // rows below this one: only columns >= cut_lo_c
                cut_lo_c = indices[tile_begin] << log2c;
                cut_hi_u = 16 * I_hi - 16;  // rows from this one: only columns < cut_hi_c
                cut_hi_c = (indices[tile_end - 1] + 1u) << log2c;
            }
        }
    }

    unsigned long long acc = 0, acc_total = 0;
    uint32_t g_cur = 0xffffffffu, g_begin = 0, g_end = 0;  // batch: current graph and its rows

    uint32_t nid = 0;  // chunks listed

    // |entry AND u's row| for an entry past the table: slot >= W, bits (x, y); u's row is the
    // chunks [p0, p1) of the store (entry i of a chunk sits in lane i % 8's word, half i / 8)
    // and its entries from `after` on lie past the table.  Most look-ups match none of them,
    // which their bit in `past` shows; a row that spans at most 32 kPastWords column blocks
    // past the table has them one per bit, and the bits' ranks number its entries, else the
    // row is bisected.  (Without `past` some lane of almost every round went on to the
    // bisection where 1% of the look-ups pass the table: R-MAT scale 22 14.4 ms, 10.9 with
    // it.  Ranks instead of bisection where 5% pass it, most of them matches: scale 18 in
    // natural order 2.0 -> 1.1 ms.)
    auto beyond = [&](uint32_t slot, uint32_t x, uint32_t y, uint32_t K0, uint32_t span, uint32_t after,
                      uint32_t p0, uint32_t p1) -> uint32_t {
        const uint32_t pb = (slot - (uint32_t)W) % (32u * kPastWords);
        const uint32_t pw = s.past[pb / 32];
        if (!((pw >> (pb & 31u)) & 1u)) return 0u;
        auto word = [&](uint32_t i) { return i / kRowChunk * kRowLanes + i % kRowLanes; };
        auto half = [&](uint32_t i) { return (i / kRowLanes) & 1u; };
        uint32_t i;
        if (span < (uint32_t)W + 32u * kPastWords) {
            i = after + s.rank[pb / 32] + __popc(pw & ((1u << (pb & 31u)) - 1u));
        } else {
            auto key_at = [&](uint32_t j) {
                const KeyWord w = key[word(j)];
                return half(j) ? Key::hi(w) : Key::lo(w);
            };
            uint32_t hi = p1 * kRowChunk;
            const uint32_t end = hi, k = slot + K0;
            i = after;
            while (i < hi) {
                const uint32_t mid = i + ((hi - i) >> 1);
                if (key_at(mid) < k) i = mid + 1;
                else hi = mid;
            }
            if (i >= end || key_at(i) != k) return 0u;
        }
        const uint4 v = bits[word(i)];
        return half(i) ? __popc(v.z & x) + __popc(v.w & y) : __popc(v.x & x) + __popc(v.y & y);
    };

    // Counts u's row (its table, first column block K0, last one K0 + span; chunks [p0, p1))
    // against the listed chunks.
    auto walk = [&](uint32_t K0, uint32_t span, uint32_t after, uint32_t p0, uint32_t p1) {
        const uint32_t n = (nid + kGroups * kBatch - 1) / (kGroups * kBatch) * (kGroups * kBatch);
        if (nid + lane < n) s.ids[nid + lane] = 0u;  // chunk 0 is empty
        __syncwarp();
        uint32_t part = 0;
        for (uint32_t j = grp * kBatch; j < n; j += kGroups * kBatch) {
            const uint4 id = *reinterpret_cast<const uint4*>(&s.ids[j]);
            const uint32_t e[kBatch] = {id.x * kRowLanes + sub, id.y * kRowLanes + sub,
                                        id.z * kRowLanes + sub, id.w * kRowLanes + sub};
            KeyWord k[kBatch];
            uint4 b[kBatch];
#pragma unroll
            for (int x = 0; x < kBatch; ++x) {
                k[x] = __ldg(key + e[x]);
                b[x] = __ldg(bits + e[x]);
            }
#pragma unroll
            for (int x = 0; x < kBatch; ++x) {
                const uint32_t s0 = Key::lo(k[x]) - K0, s1 = Key::hi(k[x]) - K0;
                const uint2 a0 = s.tab[min(s0, (uint32_t)W)], a1 = s.tab[min(s1, (uint32_t)W)];
                part += __popc(a0.x & b[x].x) + __popc(a0.y & b[x].y) + __popc(a1.x & b[x].z) +
                        __popc(a1.y & b[x].w);
                if (kPastTable<W> && span >= (uint32_t)W) {
                    if (s0 >= (uint32_t)W && s0 <= span)
                        part += beyond(s0, b[x].x, b[x].y, K0, span, after, p0, p1);
                    if (s1 >= (uint32_t)W && s1 <= span)
                        part += beyond(s1, b[x].z, b[x].w, K0, span, after, p0, p1);
                }
            }
        }
        acc += part;  // below 2^32: at most the listed rows' bits
        nid = 0;
        __syncwarp();
    };

    // Samples: chunks [fa, fb) of u's row, chunks [p0, p1).  In a lower triangle the chunks
    // past fb hold only higher columns, which no sample's row can reach: they are left out.
    auto take_row = [&](uint32_t u, uint32_t p0, uint32_t p1, uint32_t fa, uint32_t fb) {
        if (lower) p1 = fb;
        const bool small = p1 - p0 <= (uint32_t)kGroups;
        const uint32_t wb = p1 * kRowLanes;  // words end
        const uint32_t w_first = p0 * kRowLanes + lane;
        KeyWord k0{};
        uint4 b0 = make_uint4(0u, 0u, 0u, 0u);
        if (w_first < wb) {
            k0 = key[w_first];
            b0 = bits[w_first];
        }
        const uint32_t K0 = __shfl_sync(kFull, Key::lo(k0), 0);
        const uint32_t span = Key::hi(key[wb - 1]) - K0;  // up to the row's last column block
        // (padding entries have no bits and the row's last key)
        uint32_t inside = 0;  // entries in the table
        auto put = [&](uint32_t slot, uint32_t x, uint32_t y) {
            if ((x | y) == 0u) return;
            // (a small table's rows lie inside it: their store was checked or built so)
            if (slot < (uint32_t)W) {
                s.tab[slot] = make_uint2(x, y);
                ++inside;
            } else if (kPastTable<W>) {
                const uint32_t pb = (slot - (uint32_t)W) % (32u * kPastWords);
                atomicOr(&s.past[pb / 32], 1u << (pb & 31u));
            }
        };
        auto stage = [&](const KeyWord& k, const uint4& b) {
            put(Key::lo(k) - K0, b.x, b.y);
            put(Key::hi(k) - K0, b.z, b.w);
        };
        stage(k0, b0);
        if (!small)
            for (uint32_t w = w_first + kWarp; w < wb; w += kWarp) stage(key[w], bits[w]);
        __syncwarp();
        uint32_t after = 0;  // the first entry past the table
        if (kPastTable<W> && span >= (uint32_t)W) {
            after = p0 * kRowChunk + __reduce_add_sync(kFull, inside);
            if (span < (uint32_t)W + 32u * kPastWords) {
                const uint32_t c0 = __popc(s.past[2 * lane]), c1 = __popc(s.past[2 * lane + 1]);
                uint32_t incl = c0 + c1;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFull, incl, d);
                    if (lane >= d) incl += y;
                }
                s.rank[2 * lane] = (uint16_t)(incl - c0 - c1);
                s.rank[2 * lane + 1] = (uint16_t)(incl - c1);
            }
            __syncwarp();
        }
        for (uint32_t c = small ? p0 * kRowLanes : fa * kRowLanes; c < fb * kRowLanes; c += kWarp) {
            KeyWord K = k0;
            uint4 b = b0;
            if (!small && c + lane < wb) {
                K = key[c + lane];
                b = bits[c + lane];
            }
            if (c + lane < fa * kRowLanes || c + lane >= fb * kRowLanes) b = make_uint4(0u, 0u, 0u, 0u);
            if (lower && lane == 0 && c == p0 * kRowLanes && fa == p0) {
                // the row's first neighbour has no lower one in the row
                if (b.x) b.x &= b.x - 1;
                else b.y &= b.y - 1;
            }
            if (kRange && (u < cut_lo_u || u >= cut_hi_u)) {
                // a tile range's first or last row block: drop the columns outside it
                uint32_t* w = reinterpret_cast<uint32_t*>(&b);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t col = ((q < 2 ? Key::lo(K) : Key::hi(K)) << 6) + 32u * (q & 1);
                    if (u < cut_lo_u && col < cut_lo_c) w[q] = 0u;
                    if (u >= cut_hi_u && col >= cut_hi_c) w[q] = 0u;
                }
            }
            const uint32_t cnt = __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
            uint32_t incl = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, incl, d);
                if (lane >= d) incl += y;
            }
            const uint32_t total = __shfl_sync(kFull, incl, 31);
            for (uint32_t i0 = 0; i0 < total; i0 += kWarp) {
                // one neighbour per lane: the lane that holds its bit, then the bit
                const uint32_t i = min(i0 + lane, total - 1);
                int l = 0;
#pragma unroll
                for (int h = 16; h > 0; h >>= 1)
                    if (__shfl_sync(kFull, incl, l + h - 1) <= i) l += h;
                uint32_t r = i - __shfl_sync(kFull, incl - cnt, l);
                const KeyWord kk = Key::shfl(K, l);
                uint32_t w = __shfl_sync(kFull, b.x, l);
                const uint32_t w1 = __shfl_sync(kFull, b.y, l), w2 = __shfl_sync(kFull, b.z, l),
                               w3 = __shfl_sync(kFull, b.w, l);
                uint32_t v = Key::lo(kk) << 6, pc = __popc(w);
                if (r >= pc) {
                    r -= pc;
                    w = w1;
                    v += 32;
                    pc = __popc(w);
                    if (r >= pc) {
                        r -= pc;
                        w = w2;
                        v = Key::hi(kk) << 6;
                        pc = __popc(w);
                        if (r >= pc) {
                            r -= pc;
                            w = w3;
                            v += 32;
                        }
                    }
                }
                v += select_bit(w, r);
                const uint32_t vo = v + (v >> 4);  // 17 offsets per row block
                uint32_t r0 = 0, r1 = 0;
                if (i0 + lane < total && (lower || (v >> 4) < n_row_blocks)) {
                    r0 = off[vo];
                    r1 = off[vo + 1];
                }
                // list its row's chunks
                for (;;) {
                    uint32_t at = r1 - r0;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFull, at, d);
                        if (lane >= d) at += y;
                    }
                    const uint32_t sum = __shfl_sync(kFull, at, 31);
                    at += nid - (r1 - r0);
                    while (r0 < r1 && at < (uint32_t)kIdCap) s.ids[at++] = r0++;
                    nid += sum;
                    if (nid <= (uint32_t)kIdCap) break;
                    nid = kIdCap;
                    __syncwarp();
                    walk(K0, span, after, p0, p1);
                }
            }
        }
        __syncwarp();
        if (nid) walk(K0, span, after, p0, p1);
        // empty the table again
        auto clear = [&](const KeyWord& k) {
            const uint32_t s0 = Key::lo(k) - K0, s1 = Key::hi(k) - K0;
            if (s0 < (uint32_t)W) s.tab[s0] = make_uint2(0u, 0u);
            if (s1 < (uint32_t)W) s.tab[s1] = make_uint2(0u, 0u);
        };
        if (kPastTable<W> && span >= (uint32_t)W)
            for (int i = lane; i < kPastWords; i += kWarp) s.past[i] = 0u;
        if (w_first < wb) clear(k0);
        if (!small)
            for (uint32_t w = w_first + kWarp; w < wb; w += kWarp) clear(key[w]);
        __syncwarp();
    };

    // Work queue, `per` chunks each.  A warp's first grab is its own index, later ones are
    // numbered by an atomic.  A chunk of a hub row in natural order holds up to 1,024 neighbours
    // with long rows, so grabs stay at one 32nd of an even share, one to eight chunks (R-MAT scale
    // 18 in natural order: 2.83 ms with runs of four chunks and an eighth of a share, 2.05 with
    // these).
    //
    // The row blocks of a tile range lie anywhere in the store, so their chunks are numbered by
    // pass: pass p has the chunks from p * per on of every row block, up to a little more than the
    // average row block's; what longer ones have past that comes in slices, for which a grab looks
    // at up to 32 row blocks, so that the slices that are not there (most of them where a hub has a
    // hundred times the average) stay few beside the rest: a quarter of the first passes' grabs, and
    // up to eight times that where the longest row block is 32 times the average.  (A row block per grab left
    // a hub's to one warp: a quarter of R-MAT scale 20, edge factor 8, in natural order took 124
    // ms; 6.6 like this.)
    __syncwarp();
    const uint64_t nwarps = (uint64_t)gridDim.x * kSWarps;
    const uint32_t nb = I_hi - I_lo;
    uint64_t work = e_hi > kRowRun ? e_hi - kRowRun : 0u;
    uint32_t avg = 1, longest = 0;
    if constexpr (kRange) {
        avg = (uint32_t)max(rs_chunks[0] / max(n_row_blocks, 1u), 1ull);
        longest = (uint32_t)rs_chunks[kMetaRowLong - kMetaRowChunks];
        work = (uint64_t)avg * nb;
    }
    const uint64_t share = work / (nwarps * (kRange ? 8 : 32));
    const uint32_t per = (uint32_t)(share < 1 ? 1 : (share > 8 ? 8 : share));
    uint64_t grabs = (work + per - 1) / per, front = 0;
    uint32_t groups = 1, width = 1, slice = 1, from = 0;
    if constexpr (kRange) {
        const uint32_t passes = (avg + avg / 4 + per - 1) / per;
        from = passes * per;
        front = (uint64_t)passes * nb;
        grabs = front;
        if (longest > from && nb) {
            const uint64_t most = max(4 * nwarps, front / 4) * min(max(longest / (4 * avg), 1u), 8u);
            const uint64_t slices = (longest - from + per - 1) / per;
            width = (uint32_t)min((slices * nb + most - 1) / most, (uint64_t)kWarp);
            groups = (nb + width - 1) / width;
            slice = per * (uint32_t)((slices * groups + most - 1) / most);
            grabs += (uint64_t)groups * ((longest - from + slice - 1) / slice);
        }
    }
    unsigned long long kq = (unsigned long long)blockIdx.x * kSWarps + warp;
    while (kq < grabs) {
        unsigned long long next = 0;
        if (lane == 0) next = nwarps + atomicAdd(scr.work, 1ull);
        // chunks [e0, e1), row block by row block; of a range, lane l's chunks of its row block
        uint32_t e0 = 0, e1 = 0, u = 0;
        uint32_t lane_e0 = 0, lane_e1 = 0, lane_I = 0;
        unsigned pieces = 0;
        if constexpr (!kRange) {
            e0 = kRowRun + (uint32_t)(kq * per);
            e1 = min(e_hi, e0 + per);
            u = first_row[e0 / kRowRun];
        } else {
            uint32_t a, b;
            if (kq < front) {
                lane_I = lane == 0 ? I_lo + (uint32_t)(kq % nb) : I_hi;
                a = (uint32_t)(kq / nb) * per;
                b = a + per;
            } else {
                const uint64_t x = kq - front;
                lane_I = lane < width ? I_lo + (uint32_t)(x % groups) + lane * groups : I_hi;
                a = from + (uint32_t)(x / groups) * slice;
                b = a + slice;
            }
            if (lane_I < I_hi) {
                const uint32_t first = off[17u * lane_I], end = off[17u * lane_I + 16];
                lane_e0 = min(first + a, end);
                lane_e1 = min(first + b, end);
            }
            pieces = __ballot_sync(kFull, lane_e0 < lane_e1);
        }
        while (kRange ? pieces != 0u : e0 < e1) {
            uint32_t I = u >> 4;
            if constexpr (kRange) {
                const int p = __ffs(pieces) - 1;
                pieces &= pieces - 1;
                I = __shfl_sync(kFull, lane_I, p);
                e0 = __shfl_sync(kFull, lane_e0, p);
                e1 = __shfl_sync(kFull, lane_e1, p);
            }
            const uint32_t l = min(lane, 16);
            const uint32_t o = off[17u * I + l];
            const uint32_t o1 = __shfl_down_sync(kFull, o, 1);
            const uint32_t fa = max(o, e0), fb = min(o1, e1);
            unsigned todo = __ballot_sync(kFull, lane < 16 && fa < fb);
            if constexpr (kGraphs) {
                if (u < g_begin || u >= g_end) {
                    flush_graph(acc, acc_total, graph_counts, g_cur, lane);
                    g_cur = graph_of_row_block(graph_rows, num_graphs, I);
                    g_begin = 16u * graph_rows[g_cur];
                    g_end = g_cur + 1 < num_graphs ? 16u * graph_rows[g_cur + 1] : 0xffffffffu;
                }
            }
            while (todo) {
                const int r = __ffs(todo) - 1;
                todo &= todo - 1;
                take_row(16u * I + r, __shfl_sync(kFull, o, r), __shfl_sync(kFull, o1, r),
                         __shfl_sync(kFull, fa, r), __shfl_sync(kFull, fb, r));
            }
            if constexpr (!kRange) {
                // the next row block's first run
                const uint32_t end = __shfl_sync(kFull, o, 16);
                e0 = max(e0 + 1, (end + kRowRun - 1) / kRowRun * kRowRun);
                if (e0 < e1) u = first_row[e0 / kRowRun];
            }
        }
        kq = __shfl_sync(kFull, next, 0);
    }
    if constexpr (kGraphs) {
        flush_graph(acc, acc_total, graph_counts, g_cur, lane);
        acc = acc_total;
    }
    finish_count<kSThreads>(acc, scr, build_failed, s_red, &s_last);
}

using StreamKernel = decltype(&k_count_stream<1024, 3, false, false, false>);

// variant: 3 * (table size, then 32-bit keys) + (per-graph counts, then tile ranges)
constexpr int kVariants = 12;
template <int W, int kMinBlocks, bool kWide>
StreamKernel stream_kernel_of(int form)
{
    if (form == 0) return k_count_stream<W, kMinBlocks, false, kWide, false>;
    if (form == 1) return k_count_stream<W, kMinBlocks, true, kWide, false>;
    return k_count_stream<W, kMinBlocks, false, kWide, true>;
}
StreamKernel stream_kernel(int v)
{
    switch (v / 3) {
    case 0: return stream_kernel_of<256, 4, false>(v % 3);
    case 1: return stream_kernel_of<512, 4, false>(v % 3);
    case 2: return stream_kernel_of<1024, 3, false>(v % 3);
    default: return stream_kernel_of<1024, 3, true>(v % 3);
    }
}
size_t stream_smem(int v)
{
    return v / 3 == 0 ? stream_smem_bytes<256>() : v / 3 == 1 ? stream_smem_bytes<512>() : stream_smem_bytes<1024>();
}

// A variant's dynamic shared memory is an opt-in.
bool allow_stream_smem(int v)
{
    static std::atomic<unsigned long long> allowed[kVariants][kMaxDevices];
    return allow_dynamic_smem(reinterpret_cast<const void*>(stream_kernel(v)), stream_smem(v), allowed[v]);
}

// Resident CTAs per SM of a variant, cached per device; 0 on error.
int stream_blocks_per_sm(int v)
{
    static std::atomic<int> resident[kMaxDevices][kVariants];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    int per_sm = resident[dev][v].load(std::memory_order_acquire);
    if (per_sm > 0) return per_sm;
    cudaError_t e = cudaErrorInvalidValue;
    if (allow_stream_smem(v))
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stream_kernel(v), kSThreads, stream_smem(v));
    if (e != cudaSuccess || per_sm < 1) {
        note_cuda_error(e, "k_count_stream launch set-up", __FILE__, __LINE__);
        return 0;
    }
    resident[dev][v].store(per_sm, std::memory_order_release);
    return per_sm;
}

}  // namespace

// The most CTAs any variant runs at once (what a count's scratch must hold partial sums
// for), per SM; 0 on error.
int stream_blocks_per_sm_max()
{
    int most = 0;
    for (int v = 0; v < kVariants; ++v) {
        const int p = stream_blocks_per_sm(v);
        most = p > most ? p : most;
    }
    return most;
}

int launch_count_stream(const RowStore& rs, const unsigned long long* rs_chunks, int tile_cols,
                        int32_t n_row_blocks, uint32_t max_col_blocks, CountScratch scr,
                        const uint32_t* graph_rows, uint32_t num_graphs, unsigned long long* graph_counts,
                        const uint32_t* row_indices, const uint32_t* indices, uint32_t tile_begin, uint32_t tile_end, bool whole,
                        bool lower, const unsigned long long* build_meta, int grid, cudaStream_t s)
{
    const int size = row_store_wide(n_row_blocks) ? 3 : max_col_blocks <= 256 ? 0 : max_col_blocks <= 512 ? 1 : 2;
    const int v = 3 * size + (!whole ? 2 : graph_counts ? 1 : 0);
    const int per_sm = stream_blocks_per_sm(v);
    if (per_sm < 1 || !allow_stream_smem(v)) return BTC_E_CUDA;
    if (per_sm * device_sm_count() < grid) grid = per_sm * device_sm_count();
    stream_kernel(v)<<<grid, kSThreads, stream_smem(v), s>>>(
        rs.off, rs.key, rs.bits, rs.first_row, rs_chunks, (uint32_t)n_row_blocks, scr, graph_rows, num_graphs,
        graph_counts, row_indices, indices, tile_cols == 128 ? 7 : 5, tile_begin, tile_end, lower, build_meta);
    return cudaGetLastError() == cudaSuccess ? BTC_OK : BTC_E_CUDA;
}

}  // namespace btc200
