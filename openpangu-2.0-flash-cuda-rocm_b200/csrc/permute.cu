// Token histogram and permutation into expert-contiguous order.
//
// Result contract (bit-exact with the reference): position of assignment
// (row, slot) = #{assignments with a smaller expert id}
//             + #{assignments with the same id and a smaller flat index row*8+slot},
// i.e. a STABLE counting sort of the flat index by expert id.  That is the
// order the reference's ranking loop produces per projection kind
// (cuda/nvfp4_grouped.cu:117-132) and the order its host-scheduled path walks
// rows in (src/model.cpp:1528-1540).  No atomics touch the ordering, so the
// result is deterministic: each warp owns a contiguous chunk of flat indices,
// ranks inside a 32-wide step come from a vote per id bit + popcount of the
// lower lanes, and chunk bases come from an exclusive scan over (expert, chunk).
#include "expert_common.cuh"

#include <cstdio>

namespace p92b {

using ptx::pdl_launch_dependents;
using ptx::pdl_wait;

namespace {

constexpr int kChunk = 256;          // flat indices per warp in the multi-block path
constexpr int kWarps = 8;
constexpr int kSmallWarps = 32;      // of the one-block path
constexpr int kSmallChunk = 160;     // ids per warp there, at most
// 5,120: the most that the block's 48 KB of shared memory hold.  At 4,104 it takes 12.3 us against 18.5 of the three-kernel
// form (p92b_moe_permute_static; with a plan 10.3 against 16.4), at 5,120 12.4 against 18.5.
constexpr int kSmallMax = kSmallWarps * kSmallChunk;
static_assert(kSmallChunk % 32 == 0, "a warp's share is whole steps");

// Which expert ids take part.  The whole range by default; an expert-parallel GPU that holds the ids of the whole
// batch restricts the permutation to its own experts [first, first + count) - ids outside (other GPUs' experts, and
// -1 for an empty token slot) are then skipped, not clamped: they get no position and are not counted.
struct IdRange {
    int first = 0;
    int count = kExperts;
    int restricted = 0;
};

// The lanes of the warp that are valid and hold the same id (0..255) as this one, from a vote per bit: 8 votes where
// __match_any_sync goes through the distinct values (4,096 assignments: 14.3 us with it).
__device__ __forceinline__ unsigned same_id_lanes(int e, bool valid) {
    unsigned peers = __ballot_sync(0xffffffffU, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool set = (e >> b) & 1;
        const unsigned with = __ballot_sync(0xffffffffU, set);
        peers &= set ? with : ~with;
    }
    return peers;
}

// Counts the experts of one chunk into hist[256] (owned by the calling warp).
// `cached` (optional): the chunk's ids already in shared memory, cached[i - begin].
template <class T>
__device__ __forceinline__ void warp_histogram(const std::int32_t* __restrict__ ids, int begin, int end,
                                               T* hist, std::int32_t* status,
                                               const std::int16_t* cached = nullptr, IdRange range = IdRange()) {
    const int lane = threadIdx.x & 31;
    for (int e = lane; e < kExperts; e += 32) hist[e] = 0;
    __syncwarp();
    for (int base = begin; base < end; base += 32) {
        const int i = base + lane;
        bool valid = i < end;
        int e = valid ? (cached != nullptr ? static_cast<int>(cached[i - begin]) : ids[i]) : -1;
        if (range.restricted && (e < range.first || e >= range.first + range.count)) {
            valid = false;
            e = -1;
        }
        if (valid && (e < 0 || e >= kExperts)) {
            atomicCAS(status, kStatusOk, kStatusBadExpertId);
            e = e < 0 ? 0 : kExperts - 1;
        }
        const unsigned peers = same_id_lanes(e, valid);
        if (valid && (peers & ((1U << lane) - 1U)) == 0U) hist[e] += static_cast<T>(__popc(peers));
        __syncwarp();
    }
}

// A warp's ids once into shared memory, all loads in flight together, clamped to -1 .. 256 so that they fit 16 bits
// and an id out of range stays out of range.
__device__ __forceinline__ void load_chunk_ids(const std::int32_t* __restrict__ ids, int begin, int end,
                                               std::int16_t* cached) {
    for (int i = begin + (threadIdx.x & 31); i < end; i += 32) {
        const int e = ids[i];
        cached[i - begin] = static_cast<std::int16_t>(e < -1 ? -1 : (e > kExperts ? kExperts : e));
    }
    __syncwarp();
}

// Scatters one chunk.  running[e] (warp private) = first position of this chunk's rows of expert e, counted from
// expert_base[e] (null: from 0); pp_delta[e] (shared memory, read only with pp_of_flat) = padded offset - offset of expert e.
// tile_shift > 0 (with expert_base): an expert's padded rows come in tiles of 1 << tile_shift, 128 positions apart.  The steps
// of a chunk depend on one another through running[], so whatever a step reads has to be in shared memory or in
// registers already: a global load per step is a round trip to the L2 per step.
template <class T, class Order>
__device__ __forceinline__ void warp_scatter(const std::int32_t* __restrict__ ids, int begin, int end,
                                             T* running, const std::int32_t* expert_base,
                                             Order* __restrict__ order,
                                             std::int32_t* __restrict__ position,
                                             std::int32_t* __restrict__ row_token,
                                             const std::int32_t* pp_delta,
                                             std::int32_t* __restrict__ pp_of_flat,
                                             const std::int16_t* cached = nullptr, IdRange range = IdRange(),
                                             int tile_shift = 0) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    for (int step = begin; step < end; step += 32) {
        const int i = step + lane;
        bool valid = i < end;
        int e = valid ? (cached != nullptr ? static_cast<int>(cached[i - begin]) : ids[i]) : -1;
        if (range.restricted && (e < range.first || e >= range.first + range.count)) {
            if (valid) {                      // skipped: no position
                if (position != nullptr) position[i] = -1;
                if (pp_of_flat != nullptr) pp_of_flat[i] = -1;
            }
            valid = false;
            e = -1;
        }
        if (valid) e = e < 0 ? 0 : (e >= kExperts ? kExperts - 1 : e);
        const unsigned peers = same_id_lanes(e, valid);
        const int rank = __popc(peers & ((1U << lane) - 1U));
        int pos = 0;
        if (valid) {
            const int of_expert = running[e] + rank;
            pos = of_expert + (expert_base != nullptr ? expert_base[e] : 0);
            if (order != nullptr) order[pos] = static_cast<Order>(i);
            if (position != nullptr) position[i] = pos;
            if (row_token != nullptr) row_token[pos] = i / kTop;
            if (pp_of_flat != nullptr) {
                const int gaps = tile_shift > 0 ? (of_expert >> tile_shift) * (128 - (1 << tile_shift)) : 0;
                pp_of_flat[i] = pp_delta[e] + pos + gaps;
            }
        }
        __syncwarp();
        if (valid && rank == 0) running[e] += static_cast<T>(__popc(peers));
        __syncwarp();
    }
}

// Exclusive scan of 256 per-expert totals by the first 256 threads of a block: all threads that the block (still) has,
// or, with PART, the first 256 of more (named barrier 1).
template <bool PART>
__device__ __forceinline__ void scan_sync() {
    if constexpr (PART) asm volatile("bar.sync 1, 256;" ::: "memory"); else __syncthreads();
}
template <bool PART = false>
__device__ __forceinline__ int block_exclusive_scan_256(int value, std::int32_t* warp_totals) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    int inclusive = value;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        const int other = __shfl_up_sync(0xffffffffU, inclusive, offset);
        if (lane >= offset) inclusive += other;
    }
    if (lane == 31) warp_totals[warp] = inclusive;
    scan_sync<PART>();
    int before = 0;
    for (int wi = 0; wi < warp; ++wi) before += warp_totals[wi];
    scan_sync<PART>();
    return before + inclusive - value;
}

// Lists written for the expert kernels: counts/offsets extended with the shared
// expert as entry 256 (rows = tokens, positions after the routed ones), the
// compact list of entries that have rows, shared expert first (it is the largest
// group, so the persistent kernels start it first), and - for the tensor-core
// kernels - a padded position space in which every entry's rows start on a
// multiple of `pad_align`, plus the prefix of token-tile counts over the active list.  With tiles of 16 or 32 rows every
// tile starts on such a multiple (expert_common.cuh, kTileStride): the positions that takes, 128 per assignment at most,
// are what a plan reserves for as many experts with a row each.
struct RouteLists {
    std::int32_t* counts;        // [257]
    std::int32_t* offsets;       // [258]
    std::int32_t* active;        // [257]
    std::int32_t* active_count;  // [1]
    std::int32_t* pp_off;        // [258] padded offsets (null: not wanted)
    std::int32_t* tile_prefix;   // [258] exclusive prefix of token tiles over the active list, total last
    std::int32_t* tile_prefix_wide;   // the same for tiles of tile_rows_wide rows (null: not wanted)
    int pad_align;
    int tile_rows;
    int tile_rows_wide;
    bool enabled;
};

template <bool PART = false>
__device__ __forceinline__ void write_route_lists(int e, int count, int offset, int assignments, int rows,
                                                  const RouteLists& lists, std::int32_t* scan_scratch) {
    lists.counts[e] = count;
    lists.offsets[e] = offset;
    if (e == kExperts - 1) lists.offsets[kExperts] = assignments;
    if (!lists.enabled) return;
    const int slot = block_exclusive_scan_256<PART>(count > 0 ? 1 : 0, scan_scratch);
    if (count > 0) lists.active[1 + slot] = e;
    if (e == kExperts - 1) {
        lists.counts[kExperts] = rows;
        lists.offsets[kExperts + 1] = assignments + rows;
        lists.active[0] = kExperts;
        *lists.active_count = 1 + slot + (count > 0 ? 1 : 0);
    }
    if (lists.pp_off == nullptr) return;
    const int align = lists.pad_align;
    const int tiles = (count + lists.tile_rows - 1) / lists.tile_rows;
    const int padded = lists.tile_rows < 64 ? tiles * align : (count + align - 1) / align * align;
    const int pp = block_exclusive_scan_256<PART>(padded, scan_scratch);
    lists.pp_off[e] = pp;
    const int shared_tiles = (rows + lists.tile_rows - 1) / lists.tile_rows;
    const int before = block_exclusive_scan_256<PART>(tiles, scan_scratch);
    if (count > 0) lists.tile_prefix[1 + slot] = shared_tiles + before;
    if (e == kExperts - 1) {
        lists.pp_off[kExperts] = pp + padded;
        lists.pp_off[kExperts + 1] = pp + padded + (rows + align - 1) / align * align;
        lists.tile_prefix[0] = 0;
        lists.tile_prefix[1 + slot + (count > 0 ? 1 : 0)] = shared_tiles + before + tiles;   // total, after the last active
    }
    if (lists.tile_prefix_wide == nullptr) return;
    const int wide = lists.tile_rows_wide;
    const int tiles_w = (count + wide - 1) / wide;
    const int shared_w = (rows + wide - 1) / wide;
    const int before_w = block_exclusive_scan_256<PART>(tiles_w, scan_scratch);
    if (count > 0) lists.tile_prefix_wide[1 + slot] = shared_w + before_w;
    if (e == kExperts - 1) {
        lists.tile_prefix_wide[0] = 0;
        lists.tile_prefix_wide[1 + slot + (count > 0 ? 1 : 0)] = shared_w + before_w + tiles_w;
    }
}

// ---- single-block path (assignments <= kSmallMax) ---------------------------
// Both passes of a warp are chains of dependent 32-wide steps, so the ids are spread over 32 warps (4,096 assignments: four
// steps).  What lies in position order is put together in shared memory and leaves as whole lines: scattered 4-byte
// stores of one SM and the matching of ids bound the kernel before (15.5 us at 4,096 assignments, now 11.4).
constexpr int kSmallThreads = 32 * kSmallWarps;
__global__ void __launch_bounds__(kSmallThreads) permute_small_kernel(
    const std::int32_t* __restrict__ ids, int assignments, std::int32_t* order,
    std::int32_t* position, RouteLists lists, std::int32_t* row_token, std::int32_t* pp_of_flat,
    std::int32_t* status, IdRange range, int shared_rows) {
    __shared__ std::uint16_t hist[kSmallWarps][kExperts];            // counts, then positions within the expert
    __shared__ std::int16_t cached_ids[kSmallWarps][kSmallChunk];
    __shared__ std::uint16_t order_image[kSmallMax];
    __shared__ std::int32_t segment_total[kSmallThreads];
    __shared__ std::int32_t positions;
    __shared__ std::int32_t expert_base[kExperts];
    __shared__ std::int32_t scan_scratch[kWarps];
    __shared__ std::int32_t pp_delta[kExperts];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int per_warp = ((assignments + kSmallWarps - 1) / kSmallWarps + 31) / 32 * 32;
    const int begin = min(assignments, warp * per_warp);
    const int end = min(assignments, begin + per_warp);
    // the warp's ids once into shared memory, all loads in flight together: the two passes below would otherwise pay a
    // global-memory round trip per step
    load_chunk_ids(ids, begin, end, cached_ids[warp]);
    warp_histogram(ids, begin, end, hist[warp], status, cached_ids[warp], range);
    __syncthreads();
    // exclusive prefix over the warps, per expert: four threads of eight warps' counts each
    const int e = threadIdx.x % kExperts;
    constexpr int kPerSegment = kSmallWarps * kExperts / kSmallThreads;
    const int first_warp = threadIdx.x / kExperts * kPerSegment;
    int count[kPerSegment];
    int sum = 0;
#pragma unroll
    for (int wi = 0; wi < kPerSegment; ++wi) {
        count[wi] = hist[first_warp + wi][e];
        sum += count[wi];
    }
    segment_total[threadIdx.x] = sum;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int s = 0; s < kSmallThreads / kExperts; ++s) {
        const int v = segment_total[s * kExperts + e];
        if (s * kPerSegment < first_warp) before += v;
        total += v;
    }
#pragma unroll
    for (int wi = 0; wi < kPerSegment; ++wi) {
        hist[first_warp + wi][e] = static_cast<std::uint16_t>(before);
        before += count[wi];
    }
    const int rows = shared_rows >= 0 ? shared_rows : assignments / kTop;
    if (threadIdx.x < kExperts) {
        const int offset = block_exclusive_scan_256<true>(total, scan_scratch);
        write_route_lists<true>(e, total, offset, assignments, rows, lists, scan_scratch);
        expert_base[e] = offset;
        if (e == kExperts - 1) positions = offset + total;
        pp_delta[e] = (pp_of_flat != nullptr && lists.pp_off != nullptr) ? lists.pp_off[e] - offset : 0;       // write_route_lists stored both just above
    }
    __syncthreads();
    const int tile_shift = pp_of_flat != nullptr && lists.tile_rows < 64 ? 31 - __clz(lists.tile_rows) : 0;
    warp_scatter(ids, begin, end, hist[warp], expert_base, order_image, position, static_cast<std::int32_t*>(nullptr), pp_delta,
                 pp_of_flat, cached_ids[warp], range, tile_shift);
    __syncthreads();
    for (int at = threadIdx.x; at < positions; at += kSmallThreads) {
        const int i = order_image[at];
        if (order != nullptr) order[at] = i;
        if (row_token != nullptr) row_token[at] = i / kTop;
    }
    if (row_token != nullptr) {
        for (int t = threadIdx.x; t < rows; t += blockDim.x) {
            row_token[assignments + t] = t;
            if (pp_of_flat != nullptr) pp_of_flat[assignments + t] = lists.pp_off[kExperts] + t;
        }
    }
}

// ---- multi-block path -------------------------------------------------------
__global__ void __launch_bounds__(256) permute_hist_kernel(const std::int32_t* __restrict__ ids,
                                                           int assignments,
                                                           std::int32_t* __restrict__ chunk_hist,
                                                           std::int32_t* status, IdRange range) {
    __shared__ std::int32_t hist[kWarps][kExperts];
    __shared__ std::int16_t cached_ids[kWarps][kChunk];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int chunk = blockIdx.x * kWarps + warp;
    const int begin = min(assignments, chunk * kChunk);
    const int end = min(assignments, begin + kChunk);
    load_chunk_ids(ids, begin, end, cached_ids[warp]);
    warp_histogram(ids, begin, end, hist[warp], status, cached_ids[warp], range);
    if (begin < assignments) {
        for (int e = lane; e < kExperts; e += 32) chunk_hist[static_cast<std::size_t>(chunk) * kExperts + e] = hist[warp][e];
    }
}

// Exclusive prefix over the chunks, per expert, then the lists.  gridDim.x blocks of 1024 threads share the experts
// (256 / gridDim.x each); an expert has 1024 / that many threads, each owning a slice of the chunks: a sum pass, the
// slice bases through shared memory, then the pass that writes the prefixes.  The block that finishes last (a counter,
// reset by that block for the next call) adds the scan over the 256 expert totals and writes the lists.  One thread
// per expert walking 512 chunks took 60 µs at 131,072 assignments, one block with four threads per expert 22 µs.
constexpr int kScanThreads = 1024;
constexpr int kScanBlocksLarge = 8;
__global__ void __launch_bounds__(kScanThreads) permute_scan_kernel(std::int32_t* __restrict__ chunk_hist, int chunks,
                                                                    int assignments, RouteLists lists, int shared_rows,
                                                                    unsigned* __restrict__ blocks_done) {
    __shared__ std::int32_t scan_scratch[kWarps];
    __shared__ std::int32_t segment_total[kScanThreads];
    __shared__ int is_last;
    pdl_launch_dependents();
    pdl_wait();
    const int experts_here = kExperts / static_cast<int>(gridDim.x);          // 256 or 32
    const int segments = kScanThreads / experts_here;                        // 4 or 32
    const int e_local = threadIdx.x % experts_here;
    const int segment = threadIdx.x / experts_here;
    const int e = static_cast<int>(blockIdx.x) * experts_here + e_local;
    const int per_segment = (chunks + segments - 1) / segments;
    const int first = min(chunks, segment * per_segment);
    const int last = min(chunks, first + per_segment);
    int sum = 0;
#pragma unroll 16
    for (int c = first; c < last; ++c) sum += chunk_hist[static_cast<std::size_t>(c) * kExperts + e];
    segment_total[segment * experts_here + e_local] = sum;
    __syncthreads();
    int running = 0, total = 0;
    for (int s = 0; s < segments; ++s) {
        const int v = segment_total[s * experts_here + e_local];
        if (s < segment) running += v;
        total += v;
    }
#pragma unroll 16
    for (int c = first; c < last; ++c) {
        const std::size_t at = static_cast<std::size_t>(c) * kExperts + e;
        const int v = chunk_hist[at];
        chunk_hist[at] = running;
        running += v;
    }
    if (segment == 0) lists.counts[e] = total;
    // the last block to get here sees every block's totals
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned before = atomicAdd(blocks_done, 1U);
        is_last = before + 1U == gridDim.x ? 1 : 0;
        if (is_last) *blocks_done = 0U;
    }
    __syncthreads();
    if (!is_last || threadIdx.x >= kExperts) return;   // whole warps leave; the block-wide barriers below count the rest
    __threadfence();
    const int expert = threadIdx.x;
    const int expert_total = __ldcg(lists.counts + expert);
    const int offset = block_exclusive_scan_256(expert_total, scan_scratch);
    write_route_lists(expert, expert_total, offset, assignments, shared_rows >= 0 ? shared_rows : assignments / kTop, lists,
                      scan_scratch);
}

__global__ void __launch_bounds__(256) permute_scatter_kernel(
    const std::int32_t* __restrict__ ids, int assignments, const std::int32_t* __restrict__ chunk_hist,
    const std::int32_t* __restrict__ offsets, std::int32_t* order, std::int32_t* position,
    std::int32_t* row_token, const std::int32_t* __restrict__ pp_off, std::int32_t* pp_of_flat, IdRange range,
    int shared_rows) {
    __shared__ std::int32_t running[kWarps][kExperts];
    __shared__ std::int32_t pp_delta[kExperts];
    __shared__ std::int16_t cached_ids[kWarps][kChunk];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int chunk = blockIdx.x * kWarps + warp;
    const int begin = min(assignments, chunk * kChunk);
    const int end = min(assignments, begin + kChunk);
    load_chunk_ids(ids, begin, end, cached_ids[warp]);
    pp_delta[threadIdx.x] = pp_of_flat != nullptr ? pp_off[threadIdx.x] - offsets[threadIdx.x] : 0;
    if (begin < assignments) {
        for (int e = lane; e < kExperts; e += 32) {
            running[warp][e] = offsets[e] + chunk_hist[static_cast<std::size_t>(chunk) * kExperts + e];
        }
    }
    __syncthreads();
    warp_scatter(ids, begin, end, running[warp], nullptr, order, position, row_token, pp_delta, pp_of_flat,
                 cached_ids[warp], range);
    if (row_token != nullptr) {
        const int rows = shared_rows >= 0 ? shared_rows : assignments / kTop;
        const int t = blockIdx.x * blockDim.x + threadIdx.x;
        if (t < rows) {
            row_token[assignments + t] = t;
            if (pp_of_flat != nullptr) pp_of_flat[assignments + t] = pp_off[kExperts] + t;
        }
    }
}

// ---- places of the block's own routing -------------------------------------------------------
// The tensor-core router has counted the experts of every chunk of 32 tokens while it chose them, a token's eight ids are
// different, and so the rank of an assignment in its chunk is the number of earlier tokens of the chunk that have the expert
// too: eight votes of a warp whose lane l holds token l's ids.  Positions, lists and the quantised row are then one pass
// over the tokens instead of two kernels (up to 5,120 assignments; 512 rows: 13.7 + 6.4 us, now 9.4) or four (4,096 rows:
// 6 + 12 + 12 + 22 us, now 12 + 24, with the scales by row 12 + 19).
// Every block adds the counts up for itself, one expert per thread: whole spans of 512 tokens, which the router counts too, and the
// chunks of its own span; block 0 writes the lists.  At 8,192 tokens that is 31 words per thread from the L2.
// SCANNED, above that: permute_scan_kernel has turned the counts into prefixes over the chunks and written the lists.  It takes 12 us;
// at 16,384 tokens the words would cost the place kernel 9, at 4,096 they cost nothing that shows (whole calls 422.6 -> 416.9 us
// without the scan kernel).
constexpr int kPlaceRows = 8192;                 // up to here without a scan kernel
constexpr int kSpanChunks = 16;                  // chunks of 32 tokens whose counts are also kept as one
constexpr int kPlacePad = 128;                   // an expert's rows start on a multiple of this
template <int WARPS, bool SCANNED, int PER_LANE>
__global__ void __launch_bounds__(256) place_rows_kernel(const std::uint16_t* __restrict__ x, const std::int32_t* __restrict__ ids,
                                                         const std::int32_t* __restrict__ chunk_hist,
                                                         const std::int32_t* __restrict__ span_hist, RouteLists lists,
                                                         std::int32_t* __restrict__ order, std::int32_t* __restrict__ position,
                                                         std::int32_t* __restrict__ row_token, std::int32_t* __restrict__ pp_of_flat,
                                                         std::uint8_t* __restrict__ xq, std::uint8_t* __restrict__ xs, int rows, int hidden,
                                                         float global_scale) {
    __shared__ std::int32_t scan_scratch[kWarps];
    __shared__ std::int32_t first_position[kExperts], first_place[kExperts];        // of this chunk's rows of an expert
    __shared__ std::int32_t shared_place;
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // (the tokens of a block are of one chunk; !SCANNED: block 0 has none)
    const int token = (static_cast<int>(blockIdx.x) - (SCANNED ? 0 : 1)) * (kWarps / WARPS) + warp / WARPS;
    const int chunk = token >> 5;
    const int in_chunk = token & 31;
    QuantisedRow<WARPS, PER_LANE> row;             // the row is on its way while its places are found
    if (token >= 0 && token < rows) row.load(x + static_cast<std::size_t>(token) * hidden, hidden, warp % WARPS);
    if constexpr (!SCANNED) {
        const int e = threadIdx.x;
        const int spans = (rows + 32 * kSpanChunks - 1) / (32 * kSpanChunks);
        const int my_span = max(chunk, 0) / kSpanChunks;
        // all of the span's chunks in one round trip
        int of_chunk[kSpanChunks - 1];
#pragma unroll
        for (int i = 0; i < kSpanChunks - 1; ++i) {
            const int c = my_span * kSpanChunks + i;
            of_chunk[i] = c < chunk ? __ldcg(chunk_hist + c * kExperts + e) : 0;
        }
        int total = 0, before = 0;
#pragma unroll 8
        for (int s = 0; s < spans; ++s) {
            const int n = __ldcg(span_hist + s * kExperts + e);
            total += n;
            if (s < my_span) before += n;
        }
#pragma unroll
        for (int i = 0; i < kSpanChunks - 1; ++i) before += of_chunk[i];
        // both prefixes in one scan: at most 65,536 assignments and 512 + 256 pads
        static_assert(kPlaceRows * kTop < 1 << 18 && kPlaceRows * kTop / kPlacePad + kExperts < 1 << 13, "two fields of a word");
        const int pads = (total + kPlacePad - 1) / kPlacePad;
        const int prefix = block_exclusive_scan_256(pads << 18 | total, scan_scratch);
        const int position0 = prefix & ((1 << 18) - 1), pad0 = prefix >> 18;
        if (blockIdx.x == 0) {
            write_route_lists(e, total, position0, rows * kTop, rows, lists, scan_scratch);
            return;
        }
        first_position[e] = position0 + before;
        first_place[e] = pad0 * kPlacePad + before;
        if (e == kExperts - 1) shared_place = (pad0 + pads) * kPlacePad;
        __syncthreads();
    }
    if (token >= rows) return;
    // lane l holds the ids of the chunk's token l
    int id[kTop];
    {
        const int4* at = reinterpret_cast<const int4*>(ids + static_cast<std::size_t>(min(chunk * 32 + lane, token)) * kTop);
        const int4 a = __ldcg(at), b = __ldcg(at + 1);
        id[0] = a.x; id[1] = a.y; id[2] = a.z; id[3] = a.w;
        id[4] = b.x; id[5] = b.y; id[6] = b.z; id[7] = b.w;
    }
    int my_id = 0, my_rank = 0;                      // lane k < 8: of the token's slot k
#pragma unroll
    for (int k = 0; k < kTop; ++k) {
        const int e = __shfl_sync(0xffffffffU, id[k], in_chunk);
        bool has = false;
#pragma unroll
        for (int i = 0; i < kTop; ++i) has = has || id[i] == e;
        const int rank = __popc(__ballot_sync(0xffffffffU, has && lane < in_chunk));
        if (lane == k) {
            my_id = e & (kExperts - 1);
            my_rank = rank;
        }
    }
    int my_place = 0;
    if (lane < kTop) {
        int pos;
        if constexpr (SCANNED) {
            const int before = __ldcg(chunk_hist + static_cast<std::size_t>(chunk) * kExperts + my_id) + my_rank;
            pos = __ldcg(lists.offsets + my_id) + before;
            my_place = __ldcg(lists.pp_off + my_id) + before;
        } else {
            pos = first_position[my_id] + my_rank;
            my_place = first_place[my_id] + my_rank;
        }
        if (WARPS == 1 || warp % WARPS == 0) {
            const int i = token * kTop + lane;
            order[pos] = i;
            position[i] = pos;
            row_token[pos] = token;
            pp_of_flat[i] = my_place;
        }
    } else if (lane == kTop) {
        if constexpr (SCANNED) my_place = __ldcg(lists.pp_off + kExperts) + token; else my_place = shared_place + token;
        if (WARPS == 1 || warp % WARPS == 0) {
            row_token[rows * kTop + token] = token;
            pp_of_flat[rows * kTop + token] = my_place;
        }
    }
    row.quantise(global_scale);
#pragma unroll 1
    for (int place = 0; place <= kTop; ++place) {
        row.template store<WARPS == 1>(xq, xs, static_cast<std::size_t>(__shfl_sync(0xffffffffU, my_place, place)));
    }
}

// ---- lists, places and rows of a call on ids that come from the caller -------------------------------
// Up to 512 assignments (64 tokens) the front of an operator call is one kernel: every block counts the experts for itself
// (shared-memory atomics, a scan of the 256 counts), and a warp per assignment finds its rank from votes over the earlier ids,
// its padded position, and brings its row there; block 0 writes the lists.  As permutation and row kernel the two took a
// launch more: the operator sequence of four layers at four rows took 284 us, now 271.
// SOURCE 0: rows of a caller that has quantised them, with the tensor maps of the matrices in place; 1: BF16 rows, quantised here.
constexpr int kFrontMax = 512;
struct FrontRows {
    const std::uint8_t* packed;              // SOURCE 0
    const std::uint8_t* scales_swizzled;
    const std::uint16_t* rows;               // SOURCE 1
    std::uint8_t* xq;
    std::uint8_t* xs;
    int width;                               // elements of a row
    int distinct;                            // 1: a row per assignment, 0: the eight slots of a token share its row
};
template <int SOURCE>
__global__ void __launch_bounds__(256) assignment_rows_kernel(const std::int32_t* __restrict__ ids, int assignments, RouteLists lists,
                                                              std::int32_t* __restrict__ order, std::int32_t* __restrict__ position,
                                                              std::int32_t* __restrict__ row_token, std::int32_t* __restrict__ pp_of_flat,
                                                              std::int32_t* status, FrontRows from, const __grid_constant__ TableMaps maps) {
    __shared__ __align__(128) std::uint32_t map_image[kWarps][32];
    __shared__ std::int32_t cached_ids[kFrontMax];
    __shared__ std::int32_t counts[kExperts], first_position[kExperts], first_place[kExperts];
    __shared__ std::int32_t scan_scratch[kWarps];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int e = threadIdx.x;
    counts[e] = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < assignments; j += 256) {
        const int id = ids[j];
        if ((id < 0 || id >= kExperts) && blockIdx.x == 0) atomicCAS(status, kStatusOk, kStatusBadExpertId);
        const int clamped = id < 0 ? 0 : (id >= kExperts ? kExperts - 1 : id);
        cached_ids[j] = clamped;
        atomicAdd(counts + clamped, 1);
    }
    __syncthreads();
    // positions and padded positions in one scan: at most 512 assignments, each in a 128-row pad of its own
    const int count = counts[e];
    const bool spaced = lists.tile_rows < 64;                    // tiles of 16 or 32 rows lie a pad apart
    const int pads = spaced ? (count + lists.tile_rows - 1) / lists.tile_rows : (count + kPlacePad - 1) / kPlacePad;
    const int prefix = block_exclusive_scan_256(pads << 16 | count, scan_scratch);
    first_position[e] = prefix & 0xffff;
    first_place[e] = (prefix >> 16) * kPlacePad;
    __syncthreads();
    const int i = static_cast<int>(blockIdx.x) * kWarps + warp;
    if (i < assignments) {
        const int mine = cached_ids[i];
        int rank = 0;
        for (int step = 0; step < i; step += 32) {
            const int j = step + lane;
            rank += __popc(__ballot_sync(0xffffffffU, j < i && cached_ids[j] == mine));
        }
        const int gaps = spaced ? rank / lists.tile_rows * (kPlacePad - lists.tile_rows) : 0;
        const int place = first_place[mine] + rank + gaps;
        if (lane == 0) {
            const int pos = first_position[mine] + rank;
            order[pos] = i;
            position[i] = pos;
            row_token[pos] = i / kTop;
            pp_of_flat[i] = place;
        }
        const std::size_t row = static_cast<std::size_t>(from.distinct ? i : i / kTop);
        if constexpr (SOURCE == 0) {
            if (rank == 0) {
                for (int k = 0; k < maps.kinds; ++k) {
                    expert::build_table_map(maps, mine * 3 + maps.first_kind + k, map_image[warp]);
                    __syncwarp();
                }
            }
            expert::copy_quantised_row(from.packed, from.scales_swizzled, row, from.xq, from.xs, place, from.width / 2);
        } else {
            QuantisedRow<1> quantised;
            quantised.load(from.rows + row * from.width, from.width, 0);
            quantised.quantise(1.0F);
            quantised.store(from.xq, from.xs, place);
        }
    }
    if (blockIdx.x == 0) {
        const int rows = assignments / kTop;
        write_route_lists(e, count, prefix & 0xffff, assignments, rows, lists, scan_scratch);
        const int shared_place = __shfl_sync(0xffffffffU, ((prefix >> 16) + pads) * kPlacePad, 31);      // behind the last expert's: warp 7's lane 31
        if (warp == kWarps - 1) {
            for (int t = lane; t < rows; t += 32) {
                row_token[assignments + t] = t;
                pp_of_flat[assignments + t] = shared_place + t;
            }
        }
    }
}

// ---- decode front end: top-8 + permutation + lists + NVFP4 token rows, one block ------------
// For up to 8 tokens the three routing stages are a few microseconds of work each, so they run as
// one 256-thread block instead of three launches: warp w ranks token w; thread e counts expert e
// (the ranking law of cuda/nvfp4_grouped.cu:117-132 evaluated directly: 64 assignments at most);
// then every thread quantises 16-element blocks of the token rows (cuda/nvfp4_ops.cu:818-841) and
// stores them once per destination row of the padded position space, scales in the 128x4 tiling.
constexpr int kFusedMaxRows = 8;

__global__ void __launch_bounds__(256) route_fused_kernel(
    const float* __restrict__ logits, const float* __restrict__ bias, std::int32_t* __restrict__ ids,
    float* __restrict__ weights, float routed_scale, int rows, std::int32_t* __restrict__ order,
    std::int32_t* __restrict__ position, RouteLists lists, std::int32_t* __restrict__ row_token,
    std::int32_t* __restrict__ pp_of_flat, const std::uint16_t* __restrict__ x, std::uint8_t* __restrict__ xq,
    std::uint8_t* __restrict__ xs, int hidden, float quant_scale) {
    __shared__ std::int32_t s_ids[kFusedMaxRows * kTop];
    __shared__ std::int32_t s_pp[kFusedMaxRows * (kTop + 1)];
    __shared__ std::int32_t scan_scratch[kWarps];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int assignments = rows * kTop;
    if (warp < rows) {
        warp_top8(logits + static_cast<std::size_t>(warp) * kExperts, bias, ids + warp * kTop, weights + warp * kTop,
                  routed_scale);
    }
    __syncthreads();
    if (threadIdx.x < assignments) s_ids[threadIdx.x] = ids[threadIdx.x];
    __syncthreads();
    const int e = threadIdx.x;
    int count = 0;
    for (int j = 0; j < assignments; ++j) count += s_ids[j] == e;
    const int offset = block_exclusive_scan_256(count, scan_scratch);
    write_route_lists(e, count, offset, assignments, rows, lists, scan_scratch);
    __syncthreads();
    if (threadIdx.x < assignments) {
        const int i = threadIdx.x;
        const int mine = s_ids[i];
        int rank = 0;
        for (int j = 0; j < i; ++j) rank += s_ids[j] == mine;
        const int pos = lists.offsets[mine] + rank;
        order[pos] = i;
        position[i] = pos;
        row_token[pos] = i / kTop;
        const int pp = lists.pp_off[mine] + rank;
        pp_of_flat[i] = pp;
        s_pp[i] = pp;
    } else if (threadIdx.x < assignments + rows) {
        const int t = threadIdx.x - assignments;
        row_token[assignments + t] = t;
        const int pp = lists.pp_off[kExperts] + t;
        pp_of_flat[assignments + t] = pp;
        s_pp[assignments + t] = pp;
    }
    __syncthreads();
    const int blocks = hidden / 16;
    const int col_blocks = (blocks + 3) / 4;
    for (int idx = threadIdx.x; idx < rows * blocks; idx += blockDim.x) {
        const int token = idx / blocks;
        const int b = idx - token * blocks;
        const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<std::size_t>(token) * hidden + b * 16);
        const uint4 lo = __ldg(src);
        const uint4 hi = __ldg(src + 1);
        const std::uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        float v[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[2 * i] = __uint_as_float(words[i] << 16);
            v[2 * i + 1] = __uint_as_float(words[i] & 0xffff0000U);
        }
        std::uint8_t scale_bits;
        const uint2 packed = quantize_block16(v, quant_scale, &scale_bits);
#pragma unroll
        for (int slot = 0; slot <= kTop; ++slot) {
            const std::size_t pp =
                static_cast<std::size_t>(s_pp[slot < kTop ? token * kTop + slot : assignments + token]);
            *reinterpret_cast<uint2*>(xq + pp * (hidden / 2) + b * 8) = packed;
            xs[((pp >> 7) * col_blocks + (b >> 2)) * 512 + (pp & 31) * 16 + ((pp >> 5) & 3) * 4 + (b & 3)] = scale_bits;
        }
    }
}

// Front of a call without routing (the dense MLP): all `rows` rows belong to entry 256 (the bank's last entry), which
// starts at padded position 0, and no routed expert has rows; block 0 writes these lists, and every block quantises its
// rows in place of the permutation and quantisation kernels.  WARPS per row: 8 while one per row would leave most of the
// chip idle (33 to 64 rows: lists and a warp per row took 7 us in two kernels), else 1.
template <int WARPS>
__global__ void __launch_bounds__(256) dense_front_kernel(RouteLists lists, int rows, const std::uint16_t* __restrict__ x,
                                                          std::uint8_t* __restrict__ xq, std::uint8_t* __restrict__ xs, int hidden,
                                                          float quant_scale) {
    pdl_launch_dependents();
    pdl_wait();
    if (blockIdx.x == 0) {
        const int e = threadIdx.x;
        lists.counts[e] = 0;
        lists.offsets[e] = 0;
        lists.pp_off[e] = 0;
        if (e == 0) {
            lists.counts[kExperts] = rows;
            lists.offsets[kExperts] = 0;
            lists.offsets[kExperts + 1] = rows;
            lists.active[0] = kExperts;
            *lists.active_count = 1;
            lists.pp_off[kExperts] = 0;
            lists.pp_off[kExperts + 1] = (rows + lists.pad_align - 1) / lists.pad_align * lists.pad_align;
            lists.tile_prefix[0] = 0;
            lists.tile_prefix[1] = (rows + lists.tile_rows - 1) / lists.tile_rows;
            if (lists.tile_prefix_wide != nullptr) {
                lists.tile_prefix_wide[0] = 0;
                lists.tile_prefix_wide[1] = (rows + lists.tile_rows_wide - 1) / lists.tile_rows_wide;
            }
        }
    }
    const int warp = threadIdx.x >> 5;
    const int row = (blockIdx.x * 8 + warp) / WARPS;
    if (row >= rows) return;
    const int blocks = hidden / 16;
    const std::size_t col_blocks = static_cast<std::size_t>(blocks / 4);              // hidden is a multiple of 128
    std::uint8_t* row_q = xq + static_cast<std::size_t>(row) * (hidden / 2);
    std::uint8_t* row_s = xs + (row >> 7) * col_blocks * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4;
#pragma unroll 2
    for (int b = warp % WARPS * 32 + (threadIdx.x & 31); b < blocks; b += 32 * WARPS) {
        const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<std::size_t>(row) * hidden + b * 16);
        const uint4 lo = __ldg(src);
        const uint4 hi = __ldg(src + 1);
        const std::uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        float v[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[2 * i] = __uint_as_float(words[i] << 16);
            v[2 * i + 1] = __uint_as_float(words[i] & 0xffff0000U);
        }
        std::uint8_t scale_bits;
        const uint2 packed = quantize_block16(v, quant_scale, &scale_bits);
        *reinterpret_cast<uint2*>(row_q + b * 8) = packed;
        row_s[(b >> 2) * 512 + (b & 3)] = scale_bits;
    }
}

}  // namespace

int route_fused_max_rows() { return kFusedMaxRows; }

namespace {
// The lists that the block's expert kernels read, at 128 padded positions per started 128 rows.
RouteLists plan_lists(p92b_plan* plan, int tile_rows) {
    RouteLists lists {};
    lists.counts = plan->counts;
    lists.offsets = plan->offsets;
    lists.active = plan->active;
    lists.active_count = plan->active_count;
    lists.enabled = true;
    lists.pad_align = kPlacePad;
    lists.tile_rows = tile_rows;
    lists.pp_off = plan->pp_off;
    lists.tile_prefix = plan->tile_prefix;
    const bool wide = tile_rows == 64;
    lists.tile_rows_wide = wide ? 128 : tile_rows;
    lists.tile_prefix_wide = wide ? plan->tile_prefix_wide : nullptr;
    plan->wide_rows = wide ? 128 : 0;
    return lists;
}
}  // namespace

cudaError_t launch_dense_front(p92b_plan* plan, const std::uint16_t* x, int rows, int tile_rows, cudaStream_t stream, bool pdl) {
    const RouteLists lists = plan_lists(plan, tile_rows);
    plan->last_launches += 1;
    const bool few = rows <= 1024;
    return launch_kernel(few ? dense_front_kernel<8> : dense_front_kernel<1>, dim3(few ? rows : (rows + 7) / 8), dim3(256), 0, stream,
                         pdl, lists, rows, x, plan->xq_pp, plan->xs_sw, plan->hidden, 1.0F);
}

namespace {
cudaError_t launch_assignment_rows(p92b_plan* plan, const std::int32_t* ids, int assignments, int tile_rows, const FrontRows& from,
                                   const TableMaps* maps, cudaStream_t stream, bool pdl) {
    plan->last_launches += 1;
    const RouteLists lists = plan_lists(plan, tile_rows);
    return launch_kernel(maps != nullptr ? assignment_rows_kernel<0> : assignment_rows_kernel<1>, dim3((assignments + kWarps - 1) / kWarps),
                         dim3(256), 0, stream, pdl, ids, assignments, lists, plan->order, plan->position, plan->row_token,
                         plan->pp_of_flat, plan->status, from, maps != nullptr ? *maps : TableMaps {});
}
}  // namespace

cudaError_t launch_quantised_assignments(p92b_plan* plan, const std::int32_t* ids, int assignments, int tile_rows,
                                         const std::uint8_t* packed, const std::uint8_t* scales_swizzled, bool down, int k_bytes,
                                         bool distinct_rows, const TableMaps& maps, cudaStream_t stream, bool pdl) {
    if (packed == nullptr || scales_swizzled == nullptr || assignments <= 0 || k_bytes % 16 != 0 || !aligned_to(16, packed)) {
        return cudaErrorInvalidValue;
    }
    std::uint8_t* xq = down ? plan->hq_pp : plan->xq_pp;
    std::uint8_t* xs = down ? plan->hs_sw : plan->xs_sw;
    if (assignments <= kFrontMax) {
        return launch_assignment_rows(plan, ids, assignments, tile_rows, FrontRows {packed, scales_swizzled, nullptr, xq, xs, 2 * k_bytes, distinct_rows},
                                      &maps, stream, pdl);
    }
    cudaError_t st = launch_permute(plan, ids, assignments, plan->order, plan->position, plan->counts, plan->offsets, true, kPlacePad,
                                    tile_rows, stream, pdl);
    if (st != cudaSuccess) return st;
    plan->last_launches += 1;
    return launch_gather_quantized_rows(packed, scales_swizzled, plan->pp_of_flat, xq, xs, assignments, k_bytes, distinct_rows, maps,
                                        stream, pdl);
}

cudaError_t launch_token_assignments(p92b_plan* plan, const std::int32_t* ids, const std::uint16_t* x, int rows, int tile_rows, bool down,
                                     cudaStream_t stream, bool pdl) {
    const int width = down ? plan->intermediate : plan->hidden;
    if (!down && width > 4096) return cudaErrorNotSupported;
    if (!aligned_to(16, x)) return cudaErrorInvalidValue;
    if (rows * kTop <= kFrontMax && width <= 4096) {
        return launch_assignment_rows(plan, ids, rows * kTop, tile_rows,
                                      FrontRows {nullptr, nullptr, x, down ? plan->hq_pp : plan->xq_pp, down ? plan->hs_sw : plan->xs_sw, width, down},
                                      nullptr, stream, pdl);
    }
    cudaError_t st = launch_permute(plan, ids, rows * kTop, plan->order, plan->position, plan->counts, plan->offsets, true, kPlacePad,
                                    tile_rows, stream, pdl);
    if (st != cudaSuccess) return st;
    plan->last_launches += 1;
    // the down operator's rows are the (row, slot) intermediate rows, each quantised on its own (src/executor.cpp:85-91)
    return down ? launch_quantize_rows_to_pp(x, plan->pp_of_flat, plan->hq_pp, plan->hs_sw, rows * kTop, width, stream, pdl)
                : launch_quantize_padded(plan, x, rows, stream, pdl);
}

cudaError_t launch_route_fused(p92b_plan* plan, const float* bias, float routed_scale, const std::uint16_t* x,
                               int rows, int pad_align, int tile_rows, cudaStream_t stream, bool pdl) {
    if (rows <= 0 || rows > kFusedMaxRows || !aligned_to(16, x)) return cudaErrorInvalidValue;
    RouteLists lists {};
    lists.counts = plan->counts;
    lists.offsets = plan->offsets;
    lists.active = plan->active;
    lists.active_count = plan->active_count;
    lists.enabled = true;
    lists.pad_align = pad_align;
    lists.tile_rows = tile_rows;
    lists.pp_off = plan->pp_off;
    lists.tile_prefix = plan->tile_prefix;
    lists.tile_rows_wide = tile_rows;
    lists.tile_prefix_wide = nullptr;
    plan->wide_rows = 0;
    plan->last_launches += 1;
    return launch_kernel(route_fused_kernel, dim3(1), dim3(256), 0, stream, pdl, plan->logits, bias, plan->ids,
                         plan->route_weights, routed_scale, rows, plan->order, plan->position, lists, plan->row_token,
                         plan->pp_of_flat, x, plan->xq_pp, plan->xs_sw, plan->hidden, 1.0F);
}

cudaError_t launch_scan_counts(p92b_plan* plan, int rows, int tile_rows, cudaStream_t stream, bool pdl) {
    if (rows <= kPlaceRows) return cudaSuccess;
    const int chunks = (rows + 31) / 32;
    plan->last_launches += 1;
    return launch_kernel(permute_scan_kernel, dim3(kScanBlocksLarge), dim3(kScanThreads), 0, stream, pdl,
                         plan->chunk_hist, chunks, rows * kTop, plan_lists(plan, tile_rows), rows, plan->scan_blocks_done);
}

// Up to 1,024 rows eight warps per row and tiled scales: the stores of the scales don't show there, and 64 rows, where the gate/up
// product waits for memory throughout, took 747 us instead of 743 with scales by row.
bool place_scales_by_row(int rows) { return rows > 1024; }

cudaError_t launch_place_rows(p92b_plan* plan, const std::uint16_t* x, int rows, int tile_rows, cudaStream_t stream, bool pdl) {
    if (plan->hidden > 4096) return cudaErrorNotSupported;
    if (!aligned_to(16, x)) return cudaErrorInvalidValue;
    const bool scanned = rows > kPlaceRows;
    const bool few = !place_scales_by_row(rows);
    const bool narrow = plan->hidden <= 2560;
    plan->last_launches += 1;
    return launch_kernel(few       ? place_rows_kernel<8, false, 1>
                         : scanned ? narrow ? place_rows_kernel<1, true, 5> : place_rows_kernel<1, true, 8>
                                   : narrow ? place_rows_kernel<1, false, 5> : place_rows_kernel<1, false, 8>,
                         dim3((few ? rows : (rows + 7) / 8) + (scanned ? 0 : 1)), dim3(256), 0, stream, pdl, x,
                         static_cast<const std::int32_t*>(plan->ids), static_cast<const std::int32_t*>(plan->chunk_hist),
                         static_cast<const std::int32_t*>(plan->span_hist), plan_lists(plan, tile_rows), plan->order, plan->position,
                         plan->row_token, plan->pp_of_flat, plan->xq_pp, plan->xs_sw, rows, plan->hidden, 1.0F);
}

cudaError_t launch_permute(p92b_plan* plan, const std::int32_t* ids, int assignments,
                           std::int32_t* order, std::int32_t* position, std::int32_t* counts,
                           std::int32_t* offsets, bool route_lists, int pad_align, int tile_rows,
                           cudaStream_t stream, bool pdl, int range_first, int range_count, int shared_rows) {
    IdRange range;
    if (range_count >= 0) {
        range.first = range_first;
        range.count = range_count;
        range.restricted = 1;
    }
    if (plan == nullptr || ids == nullptr || counts == nullptr || offsets == nullptr || assignments <= 0 ||
        assignments > plan->max_rows * kTop) {
        return cudaErrorInvalidValue;
    }
    RouteLists lists {};
    lists.counts = counts;
    lists.offsets = offsets;
    lists.active = plan->active;
    lists.active_count = plan->active_count;
    lists.enabled = route_lists;
    lists.pad_align = pad_align > 0 ? pad_align : 1;
    lists.tile_rows = tile_rows > 0 ? tile_rows : 1;
    const bool padded = route_lists && pad_align > 0;
    lists.pp_off = padded ? plan->pp_off : nullptr;
    lists.tile_prefix = padded ? plan->tile_prefix : nullptr;
    // more than 32 rows: a second prefix in 128-row tiles, which the kernels with the tokens on the M side and the slab kernel
    // of the down product count in; the 64-row one stays for the operators on a caller's weights and the un-fused results
    const bool wide = padded && tile_rows == 64;
    lists.tile_rows_wide = wide ? 128 : lists.tile_rows;
    lists.tile_prefix_wide = wide ? plan->tile_prefix_wide : nullptr;
    plan->wide_rows = wide ? 128 : 0;
    std::int32_t* row_token = route_lists ? plan->row_token : nullptr;
    std::int32_t* pp_of_flat = padded ? plan->pp_of_flat : nullptr;
    if (assignments <= kSmallMax) {
        plan->last_launches += 1;
        return launch_kernel(permute_small_kernel, dim3(1), dim3(kSmallThreads), 0, stream, pdl, ids, assignments, order, position,
                             lists, row_token, pp_of_flat, plan->status, range, shared_rows);
    }
    const int chunks = (assignments + kChunk - 1) / kChunk;
    if (chunks > plan->chunks) return cudaErrorInvalidValue;
    const int blocks = (chunks + kWarps - 1) / kWarps;
    plan->last_launches += 3;
    cudaError_t st = launch_kernel(permute_hist_kernel, dim3(blocks), dim3(256), 0, stream, pdl, ids, assignments,
                                   plan->chunk_hist, plan->status, range);
    if (st != cudaSuccess) return st;
    st = launch_kernel(permute_scan_kernel, dim3(chunks >= 64 ? kScanBlocksLarge : 1), dim3(kScanThreads), 0, stream, pdl,
                       plan->chunk_hist, chunks, assignments, lists, shared_rows, plan->scan_blocks_done);
    if (st != cudaSuccess) return st;
    return launch_kernel(permute_scatter_kernel, dim3(blocks), dim3(256), 0, stream, pdl,
                         static_cast<const std::int32_t*>(ids), assignments,
                         static_cast<const std::int32_t*>(plan->chunk_hist), static_cast<const std::int32_t*>(offsets),
                         order, position, row_token, static_cast<const std::int32_t*>(lists.pp_off), pp_of_flat, range,
                         shared_rows);
}

}  // namespace p92b

// ---------------------------------------------------------------------------
// Allocation-free permutation (p92b_moe_permute_static).
//
// For callers that cannot give the library a plan because they cannot allocate:
// the engine has already committed all device memory to its own arena, the host
// process forbids further CUDA allocations, or the call sits in a loop that must
// not run into the device-wide synchronisation cudaMalloc / cudaFree may cause.
// The scratch of the multi-block permutation lives in this file-scope device
// array instead.  Every GPU that loads the library carries its copy of the array
// (P92B_STATIC_PERMUTE_SCRATCH_BYTES) until the process exits.
//
// In host code the array's name is only a stand-in for the symbol, not a device
// address, so the address is fetched once per device with cudaGetSymbolAddress
// (that device current) and handed to the kernels as an ordinary pointer.
// Layout: [chunks][256] int32 chunk histograms, then the status word and the scan kernel's block counter.
//
// The address cache below is filled on first use per device.  Two host threads that make their
// first call on the same device at the same time both look the address up and both store the
// same value: harmless, but the kernels of their calls would still share the one array, so such
// calls have to be serialised by the caller for that reason anyway.
// ---------------------------------------------------------------------------
namespace {

constexpr int kStaticMaxAssignments = P92B_STATIC_PERMUTE_MAX_ASSIGNMENTS;
constexpr int kStaticChunks = kStaticMaxAssignments / p92b::kChunk;
constexpr int kStaticWords = kStaticChunks * p92b::kExperts + 64;
static_assert(kStaticWords * 4 == P92B_STATIC_PERMUTE_SCRATCH_BYTES, "header and array disagree");
constexpr int kStaticMaxDevices = 64;

static __device__ __align__(256) std::int32_t g_static_permute_scratch[kStaticWords];

std::int32_t* g_static_scratch_address[kStaticMaxDevices] = {};

// Device address of the array on the current device; looked up on first use.
cudaError_t static_scratch(std::int32_t** out) {
    int device = 0;
    cudaError_t st = cudaGetDevice(&device);
    if (st != cudaSuccess) return st;
    if (device < 0 || device >= kStaticMaxDevices) return cudaErrorNotSupported;
    if (g_static_scratch_address[device] == nullptr) {
        void* address = nullptr;
        st = cudaGetSymbolAddress(&address, g_static_permute_scratch);
        if (st != cudaSuccess) return st;
        g_static_scratch_address[device] = static_cast<std::int32_t*>(address);
    }
    *out = g_static_scratch_address[device];
    return cudaSuccess;
}

}  // namespace

extern "C" int p92b_moe_permute_static(const int32_t* expert_ids, int assignments, int32_t* order,
                                       int32_t* position, int32_t* counts, int32_t* offsets, void* stream_) {
    using namespace p92b;
    if (expert_ids == nullptr || counts == nullptr || offsets == nullptr || assignments <= 0) {
        return cudaErrorInvalidValue;
    }
    if (assignments > kStaticMaxAssignments) {
        std::fprintf(stderr,
                     "p92b_moe_permute_static: %d assignments exceed the built-in scratch (limit %d = %d rows x 8); "
                     "use p92b_moe_permute with a plan\n",
                     assignments, kStaticMaxAssignments, kStaticMaxAssignments / kTop);
        return cudaErrorInvalidValue;
    }
    std::int32_t* scratch = nullptr;
    cudaError_t st = static_scratch(&scratch);
    if (st != cudaSuccess) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    std::int32_t* chunk_hist = scratch;
    std::int32_t* status = scratch + kStaticChunks * kExperts;
    // the array still holds the previous call's words: the status word and the block counter must start at zero,
    // the histograms are fully rewritten by permute_hist_kernel before anything reads them
    st = cudaMemsetAsync(status, 0, 2 * sizeof(std::int32_t), stream);       // the status word and the scan's block counter
    if (st != cudaSuccess) return st;
    RouteLists lists {};
    lists.counts = counts;
    lists.offsets = offsets;
    lists.enabled = false;
    lists.pad_align = 1;
    lists.tile_rows = 1;
    lists.tile_rows_wide = 1;
    lists.tile_prefix_wide = nullptr;
    if (assignments <= kSmallMax) {
        permute_small_kernel<<<1, kSmallThreads, 0, stream>>>(expert_ids, assignments, order, position, lists, nullptr, nullptr,
                                                    status, IdRange(), -1);
        return cudaGetLastError();
    }
    const int chunks = (assignments + kChunk - 1) / kChunk;
    const int blocks = (chunks + kWarps - 1) / kWarps;
    permute_hist_kernel<<<blocks, 256, 0, stream>>>(expert_ids, assignments, chunk_hist, status, IdRange());
    permute_scan_kernel<<<chunks >= 64 ? p92b::kScanBlocksLarge : 1, p92b::kScanThreads, 0, stream>>>(
        chunk_hist, chunks, assignments, lists, -1, reinterpret_cast<unsigned*>(status + 1));
    permute_scatter_kernel<<<blocks, 256, 0, stream>>>(expert_ids, assignments, chunk_hist, offsets, order, position,
                                                       nullptr, nullptr, nullptr, IdRange(), -1);
    return cudaGetLastError();
}

// The status word of the calls above lives in the same built-in array, where a caller cannot
// reach it; this copies it out.  Like the permutation itself it allocates nothing: one
// cudaMemcpyAsync into the caller's host word, then a synchronisation of `stream`.
extern "C" int p92b_moe_permute_static_status(int32_t* host_status, void* stream_) {
    using namespace p92b;
    if (host_status == nullptr) return cudaErrorInvalidValue;
    std::int32_t* scratch = nullptr;
    cudaError_t st = static_scratch(&scratch);
    if (st != cudaSuccess) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    st = cudaMemcpyAsync(host_status, scratch + kStaticChunks * kExperts, sizeof(std::int32_t), cudaMemcpyDeviceToHost,
                         stream);
    if (st != cudaSuccess) return st;
    return cudaStreamSynchronize(stream);
}
