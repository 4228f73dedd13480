// What the grouped expert kernels share (expert_tc.cu: weights on the M side, a stream of weight tiles over few token
// columns; expert_rows.cu: tokens on the M side, for large batches): parameters, the routing lists in shared memory
// and the decoding of a work item.
#pragma once

#include "p92b_common.cuh"
#include "tc_ptx.cuh"

namespace p92b {
namespace expert {

using namespace ptx;

constexpr int kTileM = 128;
constexpr int kBlockKBytes = 128;                 // one swizzle row: 256 E2M1 values
constexpr int kSfSlab = 2048;                     // 128 rows x 16 scales of one K block
// Padded positions from one token tile of an expert to its next.  A tile's scale factors have to start at row 0 or 64 of a
// 128-row scale tile (another row's are at an address that the MMA does not take), so tiles of 16 or 32 rows lie a
// whole scale tile apart; an expert that no token picks twice has one such tile only.
template <int N>
constexpr int kTileStride = N < 64 ? 128 : N;

struct TcParams {
    BankView bank;
    RouteView route;
    const std::int32_t* pp_off;        // [258]
    const std::int32_t* tile_prefix;   // [active_count + 1]
    const std::uint8_t* b_sf;          // token-side scales, 128x4 tiled over padded positions
    std::uint8_t* hq;                  // MODE 0 out: packed SwiGLU rows [PP][I/2]
    std::uint8_t* hs;                  // MODE 0 out: their scales, 128x4 tiled over padded positions
    std::uint16_t* out;                // MODE 1 out: BF16 down rows [PP][H]
    std::int32_t* status;
    float quant_scale;                 // 1.0, passed at run time so the quantiser's divisions stay run-time operations
    int k_bytes;                       // K/2: bytes per operand row
    int m_total;                       // output rows per expert matrix
    int m_tiles;
    int routing_is_upstream;           // 1: the routing lists are written by the kernel just before this one in the stream
    // optional redirections (stage entry points, p92b_nvfp4_grouped_rows)
    const std::int32_t* out_row;       // null: output rows sit at their padded position; else [dense position] -> output row
    std::uint16_t* gate_out;           // MODE 2: BF16 [output row][m_total]
    std::uint16_t* up_out;
    const p92b_expert_projection* table;   // SRC 1: device table of reference-format matrices, entry expert * 3 + kind
    const CUtensorMap* table_maps;     // SRC 1: maps of the matrices of the active experts, expert * 3 + kind
    int table_kind;                    // SRC 1, MODE 1: which of an expert's three matrices
    int skip_shared;                   // 1: the shared expert's items are not computed (the caller has none)
    std::uint16_t* const* row_dest;    // slab kernel of the down product: null, or [padded position] -> destination row
};

struct Item {
    int expert;
    int entry;
    int count;
    int m_tile;
    int pp0;
    int valid;     // tokens of this tile that exist
    int dense0;    // dense (unpadded) position of the tile's first row
};

// The routing lists a block needs to turn an item number into work, copied to shared memory once per block:
// every role decodes every item, and from global memory that is a dozen dependent loads (a binary search over
// the tile prefix, then the expert's entries) - about 1.4 µs per item, which in the MMA lane is time the tensor
// pipe runs dry.  Indexed by active slot.
struct RouteTable {
    std::int32_t prefix[kExperts + 2];      // exclusive prefix of token tiles over the active list, total at [active_count]
    std::int32_t expert[kExperts + 1];
    std::int32_t count[kExperts + 1];
    std::int32_t pp_off[kExperts + 1];
    std::int32_t offset[kExperts + 1];
    std::int32_t active_count;
};

// All threads of the block, after the lists are known to be written; the caller synchronises the block afterwards.
__device__ __forceinline__ void load_route_table(const TcParams& p, RouteTable* t) {
    const int n = min(*p.route.active_count, kExperts + 1);
    for (int a = threadIdx.x; a <= n; a += blockDim.x) {
        t->prefix[a] = p.tile_prefix[a];
        if (a < n) {
            const int e = p.route.active[a];
            t->expert[a] = e;
            t->count[a] = p.route.counts[e];
            t->pp_off[a] = p.pp_off[e];
            t->offset[a] = p.route.offsets[e];
        }
    }
    if (threadIdx.x == 0) t->active_count = n;
}

template <int N>
__device__ __forceinline__ bool decode_item(const TcParams& p, const RouteTable& t, int item, Item* it) {
    const int tt = item / p.m_tiles;
    it->m_tile = item - tt * p.m_tiles;
    int lo = 0, hi = t.active_count;         // find a: prefix[a] <= tt < prefix[a+1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (t.prefix[mid] <= tt) lo = mid; else hi = mid;
    }
    const int n_tile = tt - t.prefix[lo];
    it->expert = t.expert[lo];
    it->entry = it->expert == kExperts ? p.bank.local_experts : it->expert - p.bank.first_expert;
    it->count = t.count[lo];
    it->pp0 = t.pp_off[lo] + n_tile * kTileStride<N>;
    it->valid = min(N, it->count - n_tile * N);
    it->dense0 = t.offset[lo] + n_tile * N;
    if (p.skip_shared && it->expert == kExperts) return false;
    if (p.table != nullptr) {          // weights in place: the table is indexed by the global expert id
        it->entry = it->expert;
        return it->expert >= 0 && it->expert < kExperts;
    }
    return it->entry >= 0 && it->entry <= p.bank.local_experts;
}

// Two floats rounded to BF16 (nearest even) in one conversion: the first in the low half.
__device__ __forceinline__ std::uint32_t bf16x2_bits(float low, float high) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
    return *reinterpret_cast<const std::uint32_t*>(&pair);
}

// The tensor map of a matrix of the caller's table for the product kernel's loads: the host's map of a matrix of this shape
// with the matrix's own address.  By a warp, through 128 bytes of shared memory; maps of matrices off a 16-byte boundary are
// not built (the product kernel rejects them).
__device__ __forceinline__ void build_table_map(const TableMaps& maps, int which, std::uint32_t* image) {
    const int lane = threadIdx.x & 31;
    const std::uint8_t* matrix = maps.table[which].weight;
    if ((reinterpret_cast<std::uintptr_t>(matrix) & 15U) != 0U) return;
    image[lane] = reinterpret_cast<const std::uint32_t*>(&maps.box)[lane];
    __syncwarp();
    if (lane == 0) tensormap_set_address(image, matrix);
    __syncwarp();
    tensormap_publish(maps.maps + which, image);
}

// A row that the caller has quantised in the reference's layout (packed [R][K/2], scales 128x4-tiled over the R rows), copied by
// a warp to padded position pp.
__device__ __forceinline__ void copy_quantised_row(const std::uint8_t* __restrict__ packed, const std::uint8_t* __restrict__ scales_swizzled,
                                                   std::size_t src, std::uint8_t* __restrict__ xq, std::uint8_t* __restrict__ xs,
                                                   std::size_t pp, int k_bytes) {
    const int lane = threadIdx.x & 31;
    const uint4* from = reinterpret_cast<const uint4*>(packed + src * k_bytes);
    uint4* to = reinterpret_cast<uint4*>(xq + pp * k_bytes);
    for (int v = lane; v < k_bytes / 16; v += 32) to[v] = __ldg(from + v);
    const int scale_columns = k_bytes / 8;                       // K / 16
    const int col_blocks = (scale_columns + 3) / 4;
    const std::uint8_t* sf_from = scales_swizzled + (src >> 7) * col_blocks * 512 + (src & 31) * 16 + ((src >> 5) & 3) * 4;
    std::uint8_t* sf_to = xs + (pp >> 7) * col_blocks * 512 + (pp & 31) * 16 + ((pp >> 5) & 3) * 4;
    for (int c = lane; c < scale_columns; c += 32) sf_to[(c >> 2) * 512 + (c & 3)] = sf_from[(c >> 2) * 512 + (c & 3)];
}

}  // namespace expert

// Large-batch products with the tokens on the M side (expert_rows.cu); p.tile_prefix counts 128-row tiles.
cudaError_t launch_expert_rows_gate_up(const p92b_plan* plan, const expert::TcParams& p, bool scales_by_row, cudaStream_t stream, bool pdl);
cudaError_t launch_expert_rows_matrix(const p92b_plan* plan, expert::TcParams p, cudaStream_t stream, bool pdl);
// Down product whose token rows stay in shared memory, where the K extent allows it; the one kernel that honours row_dest.
bool down_slab_shape(int hidden, int intermediate);
cudaError_t launch_expert_down_slab(const p92b_plan* plan, const expert::TcParams& p, cudaStream_t stream, bool pdl);

}  // namespace p92b
