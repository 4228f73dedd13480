// Expert products for batches of more than a few rows per expert: the TOKENS are the M side of the MMA (one token row
// per TMEM lane), the weights the N side.
//
// With the weights on the M side (expert_tc.cu, right for a few token columns) a lane of the accumulator holds one
// weight row, so the 16-element blocks of the re-quantisation run ACROSS lanes: a warp reduction, a select tree, a
// shuffle per column and a nibble transposition - about 65 instructions per SwiGLU value, which is what bounded the
// kernel at 4,096 tokens (201 µs).  With the tokens on the M side a lane holds one token's 32 neighbouring values:
// maximum, scale, packing and store need no other lane.  And one MMA covers 128 tokens x 256 weight rows (the two boxes
// of a chunk are one 256-row operand), so an operand byte in shared memory is read half as often as with
// N = 64.
#include "expert_common.cuh"

namespace p92b {

using namespace ptx;
using namespace expert;

namespace {

constexpr int kTok = 128;                                   // token rows of a tile (M)
constexpr int kWRows = 256;                                 // weight rows of a tile (N)
constexpr int kEpiWarps = 16;                               // four per TMEM quarter
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kThreadsByRow = kThreads + 32;                // and a warp that turns the token scales round

constexpr int kTmemAll = 512;

// Eight sums of one row scaled and rounded to BF16: 16 bytes.
__device__ __forceinline__ uint4 scale_to_bf16x8(const std::uint32_t* v, float alpha) {
    std::uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = bf16x2_bits(__uint_as_float(v[2 * k]) * alpha, __uint_as_float(v[2 * k + 1]) * alpha);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Stores 32 rows x 64 BF16 values; lane l holds row l's eight 16-byte pieces.  Stored as they are, one instruction
// would touch 32 lines and write 16 bytes of each (a down product over 147,456 rows took 506 µs that way against 326).
// An 8 x 8 transposition of the pieces inside every group of eight lanes - three exchange rounds - makes lane j of a
// group hold piece j of the group's eight rows: one instruction then stores four whole 128-byte lines.  `out` = the first of the
// 32 rows in the output, `valid` = rows that exist (warp uniform).
__device__ __forceinline__ void store_rows64(std::uint16_t* out, int pitch, int valid, uint4 (&w)[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) {
        const bool upper = (lane & d) != 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if ((q & d) != 0) continue;
            // the lane with bit d set keeps piece q + d and gives piece q away; the other one the reverse
            const uint4 give = upper ? w[q] : w[q + d];
            uint4 got;
            got.x = __shfl_xor_sync(0xffffffffU, give.x, d);
            got.y = __shfl_xor_sync(0xffffffffU, give.y, d);
            got.z = __shfl_xor_sync(0xffffffffU, give.z, d);
            got.w = __shfl_xor_sync(0xffffffffU, give.w, d);
            if (upper) w[q] = got; else w[q + d] = got;
        }
    }
    // now w[r] is piece (lane & 7) of row (lane & ~7) + r
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int from = (lane & ~7) + r;
        if (from < valid) *reinterpret_cast<uint4*>(out + static_cast<std::size_t>(from) * pitch + (lane & 7) * 8) = w[r];
    }
}

// 32 consecutive columns of this warp's 32 TMEM lanes.
__device__ __forceinline__ void tmem_load32(std::uint32_t addr, std::uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
}

// 64 columns of this warp's 32 rows, scaled and rounded, half of them at a time to stay within the registers.
__device__ __forceinline__ void load_scale_rows64(std::uint32_t tmem, float alpha, uint4 (&w)[8]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        std::uint32_t v[32];
        tmem_load32(tmem + h * 32, v);
        tmem_load_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) w[h * 4 + q] = scale_to_bf16x8(v + q * 8, alpha);
    }
}

// One 16-element block of a token's intermediate row from its gate and up sums: bf16(alpha * sum) for both, SwiGLU
// rounded to BF16 (cuda/nvfp4_ops.cu:97-105), block maximum, E4M3 scale, E2M1 values (cuda/nvfp4_ops.cu:818-841) -
// the arithmetic of the other gate/up epilogues value for value, all of it in one lane.
__device__ __forceinline__ uint2 swiglu_block16(const std::uint32_t* g, const std::uint32_t* u, float alpha_g, float alpha_u,
                                                float quant_scale, std::uint32_t* scale_bits) {
    std::uint32_t hh[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float h[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = 2 * k + i;
            const std::uint32_t gu = bf16x2_bits(__uint_as_float(g[j]) * alpha_g, __uint_as_float(u[j]) * alpha_u);
            const float gv = __uint_as_float(gu << 16);
            const float uv = __uint_as_float(gu & 0xffff0000U);
            h[i] = (gv / (1.0F + expf(-gv))) * uv;
        }
        hh[k] = bf16x2_bits(h[0], h[1]);
    }
    // |BF16| bit patterns order like unsigned integers: the maximum of 16 as packed 16-bit maxima
    std::uint32_t m = hh[0] & 0x7fff7fffU;
#pragma unroll
    for (int k = 1; k < 8; ++k) m = __vmaxu2(m, hh[k] & 0x7fff7fffU);
    const float amax = __uint_as_float(max(m << 16, m & 0xffff0000U));
    const __nv_fp8_e4m3 scale(amax * (quant_scale / 6.0F));
    *scale_bits = scale.__x;
    const float decoded = static_cast<float>(scale);
    const float multiplier = decoded == 0.0F ? 0.0F : quant_scale / decoded;
    std::uint32_t words[2] = {0U, 0U};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float2 pair = make_float2(__uint_as_float(hh[k] << 16) * multiplier, __uint_as_float(hh[k] & 0xffff0000U) * multiplier);
        const std::uint32_t byte = __nv_fp4x2_e2m1(pair).__x;
        words[k >> 2] |= byte << ((k & 3) * 8);
    }
    return make_uint2(words[0], words[1]);
}

// A ring stage: one K block (256 values) of the weight tile and of the token tile.  The weight part of a gate/up
// stage is exactly one chunk of the bank's stream: two boxes of mixed gate and up rows, their two scale slabs.
struct Stage {
    static constexpr int kOffW = 0;
    static constexpr int kOffSfW = kWRows * kBlockKBytes;                   // 32,768
    static constexpr int kOffT = kChunkBytes;                               // 36,864
    static constexpr int kOffSfT = kOffT + kTok * kBlockKBytes;
    static constexpr int kBytes = kOffSfT + kSfSlab;                        // 55,296
    static constexpr int kCount = 4;
    static constexpr int kBarriers = 3 * kCount + 2;
    static constexpr int kSmem = kCount * kBytes + kBarriers * 8 + 16 + 1024;
    // TMEM: the accumulator (256 columns), then two buffers of scale factors: 16 columns for the tokens, 32 for the weights
    static constexpr int kSfBase = 256, kSfBufferCols = 64, kSfWeights = 16;
};

// Items that do not fill a last round of all blocks are cut into narrower ones, of 128 or 64 weight rows, where that ends
// sooner.  What a K block costs is the bytes it brings in (60 bytes per cycle and SM), and the token rows come with
// every width, so a narrow item is dearer per result but done in less time: the down product of a dense MLP of 3,807 rows
// is 300 items on 148 SMs, two rounds and four items over; one of 64 rows is 10 items.
struct Items {
    int full;          // items of 256 weight rows, whole rounds of them
    int parts;         // pieces per item after those: 1, 2 or 4
    int total;         // full items and pieces
};
__device__ __forceinline__ Items share_out(int items, int blocks) {
    Items s;
    s.full = items / blocks * blocks;
    const int over = items - s.full;
    s.parts = 1;
    int best = over > 0 ? Stage::kBytes : 0;
#pragma unroll
    for (int parts = 2; parts <= 4; parts *= 2) {
        const int bytes = kWRows / parts * kBlockKBytes + kSfSlab + kTok * kBlockKBytes + kSfSlab;
        const int cost = (over * parts + blocks - 1) / blocks * bytes;
        if (cost < best) { best = cost; s.parts = parts; }
    }
    s.total = s.full + over * s.parts;
    return s;
}
struct Piece {
    Item it;
    int width;         // weight rows: 256, 128 or 64
    int first;         // the first of them within the item's 256
};
__device__ __forceinline__ bool decode_piece(const TcParams& p, const RouteTable& t, const Items& items, int index, Piece* piece) {
    const int parts = index < items.full ? 1 : items.parts;
    const int past = index - items.full;
    const int item = parts == 1 ? index : items.full + past / parts;
    piece->width = kWRows / parts;
    piece->first = parts == 1 ? 0 : past % parts * piece->width;
    return decode_item<kTok>(p, t, item, &piece->it);
}

// MODE 0: gate/up + SwiGLU + re-quantisation; p.m_tiles row tiles of 128 intermediate rows (gate and up rows of each).
// MODE 1: one matrix, BF16 rows out; p.m_tiles pairs of the bank's 128-row tiles.
// Roles as in expert_tc.cu: producer warp, MMA warp, sixteen epilogue warps; items (128-row token tile, weight tile).
// One accumulator only - two of 256 columns and the scale factors do not fit TMEM - so the epilogue warps take their
// 64 columns into registers at once and the next item's products start after that read, not after the arithmetic.
// What bounds it with full tiles: a K block brings 54 KB into the SM, 864 cycles at 64 bytes, against 776 of the tensor pipe (512
// of products, twelve scale copies of 22); it runs at about 910, and the four stages leave some 4 % more latency no room
// (16,384 tokens: 563 -> 394 us; 4,096 tokens: 201 -> 163 us, HBM floor 116).  A pair of blocks sharing the weight rows
// (cta_group::2, 256-row token tiles) pads every expert to 256 rows and took in 25 bytes per cycle and SM: dense MLP of 3,807
// rows 230 us against 132, not kept.  Token rows gathered from token order (TMA tile::gather4, four rows per operation) take
// 46 ns per operation: 1,023 us.
// BY_ROW: the scales of a stage's 128 token rows come as 16 bytes per row, four K steps of four blocks, and the tensor core's copy
// wants them as four slabs of [row % 32][row / 32][4 bytes].  One more warp turns them round where they lie: a lane has the 16 bytes
// of rows l, l + 32, l + 64 and l + 96 and gives four words to each slab, four 16-byte loads and stores per K block of some 900
// cycles, so that the kernels in front store a row's scales in 16-byte pieces.  The scales are requested ahead of the stage's other
// bytes, on a barrier of their own, and are turned round before those have come: turned when all was there this kernel took 427 us
// at 16,384 rows, with three barriers for the MMA lane to wait on 410, with one 400, as without the turning.
// (One barrier per stage, not one for the weights and one for the tokens: dense MLP of two layers, 33 rows 56.2 -> 55.7 us, 129
// 59.6 -> 59.1, 512 70.5 -> 69.9, 1,400 133.7 -> 134.1 at a spread of 2 %, 2,000 184.2 -> 182.1, 3,807 312.2 -> 309.5.)
template <int MODE, bool BY_ROW>
__global__ void __launch_bounds__(BY_ROW ? kThreadsByRow : kThreads, 1) expert_rows_kernel(const __grid_constant__ CUtensorMap map_t32,
                                                                                            const __grid_constant__ CUtensorMap map_t128,
                                                                                            const TcParams p) {
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ RouteTable route_table;
    const std::uint32_t base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    const std::uint32_t bars = base + Stage::kCount * Stage::kBytes;
    auto full_bar = [&](int s) { return bars + 8U * s; };                              // BY_ROW: and the token scales turned round
    auto empty_bar = [&](int s) { return bars + 8U * (Stage::kCount + s); };
    auto scale_bar = [&](int s) { return bars + 8U * (2 * Stage::kCount + s); };       // BY_ROW: token scales there, as they come
    const std::uint32_t accum_full = bars + 8U * (3 * Stage::kCount);
    const std::uint32_t accum_empty = accum_full + 8U;
    const std::uint32_t tmem_slot = bars + 8U * Stage::kBarriers;
    volatile std::uint32_t* tmem_slot_ptr =
        reinterpret_cast<volatile std::uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
    volatile std::uint32_t* abort_ptr = tmem_slot_ptr + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int k_blocks = p.k_bytes / kBlockKBytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < Stage::kCount; ++s) {
            mbar_init(full_bar(s), BY_ROW ? 2 : 1);
            mbar_init(empty_bar(s), 1);
            mbar_init(scale_bar(s), 1);
        }
        mbar_init(accum_full, 1);
        mbar_init(accum_empty, kEpiWarps);
        *abort_ptr = 0;
        fence_mbar_init();
        prefetch_tensormap(&map_t32);
        prefetch_tensormap(&map_t128);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemAll);
        tmem_relinquish();
    }
    pdl_wait();                       // routing lists and token rows come from the kernels upstream
    load_route_table(p, &route_table);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const std::uint32_t tmem_base = *tmem_slot_ptr;
    const Items items = share_out(route_table.prefix[route_table.active_count] * p.m_tiles, gridDim.x);    // the prefix counts 128-row slabs here
    const int total_items = items.total;
    auto give_up = [&]() {
        *abort_ptr = 1;
        atomicCAS(p.status, kStatusOk, kStatusWaitExpired);
    };

    if (warp == 0) {
        if (elect_one()) {
            const std::uint64_t stream_policy = l2_policy_evict_first();
            int stage = 0;
            std::uint32_t phase = 0;
            for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
                Piece piece;
                if (!decode_piece(p, route_table, items, item, &piece)) continue;
                const Item& it = piece.it;
                // The entry's only tile: nobody else reads these weights, and they are the first to leave the L2 again.  The rest
                // stays there for the kernels behind (64 rows, four layers: 743 -> 730 us, 512 rows 462 -> 457.5, 2,048 rows 269 ->
                // 262.5).  For every entry, the second tile's reads go to memory: 4,096 rows, down product 101 -> 121 us.  Whole
                // items of the gate/up product only: the pieces of the last round and MODE 1 load without it.
                const bool once = it.count <= kTok;
                const int half = piece.first / kTileM;          // narrow pieces: which of the two boxes
                // token rows beyond the tile's last one are not loaded: their lanes compute on what the stage held
                // before, and nothing reads them
                const int boxes = (it.valid + 31) >> 5;
                const std::uint8_t* t_sf = p.b_sf + static_cast<std::size_t>(it.pp0 >> 7) * (p.k_bytes / 32) * 512;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1U)) { give_up(); break; }
                    const std::uint32_t st = base + stage * Stage::kBytes;
                    if constexpr (BY_ROW) {                 // ahead of the rest: turned round by the time that has come
                        mbar_arrive_expect_tx(scale_bar(stage), kSfSlab);
                        bulk_load(st + Stage::kOffSfT, t_sf + static_cast<std::size_t>(kb) * 4 * 512, kSfSlab, scale_bar(stage));
                    }
                    const std::uint32_t weight_bytes = piece.width == kWRows ? kChunkBytes : static_cast<std::uint32_t>(piece.width) * kBlockKBytes + kSfSlab;
                    mbar_arrive_expect_tx(full_bar(stage), weight_bytes + boxes * (32 * kBlockKBytes) + (BY_ROW ? 0 : kSfSlab));
                    if (piece.width == kWRows) {
                        if constexpr (MODE == 0) {
                            const std::uint8_t* from =
                                p.bank.g13 + ((static_cast<std::size_t>(it.entry) * p.m_tiles + it.m_tile) * k_blocks + kb) * kChunkBytes;
                            if (once) {
                                bulk_load_hint(st + Stage::kOffW, from, kChunkBytes, full_bar(stage), stream_policy);
                            } else {
                                bulk_load(st + Stage::kOffW, from, kChunkBytes, full_bar(stage));
                            }
                        } else {
                            // K block kb of two neighbouring row tiles: a box and a scale slab from either tile's chunk
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const std::uint8_t* chunk = p.bank.g2 +
                                    ((static_cast<std::size_t>(it.entry) * p.m_tiles * 2 + it.m_tile * 2 + h) * (k_blocks / 2) + (kb >> 1)) * kChunkBytes;
                                bulk_load(st + Stage::kOffW + h * kChunkBox, chunk + (kb & 1) * kChunkBox, kChunkBox, full_bar(stage));
                                bulk_load(st + Stage::kOffSfW + h * kSfSlab, chunk + kChunkScaleOffset + (kb & 1) * kChunkScaleBytes, kSfSlab,
                                          full_bar(stage));
                            }
                        }
                    } else {
                        const int box = MODE == 0 ? half : kb & 1;
                        const std::uint8_t* chunk = MODE == 0
                            ? p.bank.g13 + ((static_cast<std::size_t>(it.entry) * p.m_tiles + it.m_tile) * k_blocks + kb) * kChunkBytes
                            : p.bank.g2 + ((static_cast<std::size_t>(it.entry) * p.m_tiles * 2 + it.m_tile * 2 + half) * (k_blocks / 2) + (kb >> 1)) * kChunkBytes;
                        bulk_load(st + Stage::kOffW, chunk + box * kChunkBox + piece.first % kTileM * kBlockKBytes, weight_bytes - kSfSlab,
                                  full_bar(stage));
                        bulk_load(st + Stage::kOffSfW, chunk + kChunkScaleOffset + box * kChunkScaleBytes, kSfSlab, full_bar(stage));
                    }
                    if (boxes == 4) {
                        tma_load_2d(st + Stage::kOffT, &map_t128, full_bar(stage), kb * kBlockKBytes, it.pp0);
                    } else {
                        for (int b = 0; b < boxes; ++b) {
                            tma_load_2d(st + Stage::kOffT + b * 32 * kBlockKBytes, &map_t32, full_bar(stage), kb * kBlockKBytes, it.pp0 + b * 32);
                        }
                    }
                    if constexpr (!BY_ROW) {
                        bulk_load(st + Stage::kOffSfT, t_sf + static_cast<std::size_t>(kb) * 4 * 512, kSfSlab, full_bar(stage));
                    }
                    if (++stage == Stage::kCount) { stage = 0; phase ^= 1U; }
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0;
            std::uint32_t accum_phase = 0;
            int sf_buffer = 0;
            for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
                Piece piece;
                if (!decode_piece(p, route_table, items, item, &piece)) continue;
                const std::uint32_t idesc = idesc_nvf4(kTok, piece.width);
                // 64 rows from the middle of a box: their scale factors sit two TMEM columns further
                const std::uint32_t quarter = static_cast<std::uint32_t>(piece.first % kTileM) >> 5;
                bool ok = true;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(full_bar(stage), phase)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    if (kb == 0 && !mbar_wait(accum_empty, accum_phase ^ 1U)) { give_up(); ok = false; break; }
                    tc_fence_after();
                    const std::uint32_t st = base + stage * Stage::kBytes;
                    const std::uint32_t sf_t = tmem_base + Stage::kSfBase + sf_buffer * Stage::kSfBufferCols;
                    const std::uint32_t sf_w = sf_t + Stage::kSfWeights;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        tc_copy_sf(sf_t + k * 4, desc_scale_atom(st + Stage::kOffSfT + k * 512));
                        // a 256-row operand takes eight columns per K step: its rows 0..127, then 128..255
                        tc_copy_sf(sf_w + k * 8, desc_scale_atom(st + Stage::kOffSfW + k * 512));
                        if (piece.width == kWRows) tc_copy_sf(sf_w + k * 8 + 4, desc_scale_atom(st + Stage::kOffSfW + kSfSlab + k * 512));
                    }
                    const std::uint64_t a_desc = desc_k_major_sw128(st + Stage::kOffT);
                    const std::uint64_t b_desc = desc_k_major_sw128(st + Stage::kOffW);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mma_nvf4(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, sf_t + k * 4, sf_w + k * 8 + quarter, kb > 0 || k > 0);
                    }
                    tc_commit(empty_bar(stage));
                    sf_buffer ^= 1;
                    if (++stage == Stage::kCount) { stage = 0; phase ^= 1U; }
                }
                if (!ok) break;
                tc_commit(accum_full);
                accum_phase ^= 1U;
            }
        }
    } else if (BY_ROW && warp == kThreads / 32) {
        int stage = 0;
        std::uint32_t phase = 0;
        for (int item = blockIdx.x; item < total_items && !__any_sync(0xffffffffU, *abort_ptr != 0); item += gridDim.x) {
            Piece piece;
            if (!decode_piece(p, route_table, items, item, &piece)) continue;
            bool ok = true;
            for (int kb = 0; kb < k_blocks; ++kb) {
                ok = __all_sync(0xffffffffU, mbar_wait(scale_bar(stage), phase));
                if (!ok) break;
                uint4* at = reinterpret_cast<uint4*>(smem_raw + (base - smem_u32(smem_raw)) + stage * Stage::kBytes + Stage::kOffSfT) + lane;
                const uint4 a = at[0], b = at[32], c = at[64], d = at[96];
                at[0] = make_uint4(a.x, b.x, c.x, d.x);
                at[32] = make_uint4(a.y, b.y, c.y, d.y);
                at[64] = make_uint4(a.z, b.z, c.z, d.z);
                at[96] = make_uint4(a.w, b.w, c.w, d.w);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(stage));
                if (++stage == Stage::kCount) { stage = 0; phase ^= 1U; }
            }
            if (!ok) {
                give_up();
                break;
            }
        }
    } else {
        const int quarter = warp & 3;
        const int group = (warp - 2) >> 2;                  // which 32 intermediate rows (MODE 0) or 64 output columns (MODE 1)
        const std::uint32_t lane_base = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16);
        const int row = quarter * 32 + lane;                // token row of the tile
        std::uint32_t accum_phase = 0;
        for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
            Piece piece;
            if (!decode_piece(p, route_table, items, item, &piece)) continue;
            const Item& it = piece.it;
            if (!mbar_wait(accum_full, accum_phase)) { give_up(); break; }
            accum_phase ^= 1U;
            tc_fence_after();
            const bool mine = quarter * 32 < it.valid && group * 64 < piece.width;      // warp uniform
            const int column64 = piece.first + group * 64;  // of the item's 256 weight rows
            if constexpr (MODE == 0) {
                const int pp = it.pp0 + row;
                std::uint32_t first[32], second[32];
                if (mine) {
                    tmem_load32(lane_base + group * 64, first);            // gate and up sums of 16 intermediate rows
                    tmem_load32(lane_base + group * 64 + 32, second);       // ... and of the next 16
                    tmem_load_wait();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(accum_empty);
                if (mine && row < it.valid) {
                    const float alpha_g = p.bank.alpha[it.entry * 3 + 0];
                    const float alpha_u = p.bank.alpha[it.entry * 3 + 1];
                    const int inter = p.m_total;
                    std::uint32_t scale0, scale1;
                    const uint2 q0 = swiglu_block16(first, first + 16, alpha_g, alpha_u, p.quant_scale, &scale0);
                    const uint2 q1 = swiglu_block16(second, second + 16, alpha_g, alpha_u, p.quant_scale, &scale1);
                    const int column = it.m_tile * kTileM + column64 / 2;
                    *reinterpret_cast<uint4*>(p.hq + static_cast<std::size_t>(pp) * (inter / 2) + (column >> 1)) = make_uint4(q0.x, q0.y, q1.x, q1.y);
                    const int sf_col = column >> 4;         // even: the two bytes are neighbours in the tiled layout
                    std::uint8_t* sf = p.hs + (static_cast<std::size_t>(pp >> 7) * (inter / 64) + (sf_col >> 2)) * 512 + (pp & 31) * 16 +
                                       ((pp >> 5) & 3) * 4 + (sf_col & 3);
                    *reinterpret_cast<std::uint16_t*>(sf) = static_cast<std::uint16_t>(scale0 | (scale1 << 8));
                }
                __syncwarp();                               // the next accumulator read is warp wide
            } else {
                const float alpha = p.bank.alpha[it.entry * 3 + 2];
                uint4 w[8];
                if (mine) load_scale_rows64(lane_base + group * 64, alpha, w);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(accum_empty);
                if (!mine) continue;
                std::uint16_t* first_row = p.out + static_cast<std::size_t>(it.pp0 + quarter * 32) * p.m_total;
                store_rows64(first_row + static_cast<std::size_t>(it.m_tile) * kWRows + column64, p.m_total, it.valid - quarter * 32, w);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemAll);
    }
}

// ---- down product whose token rows stay in shared memory ----------------------------------------------------
// For a K extent of up to 1,024 a 128-token slab with all its K blocks (64 KB) and scale slabs (8 KB) is loaded ONCE per item and
// only the weights stream past it, chunk by chunk of the bank; the slab's scale factors stay in TMEM.  An item is a slab and
// all of the 128-row tiles of the weight, or half of them.
// A tile is 1,024 cycles of products and 32 KB of results, so what happens between the accumulator and memory decides.  Two
// teams of eight warps have an accumulator each and take the tiles in turn: a team has two tiles' time, and while one of them
// stores the other reads; the weights of the first four chunks are requested before the wait for the gate/up kernel.  With the
// weights on the M side and the results turned round through shared memory (the form before): 281 us at 16,384 tokens, even
// routing, now 262 (1.2 GB, of which 755 MB are written); 4,096 skewed 119, now 110; 512 72, now 69.  One team of sixteen warps on one
// accumulator of 256 columns took 283.
struct Slab {
    static constexpr int kKBlocksMax = 4;
    static constexpr int kChunksMax = kKBlocksMax / 2;
    static constexpr int kOffSf = kKBlocksMax * kTok * kBlockKBytes;                // scale slabs behind the boxes
    static constexpr int kBytes = kOffSf + kKBlocksMax * kSfSlab;                   // 73,728
    static constexpr int kStages = 4;                                               // of one chunk: 128 weight rows, two K blocks
    static constexpr int kTeams = 2;
    static constexpr int kTeamWarps = kEpiWarps / kTeams;
    static constexpr int kBarriers = 2 * kStages + kChunksMax + 2 * kTeams;
    static constexpr int kSmem = kBytes + kStages * kChunkBytes + kBarriers * 8 + 16 + 1024;
    // TMEM: two accumulators, the slab's scale factors (16 columns per K block), two buffers of a chunk's (32)
    static constexpr int kSfT = kTeams * kTileM, kSfW = kSfT + kKBlocksMax * 16;
    // Whole slabs once there are enough of them to share out evenly; with three slabs per SM halves balance better.
    static constexpr int kMaxGroups = 2;
    static constexpr int kWholeSlabsPerSm = 6;
};

// Items past the last whole round of blocks are cut into parts where that ends sooner, by the bytes of a part's tiles and of the
// slab that every part loads: four items left over (64 rows) took as long as another 148.  64 rows 66.7 -> 62 us, 4,096 skewed
// 110 -> 106.
struct SlabItems {
    int groups;        // items per slab
    int full;          // items of whole rounds
    int parts;         // pieces per item after those
    int total;         // full items and pieces
};
__device__ __forceinline__ SlabItems share_out_slabs(int slabs, int blocks, int m_tiles, int chunks) {
    SlabItems s;
    s.groups = slabs >= Slab::kWholeSlabsPerSm * blocks ? 1 : Slab::kMaxGroups;
    const int items = slabs * s.groups, tiles = m_tiles / s.groups;
    s.full = items / blocks * blocks;
    const int over = items - s.full;
    s.parts = 1;
    int best = 0x7fffffff;
    for (int parts = 1; parts <= tiles; ++parts) {
        const int cost = (over * parts + blocks - 1) / blocks * ((tiles + parts - 1) / parts * chunks * kChunkBytes + Slab::kBytes);
        if (cost < best) { best = cost; s.parts = parts; }
    }
    s.total = s.full + over * s.parts;
    return s;
}

// 32 bytes of a row in two 16-byte halves.
struct Piece32 {
    uint4 lo, hi;
};
__device__ __forceinline__ void store_piece32(void* to, const Piece32& v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "r"(v.lo.x), "r"(v.lo.y), "r"(v.lo.z),
                 "r"(v.lo.w), "r"(v.hi.x), "r"(v.hi.y), "r"(v.hi.z), "r"(v.hi.w) : "memory");
}
__device__ __forceinline__ uint4 shfl_xor4(uint4 v, int d) {
    return make_uint4(__shfl_xor_sync(0xffffffffU, v.x, d), __shfl_xor_sync(0xffffffffU, v.y, d), __shfl_xor_sync(0xffffffffU, v.z, d),
                      __shfl_xor_sync(0xffffffffU, v.w, d));
}
// Lane l holds row l's 64 values as four pieces of 32 bytes; afterwards piece (lane & 3) of rows (lane & ~3) + 0 .. 3: four lanes
// then store a whole 128-byte line, eight lines per instruction.
__device__ __forceinline__ void exchange_rows64(Piece32 (&w)[4]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 2; d >= 1; d >>= 1) {
        const bool upper = (lane & d) != 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if ((q & d) != 0) continue;
            const Piece32 give = upper ? w[q] : w[q + d];
            const Piece32 got = {shfl_xor4(give.lo, d), shfl_xor4(give.hi, d)};
            if (upper) w[q] = got; else w[q + d] = got;
        }
    }
}

__global__ void __launch_bounds__(kThreads, 1) expert_down_slab_kernel(const __grid_constant__ CUtensorMap map_t32,
                                                                       const __grid_constant__ CUtensorMap map_t128, const TcParams p) {
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ RouteTable route_table;
    const std::uint32_t base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    const std::uint32_t ring = base + Slab::kBytes;
    const std::uint32_t bars = ring + Slab::kStages * kChunkBytes;
    auto full_bar = [&](int s) { return bars + 8U * s; };
    auto empty_bar = [&](int s) { return bars + 8U * (Slab::kStages + s); };
    auto slab_empty = [&](int c) { return bars + 8U * (2 * Slab::kStages + c); };
    auto accum_full = [&](int t) { return bars + 8U * (2 * Slab::kStages + Slab::kChunksMax + t); };
    auto accum_empty = [&](int t) { return bars + 8U * (2 * Slab::kStages + Slab::kChunksMax + Slab::kTeams + t); };
    const std::uint32_t tmem_slot = bars + 8U * Slab::kBarriers;
    volatile std::uint32_t* tmem_slot_ptr =
        reinterpret_cast<volatile std::uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
    volatile std::uint32_t* abort_ptr = tmem_slot_ptr + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int chunks = p.k_bytes / kBlockKBytes / 2;            // <= 2

    if (threadIdx.x == 0) {
        for (int s = 0; s < Slab::kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int c = 0; c < Slab::kChunksMax; ++c) mbar_init(slab_empty(c), 1);
        for (int t = 0; t < Slab::kTeams; ++t) {
            mbar_init(accum_full(t), 1);
            mbar_init(accum_empty(t), Slab::kTeamWarps);
        }
        *abort_ptr = 0;
        fence_mbar_init();
        prefetch_tensormap(&map_t32);
        prefetch_tensormap(&map_t128);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemAll);
        tmem_relinquish();
    }
    // The SwiGLU rows come from the kernel just upstream, the routing lists from one further up.  Only the producer lane waits, and
    // not before the ring is full of weights: as the blocks of the gate/up kernel leave, the memory already works for this one.
    if (p.routing_is_upstream) pdl_wait();
    load_route_table(p, &route_table);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const std::uint32_t tmem_base = *tmem_slot_ptr;
    const int slabs = route_table.prefix[route_table.active_count];                 // the prefix counts 128-row slabs here
    const SlabItems items = share_out_slabs(slabs, gridDim.x, p.m_tiles, chunks);
    const int total_items = items.total;
    auto give_up = [&]() {
        *abort_ptr = 1;
        atomicCAS(p.status, kStatusOk, kStatusWaitExpired);
    };
    // item -> slab and the tiles [it->m_tile, *last) of the weight
    auto decode = [&](int index, Item* it, int* last) {
        const int parts = index < items.full ? 1 : items.parts;
        const int past = index - items.full;
        const int item = parts == 1 ? index : items.full + past / parts;
        const int part = parts == 1 ? 0 : past % parts;
        const int slab = item / items.groups;
        const int tiles = p.m_tiles / items.groups;
        const bool ok = decode_item<kTok>(p, route_table, slab * p.m_tiles, it);
        it->m_tile = (item - slab * items.groups) * tiles + tiles * part / parts;
        *last = (item - slab * items.groups) * tiles + tiles * (part + 1) / parts;
        return ok;
    };

    if (warp == 0) {
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0, slab_phase = 0;
            bool ok = true, upstream_done = p.routing_is_upstream != 0;
            const std::uint64_t stream_policy = l2_policy_evict_first();
            int requested = 0;                              // chunks of the first item whose weights were asked for before the wait
            for (int item = blockIdx.x; item < total_items && !*abort_ptr && ok; item += gridDim.x) {
                Item it;
                int last;
                if (!decode(item, &it, &last)) continue;
                const int boxes = (it.valid + 31) >> 5;         // rows beyond the slab's last one are not loaded
                const std::uint8_t* t_sf = p.b_sf + static_cast<std::size_t>(it.pp0 >> 7) * (p.k_bytes / 32) * 512;
                const std::uint32_t slab_bytes = 2 * (boxes * (32 * kBlockKBytes) + kSfSlab);
                const std::uint8_t* weights = p.bank.g2 + (static_cast<std::size_t>(it.entry) * p.m_tiles + it.m_tile) * chunks * kChunkBytes;
                const bool once = it.count <= kTok;             // its only slab: nobody else reads these weights (expert_rows_kernel)
                auto request = [&](int s, int n) {          // chunk n of the item into stage s
                    mbar_arrive_expect_tx(full_bar(s), kChunkBytes + (n < chunks ? slab_bytes : 0U));
                    const std::uint8_t* from = weights + static_cast<std::size_t>(n) * kChunkBytes;
                    if (once) {
                        bulk_load_hint(ring + s * kChunkBytes, from, kChunkBytes, full_bar(s), stream_policy);
                    } else {
                        bulk_load(ring + s * kChunkBytes, from, kChunkBytes, full_bar(s));
                    }
                };
                if (!upstream_done) {
                    requested = min(Slab::kStages, (last - it.m_tile) * chunks);
                    for (int n = 0; n < requested; ++n) request(n, n);
                    pdl_wait();
                    upstream_done = true;
                }
                const int total = (last - it.m_tile) * chunks;
                for (int n = 0; n < total; ++n) {
                    if (n >= requested) {
                        if (!mbar_wait(empty_bar(stage), phase ^ 1U)) { give_up(); ok = false; break; }
                        request(stage, n);
                    }
                    if (n < chunks) {
                        // two K blocks of the slab follow as soon as the last products on the one before have read their place
                        if (!mbar_wait(slab_empty(n), slab_phase ^ 1U)) { give_up(); ok = false; break; }
#pragma unroll
                        for (int o = 0; o < 2; ++o) {
                            const int kb = 2 * n + o;
                            const std::uint32_t to = base + kb * kTok * kBlockKBytes;
                            if (boxes == 4) {
                                tma_load_2d(to, &map_t128, full_bar(stage), kb * kBlockKBytes, it.pp0);
                            } else {
                                for (int b = 0; b < boxes; ++b) {
                                    tma_load_2d(to + b * 32 * kBlockKBytes, &map_t32, full_bar(stage), kb * kBlockKBytes, it.pp0 + b * 32);
                                }
                            }
                            bulk_load(base + Slab::kOffSf + kb * kSfSlab, t_sf + static_cast<std::size_t>(kb) * 4 * 512, kSfSlab, full_bar(stage));
                        }
                    }
                    if (++stage == Slab::kStages) { stage = 0; phase ^= 1U; }
                }
                requested = 0;
                slab_phase ^= 1U;
            }
            if (!upstream_done) pdl_wait();                 // no work at all: still order this grid after its predecessor
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int stage = 0, turn = 0;                            // tiles so far
            std::uint32_t phase = 0;
            int sf_buffer = 0;
            bool ok = true;
            constexpr std::uint32_t idesc = idesc_nvf4(kTok, kTileM);
            for (int item = blockIdx.x; item < total_items && !*abort_ptr && ok; item += gridDim.x) {
                Item it;
                int last;
                if (!decode(item, &it, &last)) continue;
                for (int tile = it.m_tile; tile < last && ok; ++tile, ++turn) {
                    const int team = turn & 1;
                    const std::uint32_t accum = tmem_base + team * kTileM;
                    for (int c = 0; c < chunks; ++c) {
                        if (!mbar_wait(full_bar(stage), phase)) { give_up(); ok = false; break; }
                        if (c == 0 && !mbar_wait(accum_empty(team), ((turn >> 1) & 1U) ^ 1U)) { give_up(); ok = false; break; }
                        tc_fence_after();
                        const std::uint32_t st = ring + stage * kChunkBytes;
                        const std::uint32_t sf_w = tmem_base + Slab::kSfW + sf_buffer * 32;
#pragma unroll
                        for (int o = 0; o < 2; ++o) {
                            const int kb = 2 * c + o;
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if (tile == it.m_tile) tc_copy_sf(tmem_base + Slab::kSfT + kb * 16 + k * 4, desc_scale_atom(base + Slab::kOffSf + kb * kSfSlab + k * 512));
                                tc_copy_sf(sf_w + o * 16 + k * 4, desc_scale_atom(st + kChunkScaleOffset + o * kChunkScaleBytes + k * 512));
                            }
                        }
#pragma unroll
                        for (int o = 0; o < 2; ++o) {
                            const int kb = 2 * c + o;
                            const std::uint64_t a_desc = desc_k_major_sw128(base + kb * kTok * kBlockKBytes);
                            const std::uint64_t b_desc = desc_k_major_sw128(st + o * kChunkBox);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                mma_nvf4(accum, a_desc + 2 * k, b_desc + 2 * k, idesc, tmem_base + Slab::kSfT + kb * 16 + k * 4, sf_w + o * 16 + k * 4,
                                         kb > 0 || k > 0);
                            }
                        }
                        tc_commit(empty_bar(stage));
                        if (tile == last - 1) tc_commit(slab_empty(c));
                        sf_buffer ^= 1;
                        if (++stage == Slab::kStages) { stage = 0; phase ^= 1U; }
                    }
                    if (!ok) break;
                    tc_commit(accum_full(team));
                }
            }
        }
    } else {
        const int quarter = warp & 3;
        const int team = (warp - 2) / Slab::kTeamWarps;
        const int half = ((warp - 2) >> 2) & 1;             // which 64 of the tile's 128 output columns
        const std::uint32_t accum = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16) + team * kTileM + half * 64;
        int turn = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < total_items && !*abort_ptr && ok; item += gridDim.x) {
            Item it;
            int last;
            if (!decode(item, &it, &last)) continue;
            const float alpha = p.bank.alpha[it.entry * 3 + 2];
            const int valid = it.valid - quarter * 32;      // rows of this warp; warp uniform
            // where the four rows that this lane stores parts of go: their places in the padded position space or, with a
            // table, anywhere
            std::uint16_t* rows4[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int from = (lane & ~3) + r;
                const int pp = it.pp0 + quarter * 32 + from;
                rows4[r] = p.row_dest == nullptr ? p.out + static_cast<std::size_t>(pp) * p.m_total : from < valid ? p.row_dest[pp] : p.out;
                rows4[r] += half * 64 + (lane & 3) * 16;
            }
            for (int tile = it.m_tile; tile < last; ++tile, ++turn) {
                if ((turn & 1) != team) continue;
                if (!mbar_wait(accum_full(team), (turn >> 1) & 1U)) { give_up(); ok = false; break; }
                tc_fence_after();
                Piece32 w[4];
                if (valid > 0) {
                    std::uint32_t v[32];
                    tmem_load32(accum, v);
                    tmem_load_wait();
#pragma unroll
                    for (int q = 0; q < 2; ++q) w[q] = {scale_to_bf16x8(v + q * 16, alpha), scale_to_bf16x8(v + q * 16 + 8, alpha)};
                    tmem_load32(accum + 32, v);
                    tmem_load_wait();
#pragma unroll
                    for (int q = 0; q < 2; ++q) w[2 + q] = {scale_to_bf16x8(v + q * 16, alpha), scale_to_bf16x8(v + q * 16 + 8, alpha)};
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(accum_empty(team));
                if (valid <= 0) continue;
                exchange_rows64(w);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if ((lane & ~3) + r < valid) store_piece32(rows4[r] + tile * kTileM, w[r]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemAll);
    }
}

}  // namespace

bool down_slab_shape(int hidden, int intermediate) {
    const int k_blocks = intermediate / 2 / kBlockKBytes;
    return k_blocks <= Slab::kKBlocksMax && k_blocks % 2 == 0 && hidden % (Slab::kMaxGroups * kTileM) == 0;
}

cudaError_t launch_expert_down_slab(const p92b_plan* plan, const TcParams& p, cudaStream_t stream, bool pdl) {
    if (cudaError_t st = ensure_dynamic_smem<expert_down_slab_kernel>(Slab::kSmem); st != cudaSuccess) return st;
    return launch_kernel(expert_down_slab_kernel, dim3(plan->sm_count), dim3(kThreads), Slab::kSmem, stream, pdl, plan->map_h[1],
                         plan->map_h[3], p);
}

cudaError_t launch_expert_rows_gate_up(const p92b_plan* plan, const TcParams& p, bool scales_by_row, cudaStream_t stream, bool pdl) {
    if (scales_by_row) {
        if (cudaError_t st = ensure_dynamic_smem<expert_rows_kernel<0, true>>(Stage::kSmem); st != cudaSuccess) return st;
        return launch_kernel(expert_rows_kernel<0, true>, dim3(plan->sm_count), dim3(kThreadsByRow), Stage::kSmem, stream, pdl,
                             plan->map_x[1], plan->map_x[3], p);
    }
    if (cudaError_t st = ensure_dynamic_smem<expert_rows_kernel<0, false>>(Stage::kSmem); st != cudaSuccess) return st;
    return launch_kernel(expert_rows_kernel<0, false>, dim3(plan->sm_count), dim3(kThreads), Stage::kSmem, stream, pdl, plan->map_x[1],
                         plan->map_x[3], p);
}

cudaError_t launch_expert_rows_matrix(const p92b_plan* plan, TcParams p, cudaStream_t stream, bool pdl) {
    p.m_tiles = p.m_total / kWRows;
    if (cudaError_t st = ensure_dynamic_smem<expert_rows_kernel<1, false>>(Stage::kSmem); st != cudaSuccess) return st;
    return launch_kernel(expert_rows_kernel<1, false>, dim3(plan->sm_count), dim3(kThreads), Stage::kSmem, stream, pdl, plan->map_h[1],
                         plan->map_h[3], p);
}

}  // namespace p92b
