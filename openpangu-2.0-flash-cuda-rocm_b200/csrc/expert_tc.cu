// Tensor-core expert kernels: tcgen05 block-scaled MMA (E2M1 x E2M1, one UE4M3
// scale per 16 elements along K) with TMA-staged operands and TMEM accumulators.
//
// Orientation.  The expert weight is the M side of the MMA (128 weight rows per
// tile fill the 128 TMEM lanes), the tokens routed to the expert are the N side
// (N = 16...128 columns).  With one or two tokens per expert (decode) the kernel
// is a pure weight streamer - TMA pulls 128 x 128-byte weight boxes through a
// shared-memory ring and the tensor core consumes them at a small N - and with
// hundreds of tokens per expert (prefill) the same code is a grouped GEMM.
//
// One block = 18 warps, persistent over work items (expert, token tile, 128-row tile):
//   warp 0  producer: one elected lane issues the copies of a K block (256 elements = 128 bytes per row): the
//           weight side is one untiled bulk copy of a contiguous chunk of the bank's tile stream (boxes already in
//           the swizzled shared-memory image, scale slabs behind them), the token side a tiled box load plus its
//           2 KB scale slab; weights and tokens complete on separate mbarriers.  When the weights are read in place
//           from a caller's table of reference-format matrices (SRC 1) the box is a tiled load as well;
//   warp 1  MMA issuer: owns TMEM; per K block copies the scale slabs SMEM->TMEM (tcgen05.cp) and issues 4 MMAs of
//           K=64 per weight operand; commits the stage back to the producer and, after the last K block, the
//           accumulator to the epilogue;
//   warps 2-17  epilogue, four per TMEM quarter: each reads 16-column chunks of its 32 lanes of the accumulator
//           (tcgen05.ld), applies the per-tensor scale, rounds to BF16 where the reference does, and either fuses
//           SwiGLU + re-quantisation to NVFP4 (MODE 0), stores the BF16 down rows (MODE 1) or stores BF16 gate and
//           up rows un-fused (MODE 2, the reference's project_expert_gate_up result).
// Every role turns an item number into work from a copy of the routing lists in shared memory (RouteTable), and an
// epilogue warp hands its accumulator buffer back as soon as it has read its columns into registers.
// The products of more than 32 rows, with the tokens on the M side, are in expert_rows.cu.
// Scale factors stay in the 128x4-tiled layout the reference keeps them in
// (cuda/nvfp4_ops.cu:869-890): one 512-byte tile is exactly one tcgen05.cp atom.
//
// Every mbarrier wait is bounded; on expiry the block records kStatusWaitExpired,
// stops issuing work, frees its TMEM and returns.
#include "expert_common.cuh"

#include <algorithm>
#include <cstdlib>

namespace p92b {

using namespace ptx;
using namespace expert;

namespace {

constexpr int kEpilogueWarps = 16;                // four per TMEM quarter: they split the 16-column chunks
constexpr int kThreadsTc = 64 + 32 * kEpilogueWarps;

template <int MODE, int N>
struct Tc {
    static constexpr int kA = MODE == 1 ? 1 : 2;          // gate and up share a token tile (MODE 0 fused, MODE 2 un-fused)
    static constexpr int kABytes = kTileM * kBlockKBytes;
    static constexpr int kBBytes = N * kBlockKBytes;
    static constexpr int kWeightBytes = kA * (kABytes + kSfSlab);          // per stage, independent of the tokens
    // stage image: weight boxes | their scale slabs | token box | token scale slab; for the gate/up
    // kernel the first kWeightBytes are exactly one chunk of the bank's tile stream
    static constexpr int kOffSfA = kA * kABytes;
    static constexpr int kOffB = kA * (kABytes + kSfSlab);
    static constexpr int kOffSfB = kOffB + kBBytes;
    static constexpr int kTokenBytes = kBBytes + kSfSlab;
    static constexpr int kStageBytes = kWeightBytes + kTokenBytes;
    static constexpr int kStagesRaw = (196 * 1024) / kStageBytes;
    static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
    static constexpr int kAccumStride = N < 32 ? 32 : N;          // each accumulator starts on a multiple of 32 columns
    static constexpr int kAccumCols = kA * kAccumStride;
    static constexpr int kSfCols = (kA + 1) * 16;                 // per buffer: 4 columns per K=64 step
    static constexpr int kAccumBuffers = 2 * kAccumCols + 2 * kSfCols <= 512 ? 2 : 1;
    static constexpr int kNeedCols = kAccumBuffers * kAccumCols + 2 * kSfCols;
    static constexpr int kTmemCols = kNeedCols <= 32 ? 32 : kNeedCols <= 64 ? 64 : kNeedCols <= 128 ? 128
                                     : kNeedCols <= 256 ? 256 : 512;
    static constexpr int kBarriers = 3 * kStages + 2 * kAccumBuffers;
    static constexpr int kBarrierBytes = kBarriers * 8 + 16;
    static constexpr int kSmemBytes = kStages * kStageBytes + kBarrierBytes + 1024;   // + alignment slack
    static_assert(kNeedCols <= 512, "accumulators and scale factors must fit TMEM");
};

// The gate/up epilogue for one chunk of 16 token columns (of expert_tc_kernel<0, N>).  A lane holds one weight row (row0 + lane of the intermediate dimension): gate g[j] and
// up u[j] for token column c0 + j.  bf16(alpha * product) for both, SwiGLU rounded to BF16
// (cuda/nvfp4_ops.cu:97-105), then the activation quantiser (cuda/nvfp4_ops.cu:818-841) along the intermediate
// dimension, whose 16-element blocks are the two 16-lane halves of the warp:
//   * block maximum of every column: one warp reduction per column over the half (|h| is a non-negative float, so
//     its bit pattern orders like an unsigned integer);
//   * the E4M3 scale and the multiplier of column c are computed ONCE, by lane c of the half, which also stores the
//     scale byte; the other lanes fetch the multiplier with one shuffle per column;
//   * a lane packs its 16 quantised values (one row, 16 tokens) into 64 bits, and a four-round butterfly over the
//     half transposes the 16 x 16 nibble matrix, after which lane c holds the 16 rows of token c0 + c: one 8-byte
//     store per lane instead of a byte store per lane pair and column.
// The arithmetic per element is the reference's; only who computes what has changed.
// hq_rows = packed rows of the tile's first token (p.hq + pp0 * inter / 2); hs_tile = the 128-row scale tile row of
// that token (p.hs + (pp0 >> 7) * (inter / 64) * 512); n_base = pp0 & 127; columns from `valid` on are not stored.
__device__ __forceinline__ void swiglu_requant_chunk(const std::uint32_t (&g)[16], const std::uint32_t (&u)[16], float alpha_g,
                                                     float alpha_u, float quant_scale, int lane, int c0, int valid, int n_base,
                                                     int inter, int row0, std::uint8_t* hq_rows, std::uint8_t* hs_tile) {
    const int half = lane >> 4;                       // which 16-row block of the warp's 32 rows
    const int c = lane & 15;                          // the column this lane owns after the reductions
    const unsigned half_mask = half ? 0xffff0000U : 0x0000ffffU;
    float h[16];
    std::uint32_t amax_bits[16];
    // the three BF16 roundings per element go through the two-wide conversion (one instruction for gate and up of a
    // column, one for the results of two columns): same round-to-nearest-even, fewer trips through the conversion pipe
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float silu_times_up[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = 2 * k + i;
            const std::uint32_t gu = bf16x2_bits(__uint_as_float(g[j]) * alpha_g, __uint_as_float(u[j]) * alpha_u);
            const float gv = __uint_as_float(gu << 16);
            const float uv = __uint_as_float(gu & 0xffff0000U);
            silu_times_up[i] = (gv / (1.0F + expf(-gv))) * uv;
        }
        const std::uint32_t hh = bf16x2_bits(silu_times_up[0], silu_times_up[1]);
        h[2 * k] = __uint_as_float(hh << 16);
        h[2 * k + 1] = __uint_as_float(hh & 0xffff0000U);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) amax_bits[j] = __reduce_max_sync(half_mask, __float_as_uint(h[j]) & 0x7fffffffU);
    // amax of the column this lane owns: a select tree over the 16 results (register arrays take no run-time index)
    std::uint32_t mine8[8], mine4[4], mine2[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) mine8[i] = (c & 8) ? amax_bits[8 + i] : amax_bits[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) mine4[i] = (c & 4) ? mine8[4 + i] : mine8[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) mine2[i] = (c & 2) ? mine4[2 + i] : mine4[i];
    const float amax = __uint_as_float((c & 1) ? mine2[1] : mine2[0]);
    const __nv_fp8_e4m3 scale(amax * (quant_scale / 6.0F));
    const float decoded = static_cast<float>(scale);
    const float my_multiplier = decoded == 0.0F ? 0.0F : quant_scale / decoded;
    const int n_mine = c0 + c;
    if (n_mine < valid) {
        const int sf_col = row0 >> 4;
        const int tn = n_base + n_mine;
        hs_tile[static_cast<std::size_t>(sf_col >> 2) * 512 + (sf_col & 3) + (tn & 31) * 16 + (tn >> 5) * 4] = scale.__x;
    }
    // this lane's row: 16 E2M1 values, column j at nibble j
    std::uint32_t w0 = 0U, w1 = 0U;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float m0 = __shfl_sync(0xffffffffU, my_multiplier, (lane & 16) | (2 * k));
        const float m1 = __shfl_sync(0xffffffffU, my_multiplier, (lane & 16) | (2 * k + 1));
        const std::uint32_t byte = __nv_fp4x2_e2m1(make_float2(h[2 * k] * m0, h[2 * k + 1] * m1)).__x;
        if (k < 4) w0 |= byte << (8 * k); else w1 |= byte << (8 * (k - 4));
    }
    // transpose the half's 16 x 16 nibble matrix: afterwards nibble r of lane c is (row r, column c)
    {
        const bool up8 = (lane & 8) != 0;                  // distance 8: whole words change hands
        const std::uint32_t got = __shfl_xor_sync(0xffffffffU, up8 ? w0 : w1, 8);
        if (up8) w0 = got; else w1 = got;
    }
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) {
        const std::uint32_t low = d == 4 ? 0x0000ffffU : d == 2 ? 0x00ff00ffU : 0x0f0f0f0fU;
        const int shift = 4 * d;
        const bool upper = (lane & d) != 0;
        const std::uint32_t s0 = upper ? (w0 & low) << shift : (w0 >> shift) & low;
        const std::uint32_t s1 = upper ? (w1 & low) << shift : (w1 >> shift) & low;
        const std::uint32_t r0 = __shfl_xor_sync(0xffffffffU, s0, d);
        const std::uint32_t r1 = __shfl_xor_sync(0xffffffffU, s1, d);
        w0 = (upper ? w0 & ~low : w0 & low) | r0;
        w1 = (upper ? w1 & ~low : w1 & low) | r1;
    }
    if (n_mine < valid) {
        *reinterpret_cast<uint2*>(hq_rows + static_cast<std::size_t>(n_mine) * (inter / 2) + (row0 >> 1)) =
            make_uint2(w0, w1);
    }
}

template <int MODE, int N, int SRC>
__global__ void __launch_bounds__(kThreadsTc, 1) expert_tc_kernel(const __grid_constant__ CUtensorMap map_b,
                                                                   const TcParams p) {
    using C = Tc<MODE, N>;
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ RouteTable route_table;
    const std::uint32_t base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    const std::uint32_t bars = base + C::kStages * C::kStageBytes;
    // per stage: weights landed, tokens landed, stage free; per accumulator buffer: full, empty
    auto weight_bar = [&](int s) { return bars + 8U * s; };
    auto token_bar = [&](int s) { return bars + 8U * (C::kStages + s); };
    auto empty_bar = [&](int s) { return bars + 8U * (2 * C::kStages + s); };
    auto accum_full = [&](int b) { return bars + 8U * (3 * C::kStages + b); };
    auto accum_empty = [&](int b) { return bars + 8U * (3 * C::kStages + C::kAccumBuffers + b); };
    const std::uint32_t tmem_slot = bars + 8U * C::kBarriers;
    volatile std::uint32_t* tmem_slot_ptr =
        reinterpret_cast<volatile std::uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
    volatile std::uint32_t* abort_ptr = tmem_slot_ptr + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int k_blocks = p.k_bytes / kBlockKBytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(weight_bar(s), 1);
            mbar_init(token_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < C::kAccumBuffers; ++b) {
            mbar_init(accum_full(b), 1);
            mbar_init(accum_empty(b), kEpilogueWarps);
        }
        *abort_ptr = 0;
        fence_mbar_init();
        prefetch_tensormap(&map_b);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::kTmemCols);
        tmem_relinquish();
    }
    // the routing lists come from the kernel just upstream (gate/up) or from one further up (down):
    // only the former has to wait for its predecessor before it can look at its work list
    if (p.routing_is_upstream || SRC == 1) pdl_wait();
    load_route_table(p, &route_table);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const std::uint32_t tmem_base = *tmem_slot_ptr;
    const int total_items = route_table.prefix[route_table.active_count] * p.m_tiles;
    auto give_up = [&]() {
        *abort_ptr = 1;
        atomicCAS(p.status, kStatusOk, kStatusWaitExpired);
    };

    if (warp == 0 && SRC == 1) {
        // ------------------------------------------------ producer, weights read in place
        // The matrices are row-major [rows][K/2] wherever the caller keeps them; the kernel upstream has built a tensor
        // map of each (assignment_rows_kernel, above 64 rows gather_quantized_rows_kernel), so a box of 128 rows is one tiled load.  (Gathered in 16-byte
        // pieces by this warp, 31 experts at 4 tokens took 35 us for gate and up against 20 from the bank's stream.)
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0;
            for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
                Item it;
                if (!decode_item<N>(p, route_table, item, &it)) continue;
                const int which = it.entry * 3 + (MODE == 1 ? p.table_kind : 0);
                bool aligned = true;
                const std::uint8_t* scales[C::kA];
#pragma unroll
                for (int a = 0; a < C::kA; ++a) {
                    scales[a] = p.table[which + a].scales_swizzled;
                    aligned = aligned && ((reinterpret_cast<std::uintptr_t>(p.table[which + a].weight) |
                                           reinterpret_cast<std::uintptr_t>(scales[a])) & 15U) == 0U;
                }
                if (!aligned) {
                    *abort_ptr = 1;                                   // the copies need 16-byte aligned matrices
                    atomicCAS(p.status, kStatusOk, kStatusBadPointer);
                    break;
                }
#pragma unroll
                for (int a = 0; a < C::kA; ++a) tensormap_acquire(p.table_maps + which + a);
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1U)) { give_up(); break; }
                    const std::uint32_t st = base + stage * C::kStageBytes;
                    mbar_arrive_expect_tx(weight_bar(stage), C::kWeightBytes);
#pragma unroll
                    for (int a = 0; a < C::kA; ++a) {
                        tma_load_2d(st + a * C::kABytes, p.table_maps + which + a, weight_bar(stage), kb * kBlockKBytes, it.m_tile * kTileM);
                        // scale slabs: row block m_tile, scale column blocks 4 kb .. 4 kb + 3 of the 128x4 tiling: 2 KB contiguous
                        bulk_load(st + C::kOffSfA + a * kSfSlab, scales[a] + (static_cast<std::size_t>(it.m_tile) * (k_blocks * 4) + kb * 4) * 512,
                                  kSfSlab, weight_bar(stage));
                    }
                    mbar_arrive_expect_tx(token_bar(stage), C::kTokenBytes);
                    tma_load_2d(st + C::kOffB, &map_b, token_bar(stage), kb * kBlockKBytes, it.pp0);
                    const std::uint8_t* bsf = p.b_sf + (static_cast<std::size_t>(it.pp0 >> 7) * (p.k_bytes / 32) + kb * 4) * 512;
                    bulk_load(st + C::kOffSfB, bsf, kSfSlab, token_bar(stage));
                    if (++stage == C::kStages) { stage = 0; phase ^= 1U; }
                }
            }
        }
    } else if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0;
            bool upstream_done = p.routing_is_upstream != 0;
            for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
                Item it;
                if (!decode_item<N>(p, route_table, item, &it)) continue;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1U)) { give_up(); break; }
                    const std::uint32_t st = base + stage * C::kStageBytes;
                    // weights never depend on the upstream kernel: they start streaming at once
                    mbar_arrive_expect_tx(weight_bar(stage), C::kWeightBytes);
                    if constexpr (MODE != 1) {
                        // one chunk = both boxes and both scale slabs of this (row tile, K block)
                        const std::uint8_t* chunk = p.bank.g13 +
                            ((static_cast<std::size_t>(it.entry) * p.m_tiles + it.m_tile) * k_blocks + kb) * kChunkBytes;
                        bulk_load(st, chunk, kChunkBytes, weight_bar(stage));
                    } else {
                        // chunks of the down stream hold two K blocks: take this block's box and slab
                        const std::uint8_t* chunk = p.bank.g2 +
                            ((static_cast<std::size_t>(it.entry) * p.m_tiles + it.m_tile) * (k_blocks / 2) + (kb >> 1)) *
                                kChunkBytes;
                        bulk_load(st, chunk + (kb & 1) * kChunkBox, kChunkBox, weight_bar(stage));
                        bulk_load(st + C::kOffSfA, chunk + kChunkScaleOffset + (kb & 1) * kChunkScaleBytes, kSfSlab,
                                  weight_bar(stage));
                    }
                    if (upstream_done) {
                        mbar_arrive_expect_tx(token_bar(stage), C::kTokenBytes);
                        tma_load_2d(st + C::kOffB, &map_b, token_bar(stage), kb * kBlockKBytes, it.pp0);
                        const std::uint8_t* bsf = p.b_sf +
                            (static_cast<std::size_t>(it.pp0 >> 7) * (p.k_bytes / 32) + kb * 4) * 512;
                        bulk_load(st + C::kOffSfB, bsf, kSfSlab, token_bar(stage));
                    }
                    const bool ring_full = stage == C::kStages - 1;
                    const bool last_load = kb == k_blocks - 1 && item + static_cast<int>(gridDim.x) >= total_items;
                    if (!upstream_done && (ring_full || last_load)) {
                        // every stage now has its weights in flight; the token rows are written by the
                        // upstream kernel, so wait for it, then issue the token loads that were held back
                        pdl_wait();
                        upstream_done = true;
                        int it_item = blockIdx.x, it_kb = 0;
                        for (int s = 0; s <= stage; ++s) {
                            Item held;
                            while (!decode_item<N>(p, route_table, it_item, &held)) it_item += gridDim.x;
                            const std::uint32_t hst = base + s * C::kStageBytes;
                            mbar_arrive_expect_tx(token_bar(s), C::kTokenBytes);
                            tma_load_2d(hst + C::kOffB, &map_b, token_bar(s), it_kb * kBlockKBytes, held.pp0);
                            const std::uint8_t* hsf = p.b_sf +
                                (static_cast<std::size_t>(held.pp0 >> 7) * (p.k_bytes / 32) + it_kb * 4) * 512;
                            bulk_load(hst + C::kOffSfB, hsf, kSfSlab, token_bar(s));
                            if (++it_kb == k_blocks) { it_kb = 0; it_item += gridDim.x; }
                        }
                    }
                    if (++stage == C::kStages) { stage = 0; phase ^= 1U; }
                }
            }
            if (!upstream_done) pdl_wait();      // no work at all: still order this grid after its predecessor
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------- MMA issuer
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0;
            int buffer = 0;
            std::uint32_t accum_phase[2] = {0U, 0U};
            constexpr std::uint32_t idesc = idesc_nvf4(kTileM, N);
            const std::uint32_t sf_tmem = tmem_base + C::kAccumBuffers * C::kAccumCols;
            int sf_buffer = 0;
            for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
                Item it;
                if (!decode_item<N>(p, route_table, item, &it)) continue;
                if (!mbar_wait(accum_empty(buffer), accum_phase[buffer] ^ 1U)) { give_up(); break; }
                tc_fence_after();
                const std::uint32_t accum = tmem_base + buffer * C::kAccumCols;
                // a 64-row token tile may start in the middle of a 128-row scale tile: its scales then sit
                // two TMEM columns further (rows 64..127 are quarters 2 and 3 of the tile)
                const std::uint32_t b_quarter = static_cast<std::uint32_t>((it.pp0 & 127) >> 5);
                bool ok = true;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(weight_bar(stage), phase) || !mbar_wait(token_bar(stage), phase)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const std::uint32_t st = base + stage * C::kStageBytes;
                    const std::uint32_t sfc = sf_tmem + sf_buffer * C::kSfCols;
#pragma unroll
                    for (int o = 0; o < C::kA + 1; ++o) {
                        const std::uint32_t slab = o < C::kA ? st + C::kOffSfA + o * kSfSlab : st + C::kOffSfB;
#pragma unroll
                        for (int k = 0; k < 4; ++k) tc_copy_sf(sfc + o * 16 + k * 4, desc_scale_atom(slab + k * 512));
                    }
                    const std::uint64_t b_desc = desc_k_major_sw128(st + C::kOffB);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
#pragma unroll
                        for (int a = 0; a < C::kA; ++a) {
                            const std::uint64_t a_desc = desc_k_major_sw128(st + a * C::kABytes);
                            mma_nvf4(accum + a * C::kAccumStride, a_desc + 2 * k, b_desc + 2 * k, idesc,
                                     sfc + a * 16 + k * 4, sfc + C::kA * 16 + k * 4 + b_quarter, kb > 0 || k > 0);
                        }
                    }
                    tc_commit(empty_bar(stage));
                    sf_buffer ^= 1;
                    if (++stage == C::kStages) { stage = 0; phase ^= 1U; }
                }
                if (!ok) break;
                tc_commit(accum_full(buffer));
                accum_phase[buffer] ^= 1U;
                if (C::kAccumBuffers == 2) buffer ^= 1;
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        // Sixteen warps: warp w reads TMEM lanes 32*(w & 3) .. +31 (one output row per lane) and the four
        // warps of a quarter take every fourth 16-column chunk.  A chunk is processed without any
        // data-dependent branch so the sixteen per-column dependency chains interleave; only the
        // stores are predicated on the column being a real token.
        const int quarter = warp & 3;
        const int half = (warp - 2) >> 2;
        int buffer = 0;
        std::uint32_t accum_phase[2] = {0U, 0U};
        for (int item = blockIdx.x; item < total_items && !*abort_ptr; item += gridDim.x) {
            Item it;
            if (!decode_item<N>(p, route_table, item, &it)) continue;
            if (!mbar_wait(accum_full(buffer), accum_phase[buffer])) { give_up(); break; }
            accum_phase[buffer] ^= 1U;
            tc_fence_after();
            const std::uint32_t lane_base =
                tmem_base + buffer * C::kAccumCols + (static_cast<std::uint32_t>(quarter * 32) << 16);
            const int row = it.m_tile * kTileM + quarter * 32 + lane;          // output row of this lane
            if constexpr (MODE == 0) {
                const float alpha_g = p.bank.alpha[it.entry * 3 + 0];
                const float alpha_u = p.bank.alpha[it.entry * 3 + 1];
                const int inter = p.m_total;
                // the token tile's packed rows and its 128-row scale tile; pp0 is a multiple of N
                std::uint8_t* hs_tile = p.hs + static_cast<std::size_t>(it.pp0 >> 7) * (inter / 64) * 512;
                std::uint8_t* hq_rows = p.hq + static_cast<std::size_t>(it.pp0) * (inter / 2);
                const int n_base = it.pp0 & 127;
                const int row0 = it.m_tile * kTileM + gu_tile_row(quarter, lane & 16);      // of this half warp's 16 rows
#pragma unroll 1
                for (int c0 = half * 16; c0 < N; c0 += 16 * (kEpilogueWarps / 4)) {
                    if (c0 >= it.valid) break;                                    // warp uniform
                    std::uint32_t g[16], u[16];
                    tmem_load16(lane_base + c0, g);
                    tmem_load16(lane_base + C::kAccumStride + c0, u);
                    tmem_load_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) gu_exchange(g[j], u[j], lane, &g[j], &u[j]);
                    swiglu_requant_chunk(g, u, alpha_g, alpha_u, p.quant_scale, lane, c0, it.valid, n_base, inter, row0, hq_rows, hs_tile);
                }
            } else if constexpr (MODE == 2) {
                // gate and up rows as the reference's project_expert_gate_up returns them: bf16(alpha * product),
                // row (token, slot) of the caller's [rows * 8][intermediate] buffers
                const float alpha_g = SRC == 1 ? *p.table[it.entry * 3 + 0].alpha : p.bank.alpha[it.entry * 3 + 0];
                const float alpha_u = SRC == 1 ? *p.table[it.entry * 3 + 1].alpha : p.bank.alpha[it.entry * 3 + 1];
                const int inter = p.m_total;
                // a caller's table is read in place, gate rows and up rows apart; the bank's boxes mix them
                const int my_row = SRC == 1 ? row : it.m_tile * kTileM + gu_tile_row(quarter, lane);
#pragma unroll 1
                for (int c0 = half * 16; c0 < N; c0 += 16 * (kEpilogueWarps / 4)) {
                    if (c0 >= it.valid) break;
                    std::uint32_t g[16], u[16];
                    tmem_load16(lane_base + c0, g);
                    tmem_load16(lane_base + C::kAccumStride + c0, u);
                    tmem_load_wait();
                    if constexpr (SRC == 0) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) gu_exchange(g[j], u[j], lane, &g[j], &u[j]);
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int n = c0 + j;
                        if (n < it.valid) {
                            const std::size_t r = static_cast<std::size_t>(p.out_row != nullptr ? p.out_row[it.dense0 + n] : it.pp0 + n);
                            p.gate_out[r * inter + my_row] = float_to_bf16_bits(__uint_as_float(g[j]) * alpha_g);
                            p.up_out[r * inter + my_row] = float_to_bf16_bits(__uint_as_float(u[j]) * alpha_u);
                        }
                    }
                }
            } else {
                const float alpha = SRC == 1 ? *p.table[it.entry * 3 + p.table_kind].alpha : p.bank.alpha[it.entry * 3 + 2];
                const int hidden = p.m_total;
#pragma unroll 1
                for (int c0 = half * 16; c0 < N; c0 += 16 * (kEpilogueWarps / 4)) {
                    if (c0 >= it.valid) break;
                    std::uint32_t d[16];
                    tmem_load16(lane_base + c0, d);
                    tmem_load_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int n = c0 + j;
                        if (n < it.valid) {
                            const std::size_t r = static_cast<std::size_t>(p.out_row != nullptr ? p.out_row[it.dense0 + n] : it.pp0 + n);
                            p.out[r * hidden + row] = float_to_bf16_bits(__uint_as_float(d[j]) * alpha);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accum_empty(buffer));
            if (C::kAccumBuffers == 2) buffer ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// Quantises the token rows into the padded position space of the tensor-core kernels: a row is read and quantised once and
// written to the nine places it is needed, its eight routed slots and its shared-expert row.  WARPS per token: 8 while
// there are fewer tokens than would fill the chip with one each - a lane then has one block to read and nine pieces to
// write instead of five of each one after the other (9.0 us at 64 and at 512 rows) - else 1.
template <int WARPS>
__global__ void __launch_bounds__(256) quantize_padded_kernel(const std::uint16_t* __restrict__ x,
                                                              const std::int32_t* __restrict__ pp_of_flat,
                                                              std::uint8_t* __restrict__ xq,
                                                              std::uint8_t* __restrict__ xs, int rows, int hidden,
                                                              float global_scale) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int token = (blockIdx.x * (blockDim.x >> 5) + warp) / WARPS;
    if (token >= rows) return;
    // the nine destinations of the row, fetched before the row itself so that the stores wait for nothing
    const int place_index = lane < kTop ? token * kTop + lane : rows * kTop + token;
    const int my_pp = lane <= kTop ? __ldg(pp_of_flat + place_index) : 0;
    QuantisedRow<WARPS> row;
    row.load(x + static_cast<std::size_t>(token) * hidden, hidden, warp % WARPS);
    row.quantise(global_scale);
#pragma unroll 1
    for (int place = 0; place <= kTop; ++place) row.store(xq, xs, static_cast<std::size_t>(__shfl_sync(0xffffffffU, my_pp, place)));
}

// The same for rows that each have ONE destination (the dense MLP's token rows, the (row, slot) intermediate rows
// of the down stage entry point): row i of `x` [n][width] goes to padded position index[i] (i itself if index is null).
__global__ void __launch_bounds__(256) quantize_rows_to_pp_kernel(const std::uint16_t* __restrict__ x,
                                                                  const std::int32_t* __restrict__ index,
                                                                  std::uint8_t* __restrict__ xq,
                                                                  std::uint8_t* __restrict__ xs, int n, int width,
                                                                  float global_scale) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n) return;
    const int blocks = width / 16;
    const int col_blocks = (blocks + 3) / 4;
    const std::size_t pp = static_cast<std::size_t>(index != nullptr ? index[row] : row);
    std::uint8_t* row_q = xq + pp * (width / 2);
    std::uint8_t* row_s = xs + (pp >> 7) * col_blocks * 512 + (pp & 31) * 16 + ((pp >> 5) & 3) * 4;
    for (int b = lane; b < blocks; b += 32) {
        const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<std::size_t>(row) * width + b * 16);
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
        const uint2 packed = quantize_block16(v, global_scale, &scale_bits);
        *reinterpret_cast<uint2*>(row_q + b * 8) = packed;
        row_s[(b >> 2) * 512 + (b & 3)] = scale_bits;
    }
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    if (fn == nullptr) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult query;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &query) == cudaSuccess &&
            query == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiled>(sym);
        }
    }
    return fn;
}

template <int MODE, int N, int SRC = 0>
cudaError_t launch_tc(const p92b_plan* plan, const CUtensorMap& map_b, const TcParams& p, cudaStream_t stream,
                      bool pdl) {
    using C = Tc<MODE, N>;
    auto kernel = expert_tc_kernel<MODE, N, SRC>;
    if (cudaError_t st = ensure_dynamic_smem<expert_tc_kernel<MODE, N, SRC>>(C::kSmemBytes); st != cudaSuccess) return st;
    return launch_kernel(kernel, dim3(plan->sm_count), dim3(kThreadsTc), C::kSmemBytes, stream, pdl, map_b, p);
}

}  // namespace

// Row-major byte matrix [rows][row_bytes] as a 2-D tensor map with a 128-byte x box_rows box and
// the 128-byte swizzle (what the K-major operand descriptors expect).
cudaError_t make_operand_map(CUtensorMap* map, const void* base, std::size_t rows, std::size_t row_bytes,
                             int box_rows) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kBlockKBytes), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Token tile of the expert kernels.  Above 32 rows it stays at 64 columns: two gate/up accumulator pairs
// then fit TMEM side by side, so the epilogue of one tile overlaps the MMAs of the next.
int tc_tile_rows(int rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : 64; }
// Every entry's rows start on a multiple of 128 padded positions, so a token tile always begins at
// row 0 of a 128-row scale-factor tile (TMEM lane 0, first scale column).
int tc_pad_align(int rows) { (void)rows; return 128; }

cudaError_t launch_quantize_padded(const p92b_plan* plan, const std::uint16_t* x, int rows, cudaStream_t stream,
                                   bool pdl) {
    if (plan->hidden > 4096) return cudaErrorNotSupported;
    if (!aligned_to(16, x)) return cudaErrorInvalidValue;
    const bool few = rows <= 1024;
    return launch_kernel(few ? quantize_padded_kernel<8> : quantize_padded_kernel<1>, dim3(few ? rows : (rows + 7) / 8), dim3(256), 0,
                         stream, pdl, x, static_cast<const std::int32_t*>(plan->pp_of_flat), plan->xq_pp, plan->xs_sw, rows,
                         plan->hidden, 1.0F);
}

cudaError_t launch_quantize_rows_to_pp(const std::uint16_t* x, const std::int32_t* index, std::uint8_t* xq,
                                       std::uint8_t* xs, int n, int width, cudaStream_t stream, bool pdl) {
    if (x == nullptr || xq == nullptr || xs == nullptr || n <= 0 || width <= 0 || width % 64 != 0 || !aligned_to(16, x)) {
        return cudaErrorInvalidValue;
    }
    return launch_kernel(quantize_rows_to_pp_kernel, dim3((n + 7) / 8), dim3(256), 0, stream, pdl, x, index, xq, xs, n, width,
                         1.0F);
}

namespace {
bool slab_shape(const p92b_plan* plan) {
    return plan->wide_rows == 128 && down_slab_shape(plan->hidden, plan->intermediate) && std::getenv("P92B_NO_DOWN_SLAB") == nullptr;
}
}  // namespace

bool down_slab_applies(const p92b_plan* plan, int rows) { return tc_tile_rows(rows) == 64 && slab_shape(plan); }

cudaError_t launch_experts_tc(const p92b_plan* plan, const p92b_bank* bank, int rows, bool down,
                              cudaStream_t stream, bool pdl, const TcIo* io) {
    const bool in_place = io != nullptr && io->table != nullptr;
    if (!plan->tc_ready || (!in_place && (bank == nullptr || !bank->tc_ready))) return cudaErrorNotSupported;
    TcParams p {};
    if (bank != nullptr) p.bank = bank->view;
    p.route.counts = plan->counts;
    p.route.offsets = plan->offsets;
    p.route.row_token = plan->row_token;
    p.route.active = plan->active;
    p.route.active_count = plan->active_count;
    p.pp_off = plan->pp_off;
    p.tile_prefix = plan->tile_prefix;
    p.status = plan->status;
    p.quant_scale = 1.0F;
    if (io != nullptr) {
        p.out_row = io->out_row;
        p.gate_out = io->gate_out;
        p.up_out = io->up_out;
        p.table = io->table;
        p.table_kind = io->table_kind;
        p.table_maps = plan->table_maps;
        p.skip_shared = io->skip_shared ? 1 : 0;
        p.row_dest = io->row_dest;
    }
    const bool unfused = io != nullptr && io->gate_out != nullptr;
    const bool single = io != nullptr && io->single_matrix;      // one matrix of the token-row side (gate or up alone)
    const int n = tc_tile_rows(rows);
    const int which = n == 16 ? 0 : n == 32 ? 1 : 2;
    p.routing_is_upstream = down && !(io != nullptr && io->wait_upstream) ? 0 : 1;
    if (!down) {
        p.b_sf = plan->xs_sw;
        p.hq = plan->hq_pp;
        p.hs = plan->hs_sw;
        p.k_bytes = plan->hidden / 2;
        p.m_total = plan->intermediate;
        p.m_tiles = plan->intermediate / kTileM;
        if (single) {
            if (!in_place || io->down_out == nullptr) return cudaErrorInvalidValue;
            p.out = io->down_out;
            switch (which) {
                case 0: return launch_tc<1, 16, 1>(plan, plan->map_x[0], p, stream, pdl);
                case 1: return launch_tc<1, 32, 1>(plan, plan->map_x[1], p, stream, pdl);
                default: return launch_tc<1, 64, 1>(plan, plan->map_x[2], p, stream, pdl);
            }
        }
        if (unfused) {
            if (io->up_out == nullptr) return cudaErrorInvalidValue;
            switch (which) {
                case 0: return in_place ? launch_tc<2, 16, 1>(plan, plan->map_x[0], p, stream, pdl)
                                        : launch_tc<2, 16, 0>(plan, plan->map_x[0], p, stream, pdl);
                case 1: return in_place ? launch_tc<2, 32, 1>(plan, plan->map_x[1], p, stream, pdl)
                                        : launch_tc<2, 32, 0>(plan, plan->map_x[1], p, stream, pdl);
                default: return in_place ? launch_tc<2, 64, 1>(plan, plan->map_x[2], p, stream, pdl)
                                         : launch_tc<2, 64, 0>(plan, plan->map_x[2], p, stream, pdl);
            }
        }
        if (io != nullptr && io->scales_by_row && (which != 2 || plan->wide_rows != 128)) return cudaErrorNotSupported;
        if (in_place) return cudaErrorNotSupported;              // the fused gate/up epilogue reads the bank's stream
        switch (which) {
            case 0: return launch_tc<0, 16>(plan, plan->map_x[0], p, stream, pdl);
            case 1: return launch_tc<0, 32>(plan, plan->map_x[1], p, stream, pdl);
            default:
                // Lists with 128-row tiles (every call of more than 32 rows except the expert-parallel ones that build
                // their lists themselves): tokens on the M side.  It is the quicker form over the whole range: by 2 % at 64
                // rows and 5 % at 512, where both run near the HBM time of the weights, 163 against 201 us at 4,096, 394
                // against 563 at 16,384.
                if (plan->wide_rows == 128) {
                    p.tile_prefix = plan->tile_prefix_wide;
                    return launch_expert_rows_gate_up(plan, p, io != nullptr && io->scales_by_row, stream, pdl);
                }
                return launch_tc<0, 64>(plan, plan->map_x[2], p, stream, pdl);
        }
    }
    p.b_sf = plan->hs_sw;
    p.out = io != nullptr && io->down_out != nullptr ? io->down_out : plan->mixed_pp;
    p.k_bytes = plan->intermediate / 2;
    p.m_total = plan->hidden;
    p.m_tiles = plan->hidden / kTileM;
    if (in_place) {
        switch (which) {
            case 0: return launch_tc<1, 16, 1>(plan, plan->map_h[0], p, stream, pdl);
            case 1: return launch_tc<1, 32, 1>(plan, plan->map_h[1], p, stream, pdl);
            default: return launch_tc<1, 64, 1>(plan, plan->map_h[2], p, stream, pdl);
        }
    }
    if (p.row_dest != nullptr && which != 2) return cudaErrorNotSupported;
    switch (which) {
        case 0: return launch_tc<1, 16>(plan, plan->map_h[0], p, stream, pdl);
        case 1: return launch_tc<1, 32>(plan, plan->map_h[1], p, stream, pdl);
        default:
            if (plan->wide_rows == 128) {
                // every expert segment starts on a multiple of 128 padded rows, so 128-row tiles stay inside it
                p.tile_prefix = plan->tile_prefix_wide;
                const bool plain = io == nullptr || (io->down_out == nullptr && io->out_row == nullptr && !io->skip_shared);
                if (plain && slab_shape(plan)) {
                    // the token slab resident in shared memory, only weights streaming
                    return launch_expert_down_slab(plan, p, stream, pdl);
                }
                if (p.row_dest != nullptr) return cudaErrorNotSupported;
                // any K: 128 x 256 tiles with the tokens on the M side (dense MLP, 3,807 rows: both products together 196 ->
                // 141 us per layer); it stores whole token tiles of every entry at their padded positions, 16 bytes at a time
                if (p.out_row == nullptr && p.skip_shared == 0 && (reinterpret_cast<std::uintptr_t>(p.out) & 15U) == 0U) {
                    return launch_expert_rows_matrix(plan, p, stream, pdl);
                }
                return launch_tc<1, 128>(plan, plan->map_h[3], p, stream, pdl);
            }
            if (p.row_dest != nullptr) return cudaErrorNotSupported;
            return launch_tc<1, 64>(plan, plan->map_h[2], p, stream, pdl);
    }
}

// Rows that the caller has already quantised in the reference's layout (packed [R][K/2], scales 128x4-tiled over
// the R rows): assignment i takes source row src_row (i itself, or its token i / 8 when the eight slots of a token
// share one row) and is copied to padded position pp_of_flat[i], its scale bytes to the tiled position of that row.
namespace {
__global__ void __launch_bounds__(256) gather_quantized_rows_kernel(const std::uint8_t* __restrict__ packed,
                                                                    const std::uint8_t* __restrict__ scales_swizzled,
                                                                    const std::int32_t* __restrict__ pp_of_flat,
                                                                    std::uint8_t* __restrict__ xq, std::uint8_t* __restrict__ xs,
                                                                    int assignments, int k_bytes, int distinct_rows,
                                                                    const __grid_constant__ TableMaps maps) {
    __shared__ __align__(128) std::uint32_t map_image[8][32];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int gather_blocks = (assignments + 7) / 8;
    const int i = blockIdx.x * 8 + warp;
    if (static_cast<int>(blockIdx.x) >= gather_blocks) {
        // a warp per matrix of an active expert; slot 0 is the shared expert, which has no rows here
        const int m = i - gather_blocks * 8;
        const int slot = 1 + m / maps.kinds;
        if (slot < *maps.active_count) build_table_map(maps, maps.active[slot] * 3 + maps.first_kind + m % maps.kinds, map_image[warp]);
        return;
    }
    if (i >= assignments) return;
    const std::size_t src = static_cast<std::size_t>(distinct_rows ? i : i / kTop);
    const std::size_t pp = static_cast<std::size_t>(pp_of_flat[i]);
    copy_quantised_row(packed, scales_swizzled, src, xq, xs, pp, k_bytes);
}
}  // namespace

cudaError_t launch_gather_quantized_rows(const std::uint8_t* packed, const std::uint8_t* scales_swizzled,
                                         const std::int32_t* pp_of_flat, std::uint8_t* xq, std::uint8_t* xs, int assignments,
                                         int k_bytes, bool distinct_rows, const TableMaps& maps, cudaStream_t stream, bool pdl) {
    if (packed == nullptr || scales_swizzled == nullptr || assignments <= 0 || k_bytes % 16 != 0 ||
        (reinterpret_cast<std::uintptr_t>(packed) & 15U) != 0U) {
        return cudaErrorInvalidValue;
    }
    const int map_warps = std::min(assignments, kExperts) * maps.kinds;
    return launch_kernel(gather_quantized_rows_kernel, dim3((assignments + 7) / 8 + (map_warps + 7) / 8), dim3(256), 0, stream, pdl,
                         packed, scales_swizzled, pp_of_flat, xq, xs, assignments, k_bytes, distinct_rows ? 1 : 0, maps);
}

}  // namespace p92b
