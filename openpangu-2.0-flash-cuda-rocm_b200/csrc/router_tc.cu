// Router for large batches: tensor-core logits, then exact repair of the few that decide the routing.
//
// The reference's logits are FP32 fmaf chains in a fixed order (cuda/nvfp4_ops.cu:178-207): lane l of a warp sums
// columns l, l+32, ... and a shuffle-down tree adds the 32 partial sums.  Expert ids must equal the reference's, so
// every logit that can influence the top-8 has to be THAT number - but almost none can: of 256 logits per token only
// those near the top-8 boundary matter.  Two kernels:
//
//   1. logits_tc_kernel      approximate logits of every (token, expert) as one BF16 x BF16 -> FP32 product on the
//                            5th-generation tensor cores (tcgen05.mma kind::f16, M = 128 tokens, N = 64 to 256 experts
//                            per block, operands by TMA, accumulator in TMEM), and beside it ||w_e||_2 of the 256 router
//                            rows (the error bound below needs them);
//   2. route_repair_kernel   one warp per token: corrected scores from the approximate logits, the approximate 8th
//                            best, the candidate set = every expert whose approximate score is within 2 delta of it,
//                            the candidates' logits recomputed in the reference's exact order, and the reference's
//                            top-8 (cuda/nvfp4_ops.cu:357-433: higher corrected score first, ties to the lower id,
//                            weights from the uncorrected sigmoid, renormalised) taken over the exact values.
//
// Why that is exact.  Let delta bound |approximate - exact| of a corrected score.  An expert outside the candidate set
// has approximate score < a8 - 2 delta (a8 = approximate 8th best), so its exact score is < a8 - delta, while each of
// the eight approximately best experts has exact score >= a8 - delta: eight experts beat it, it is not in the exact
// top-8.  Hence the exact top-8 is a subset of the candidates, and selecting among exactly recomputed candidates
// gives the reference's ids and weights bit for bit.  delta = 0.25 * kLogitBound * ||x_t|| * ||w_e|| + 4e-6: the
// sigmoid's slope is at most 1/4; both the reference chain and the tensor-core sum differ from the true dot product by
// at most (number of sequential roundings) * 2^-23 * sum|x_i w_i| <= that * ||x|| ||w||, with about 85 roundings in the
// reference's order and fewer than 200 in the tensor core's; kLogitBound = 2^-14 is more than twice their sum; 4e-6
// covers the fast-math sigmoid's own error on both sides.  A token whose candidate set would exceed 24 experts or
// has fewer than eight, or that holds a non-finite logit, has its whole row recomputed exactly instead.
//
// The logits buffer keeps the approximate values except at the recomputed positions, which hold the exact ones.
#include "p92b_common.cuh"
#include "tc_ptx.cuh"

#include <algorithm>
#include <cstdlib>

namespace p92b {

using namespace ptx;

namespace {

constexpr int kTokTile = 128;                 // M: tokens per block (TMEM lanes)
constexpr int kKBytes = 128;                  // one swizzle row: 64 BF16
constexpr int kStageA = kTokTile * kKBytes;   // 16 KB
// N: experts per block, 64, 128 or 256.  A block is bound by the bytes it brings in, and the token rows come once per expert
// tile: with 64 experts a block 16,384 tokens took 50 us, four rounds of blocks that read every row four times.
template <int N>
struct Logits {
    static constexpr int kStageBytes = kStageA + N * kKBytes;          // 24, 32 or 48 KB
    static constexpr int kStages = 196 * 1024 / kStageBytes;          // 8, 6 or 4
    static constexpr int kSmem = kStages * kStageBytes + 1024;
};
constexpr int kLogitThreads = 192;            // producer warp, MMA warp, four epilogue warps
constexpr float kLogitBound = 1.0F / 16384.0F;
constexpr int kMaxCandidates = 24;

// D[tmem] (+)= A[smem] * B[smem], BF16 operands (both K-major), FP32 accumulate, M=128, K=16 per instruction.
__device__ __forceinline__ void mma_bf16(std::uint32_t d_tmem, std::uint64_t a_desc, std::uint64_t b_desc,
                                         std::uint32_t idesc, bool accumulate) {
    asm volatile(
        "{ .reg .pred p;\n"
        "  setp.ne.b32 p, %4, 0;\n"
        "  tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<std::uint32_t>(accumulate))
        : "memory");
}

// Instruction descriptor for kind::f16: FP32 accumulator (bits [4,6) = 1), BF16 A and B (bits [7,10) and [10,13) = 1),
// both K-major, N >> 3 in [17,23), M >> 4 in [24,29).
__host__ __device__ constexpr std::uint32_t idesc_bf16(int m, int n) {
    return (1U << 4) | (1U << 7) | (1U << 10) | (static_cast<std::uint32_t>(n >> 3) << 17) |
           (static_cast<std::uint32_t>(m >> 4) << 24);
}

// ||w_e|| of one router row, by a warp; and, for hidden = 2,560, the row once more in the order in which the exact chains
// take it: piece (c, lane) of 16 bytes holds columns lane + 32 (8 c + i), i = 0 .. 7, so that a lane of the repair kernel
// reads eight steps of its chain with one load.
constexpr int kChunksInRegisters = 80;                    // hidden / 32
__device__ __forceinline__ void row_norm(const std::uint16_t* __restrict__ w, float* __restrict__ norms,
                                         std::uint16_t* __restrict__ w_chains, int e, int hidden) {
    const int lane = threadIdx.x & 31;
    float s = 0.0F;
    if (w_chains != nullptr) {
        const std::uint16_t* row = w + static_cast<std::size_t>(e) * hidden + lane;
        uint4* to = reinterpret_cast<uint4*>(w_chains + static_cast<std::size_t>(e) * hidden) + lane;
#pragma unroll 5
        for (int c = 0; c < kChunksInRegisters / 8; ++c) {
            std::uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __ldg(row + 32 * (8 * c + i));
#pragma unroll
            for (int i = 0; i < 8; ++i) s = fmaf(__uint_as_float(v[i] << 16), __uint_as_float(v[i] << 16), s);
            to[32 * c] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
        }
    } else {
        const uint4* row = reinterpret_cast<const uint4*>(w + static_cast<std::size_t>(e) * hidden);
#pragma unroll 10
        for (int v = lane; v < hidden / 8; v += 32) {
            const uint4 q = __ldg(row + v);
            const std::uint32_t words[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float lo = __uint_as_float(words[k] << 16), hi = __uint_as_float(words[k] & 0xffff0000U);
                s = fmaf(lo, lo, s);
                s = fmaf(hi, hi, s);
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffU, s, off);
    if (lane == 0) norms[e] = sqrtf(s) * 1.0001F;             // rounded up a little: it feeds a bound
}

template <int kExpTile>
__global__ void __launch_bounds__(kLogitThreads, 1) logits_tc_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                     const __grid_constant__ CUtensorMap map_w,
                                                                     float* __restrict__ logits, int rows, int hidden,
                                                                     std::int32_t* status, const std::uint16_t* __restrict__ w,
                                                                     float* __restrict__ norms,
                                                                     std::uint16_t* __restrict__ w_chains) {
    // gridDim.z > 1: block z takes a slice of the K blocks and writes its partial sums to slice z of `logits`
    // ([gridDim.z][rows][256]); the repair kernel adds the slices (small batches: 4 blocks would otherwise walk all of
    // K one after the other while 144 SMs idle)
    constexpr int kLogitStages = Logits<kExpTile>::kStages, kStageBytes = Logits<kExpTile>::kStageBytes;
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ __align__(8) std::uint64_t barrier_words[2 * kLogitStages + 1];
    __shared__ std::uint32_t tmem_slot_word;
    __shared__ volatile std::uint32_t abort_word;
    const std::uint32_t base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    const std::uint32_t bars = smem_u32(barrier_words);
    auto full_bar = [&](int s) { return bars + 8U * s; };
    auto empty_bar = [&](int s) { return bars + 8U * (kLogitStages + s); };
    const std::uint32_t accum_bar = bars + 8U * (2 * kLogitStages);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int all_k_blocks = hidden * 2 / kKBytes;
    const int per_split = (all_k_blocks + static_cast<int>(gridDim.z) - 1) / static_cast<int>(gridDim.z);
    const int kb_first = min(all_k_blocks, static_cast<int>(blockIdx.z) * per_split);
    const int k_blocks = min(all_k_blocks, kb_first + per_split) - kb_first;       // this block's share
    const int t0 = blockIdx.x * kTokTile;
    const int e0 = blockIdx.y * kExpTile;
    logits += static_cast<std::size_t>(blockIdx.z) * rows * kExperts;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kLogitStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(accum_bar, 1);
        abort_word = 0;
        fence_mbar_init();
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_w);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_slot_word), kExpTile);
        tmem_relinquish();
    }
    pdl_wait();                       // the token rows come from the kernel before this one
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const std::uint32_t tmem_base = tmem_slot_word;
    auto give_up = [&]() {
        abort_word = 1;
        atomicCAS(status, kStatusOk, kStatusWaitExpired);
    };

    if (warp == 0) {
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0;
            for (int kb = 0; kb < k_blocks && !abort_word; ++kb) {
                if (!mbar_wait(empty_bar(stage), phase ^ 1U)) { give_up(); break; }
                const std::uint32_t st = base + stage * kStageBytes;
                mbar_arrive_expect_tx(full_bar(stage), kStageBytes);
                tma_load_2d(st, &map_x, full_bar(stage), (kb_first + kb) * kKBytes, t0);        // rows beyond the batch read as zero
                tma_load_2d(st + kStageA, &map_w, full_bar(stage), (kb_first + kb) * kKBytes, e0);
                if (++stage == kLogitStages) { stage = 0; phase ^= 1U; }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int stage = 0;
            std::uint32_t phase = 0;
            constexpr std::uint32_t idesc = idesc_bf16(kTokTile, kExpTile);
            bool ok = true;
            for (int kb = 0; kb < k_blocks && !abort_word; ++kb) {
                if (!mbar_wait(full_bar(stage), phase)) { give_up(); ok = false; break; }
                tc_fence_after();
                const std::uint32_t st = base + stage * kStageBytes;
                const std::uint64_t a_desc = desc_k_major_sw128(st);
                const std::uint64_t b_desc = desc_k_major_sw128(st + kStageA);
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_bf16(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, kb > 0 || k > 0);
                tc_commit(empty_bar(stage));
                if (++stage == kLogitStages) { stage = 0; phase ^= 1U; }
            }
            if (ok && k_blocks > 0) tc_commit(accum_bar);
        }
    } else {
        // while the products run, the epilogue warps take the norms of the tile's router rows, shared out over the blocks of
        // this expert tile (a kernel of its own in front of this one cost the chain 2 us)
        const int sharers = static_cast<int>(gridDim.x * gridDim.z) * 4;
        for (int i = static_cast<int>(blockIdx.x * gridDim.z + blockIdx.z) * 4 + (warp - 2); i < kExpTile; i += sharers) {
            row_norm(w, norms, w_chains, e0 + i, hidden);
        }
        const int quarter = warp & 3;                       // TMEM lanes 32 * quarter ..: the token rows of this warp
        if (k_blocks == 0) {
            // an empty slice: nothing was issued
        } else if (mbar_wait(accum_bar, 0)) {
            tc_fence_after();
            const int token = t0 + quarter * 32 + lane;
            const std::uint32_t lane_base = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16);
#pragma unroll
            for (int c0 = 0; c0 < kExpTile; c0 += 16) {
                std::uint32_t v[16];
                tmem_load16(lane_base + c0, v);
                tmem_load_wait();
                if (token < rows) {
                    float4* dst = reinterpret_cast<float4*>(logits + static_cast<std::size_t>(token) * kExperts + e0 + c0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        dst[q] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                             __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
                    }
                }
            }
        } else {
            give_up();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kExpTile);
    }
}

// Exact logit of (token row in shared memory, router row in global memory) in the reference's T > 1 order.
__device__ __forceinline__ float exact_logit(const std::uint16_t* __restrict__ x_row, const std::uint16_t* __restrict__ w_row,
                                             int hidden, int lane) {
    float value = 0.0F;
#pragma unroll 8
    for (int c = lane; c < hidden; c += 32) {
        value = fmaf(bf16_bits_to_float(x_row[c]), bf16_bits_to_float(__ldg(w_row + c)), value);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) value += __shfl_down_sync(0xffffffffU, value, off);
    return __shfl_sync(0xffffffffU, value, 0);
}

constexpr int kRepairWarps = 4;

// CHUNKS = hidden / 32 > 0: the lane's columns of the token row (l, l+32, ...) stay in registers and the candidates' router
// rows are read in chain order (row_norm) two at a time: ten 16-byte loads a row, two independent chains, three
// instructions per column of a pair's row and no shared memory.  Rows brought into shared memory as they are cost a 2-byte
// read, a shift and an fmaf per column of one dependent chain, and three blocks of four warps per SM (124 us at 16,384
// tokens, 38 at 4,096).  CHUNKS = 0: any hidden size, token row in shared memory, router rows read in place.
// WPT (warps per token) = 1: a warp does everything for its token, four tokens per block - the form for thousands of
// tokens.  WPT = 8: one token per block; the eight warps each build the candidate list (the same list) and then share
// the candidates' exact logits out among themselves, warp 0 finishes - a few hundred tokens would otherwise leave
// most SMs idle while every warp walks eight 2560-step chains one after the other.
// `partials` (splits > 1): the approximate logits arrive as `splits` slices of partial sums ([splits][rows][256]).
template <int CHUNKS, int WPT>
__global__ void __launch_bounds__((WPT > 1 ? WPT : kRepairWarps) * 32) route_repair_kernel(
    const std::uint16_t* __restrict__ x, const std::uint16_t* __restrict__ w, const float* __restrict__ bias,
    const float* __restrict__ w_norms, float* __restrict__ logits, std::int32_t* __restrict__ ids,
    float* __restrict__ weights, int rows, int hidden, float routed_scale, int* __restrict__ stats,
    const float* __restrict__ partials, int splits, const std::uint16_t* __restrict__ w_chains) {
    extern __shared__ __align__(16) std::uint16_t repair_smem[];
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kWarps = WPT > 1 ? WPT : kRepairWarps;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int token = WPT > 1 ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) * kRepairWarps + warp;
    if (token >= rows) return;                     // WPT > 1: the grid is exactly `rows` blocks
    // per warp: [CHUNKS == 0: the token row], then 256 exact logits, then the candidate list
    constexpr int kRowSlots = CHUNKS > 0 ? 0 : 1;
    std::uint16_t* x_row = repair_smem + static_cast<std::size_t>(warp) * kRowSlots * hidden;
    std::uint8_t* tail = reinterpret_cast<std::uint8_t*>(repair_smem + static_cast<std::size_t>(kWarps) * kRowSlots * hidden);
    float* exact_row = reinterpret_cast<float*>(tail) + (WPT > 1 ? 0 : warp) * kExperts;      // WPT > 1: one row per block
    std::uint16_t* cand = reinterpret_cast<std::uint16_t*>(tail + kWarps * kExperts * 4) + warp * kExperts;
    float xr[CHUNKS > 0 ? CHUNKS : 1];
    float square = 0.0F;
    if constexpr (CHUNKS > 0) {
        const std::uint16_t* xg = x + static_cast<std::size_t>(token) * hidden + lane;
#pragma unroll
        for (int j = 0; j < CHUNKS; ++j) xr[j] = bf16_bits_to_float(__ldg(xg + 32 * j));
#pragma unroll
        for (int j = 0; j < CHUNKS; ++j) square = fmaf(xr[j], xr[j], square);
    } else {
        for (int v = lane; v < hidden / 8; v += 32) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(x + static_cast<std::size_t>(token) * hidden) + v);
            reinterpret_cast<uint4*>(x_row)[v] = q;
            const std::uint32_t words[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float lo = __uint_as_float(words[k] << 16), hi = __uint_as_float(words[k] & 0xffff0000U);
                square = fmaf(lo, lo, square);
                square = fmaf(hi, hi, square);
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) square += __shfl_xor_sync(0xffffffffU, square, off);
    const float x_norm = sqrtf(square) * 1.0001F;
    __syncwarp();

    float* lg = logits + static_cast<std::size_t>(token) * kExperts;
    float approx[8], score[8];
    bool finite = true;
    if (splits > 1) {
        // all loads of the slices are issued before the first sum: one round trip, not one per slice
        float part[kRouterSplits][8];
#pragma unroll
        for (int z = 0; z < kRouterSplits; ++z) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                part[z][i] = z < splits ? __ldg(partials + (static_cast<std::size_t>(z) * rows + token) * kExperts + lane + 32 * i) : 0.0F;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float sum = part[0][i];
#pragma unroll
            for (int z = 1; z < kRouterSplits; ++z) sum += part[z][i];
            approx[i] = sum;
            if (WPT == 1 || warp == 0) lg[lane + 32 * i] = sum;           // the logits buffer holds the approximate values
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) approx[i] = lg[lane + 32 * i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = lane + 32 * i;
        finite = finite && (fabsf(approx[i]) <= 3.0e38F);
        score[i] = 1.0F / (1.0F + expf(-approx[i])) + bias[e];
    }
    finite = __all_sync(0xffffffffU, finite);
    // approximate 8th best corrected score: eight rounds of (remove the current maximum), value only
    float eighth = 0.0F;
    {
        float work[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) work[i] = score[i];
#pragma unroll 1
        for (int round = 0; round < 8; ++round) {
            float best = work[0];
            int at = 0;
#pragma unroll
            for (int i = 1; i < 8; ++i) {
                if (work[i] > best) { best = work[i]; at = i; }
            }
            const std::uint32_t bits = __float_as_uint(best);
            const std::uint32_t key = bits & 0x80000000U ? ~bits : bits | 0x80000000U;
            const std::uint32_t top = __reduce_max_sync(0xffffffffU, key);
            const unsigned holders = __ballot_sync(0xffffffffU, key == top);
            if (lane == __ffs(holders) - 1) {                 // one holder gives its maximum up
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i == at) work[i] = -3.0e38F;
                }
            }
            const std::uint32_t top_bits = top & 0x80000000U ? top & 0x7fffffffU : ~top;
            eighth = __uint_as_float(top_bits);
        }
    }
    // candidates: approximate score within 2 delta of the approximate 8th
    unsigned member[8];
    int candidates = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = lane + 32 * i;
        const float delta = 0.25F * kLogitBound * x_norm * w_norms[e] + 4.0e-6F;
        member[i] = __ballot_sync(0xffffffffU, score[i] >= eighth - 2.0F * delta);
        candidates += __popc(member[i]);
    }
    // (fewer than eight: a NaN in the bias upset the 8th best, or fewer than eight experts are not masked by -infinity)
    const bool whole_row = !finite || candidates > kMaxCandidates || candidates < kTop;
    if (whole_row) {
#pragma unroll
        for (int i = 0; i < 8; ++i) member[i] = 0xffffffffU;
    }
    // exact logits of the candidates (or of the whole row), into the logits buffer and into this warp's row
    const float not_recomputed = __uint_as_float(0x7fc00000U);        // a NaN is picked behind every number
    if constexpr (WPT > 1) {
        for (int e = threadIdx.x; e < kExperts; e += WPT * 32) exact_row[e] = not_recomputed;
        __syncthreads();                               // before any warp stores a result into the shared row
    } else {
        for (int e = lane; e < kExperts; e += 32) exact_row[e] = not_recomputed;
    }
    int n_cand = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if ((member[i] >> lane) & 1U) cand[n_cand + __popc(member[i] & ((1U << lane) - 1U))] = static_cast<std::uint16_t>(lane + 32 * i);
        n_cand += __popc(member[i]);
    }
    __syncwarp();
    // this warp's share of the candidates: all of them (WPT = 1) or every WPT-th, starting with its own number
    const int first = WPT > 1 ? warp : 0;
    constexpr int kStep = WPT > 1 ? WPT : 1;
    const int n_mine = n_cand > first ? (n_cand - first + kStep - 1) / kStep : 0;
    if constexpr (CHUNKS > 0) {
#pragma unroll 1
        for (int i = 0; i < n_mine; i += 2) {
            const int ea = cand[first + i * kStep];
            const int eb = i + 1 < n_mine ? cand[first + (i + 1) * kStep] : ea;
            const uint4* wa = reinterpret_cast<const uint4*>(w_chains + static_cast<std::size_t>(ea) * hidden) + lane;
            const uint4* wb = reinterpret_cast<const uint4*>(w_chains + static_cast<std::size_t>(eb) * hidden) + lane;
            float va = 0.0F, vb = 0.0F;
#pragma unroll
            for (int h = 0; h < 2; ++h) {                         // half a row of both in flight
                uint4 qa[CHUNKS / 16], qb[CHUNKS / 16];
#pragma unroll
                for (int c = 0; c < CHUNKS / 16; ++c) {
                    qa[c] = __ldg(wa + 32 * (h * (CHUNKS / 16) + c));
                    qb[c] = __ldg(wb + 32 * (h * (CHUNKS / 16) + c));
                }
#pragma unroll
                for (int c = 0; c < CHUNKS / 16; ++c) {
                    const std::uint32_t ua[4] = {qa[c].x, qa[c].y, qa[c].z, qa[c].w};
                    const std::uint32_t ub[4] = {qb[c].x, qb[c].y, qb[c].z, qb[c].w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int j = 8 * (h * (CHUNKS / 16) + c) + 2 * k;
                        va = fmaf(xr[j], __uint_as_float(ua[k] << 16), va);
                        vb = fmaf(xr[j], __uint_as_float(ub[k] << 16), vb);
                        va = fmaf(xr[j + 1], __uint_as_float(ua[k] & 0xffff0000U), va);
                        vb = fmaf(xr[j + 1], __uint_as_float(ub[k] & 0xffff0000U), vb);
                    }
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                va += __shfl_down_sync(0xffffffffU, va, off);
                vb += __shfl_down_sync(0xffffffffU, vb, off);
            }
            if (lane == 0) {
                exact_row[ea] = va;
                lg[ea] = va;
                exact_row[eb] = vb;
                lg[eb] = vb;
            }
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < n_mine; ++i) {
            const int e = cand[first + i * kStep];
            const float value = exact_logit(x_row, w + static_cast<std::size_t>(e) * hidden, hidden, lane);
            if (lane == 0) {
                exact_row[e] = value;
                lg[e] = value;
            }
        }
    }
    if constexpr (WPT > 1) {
        __syncthreads();                                        // every warp's results are in the block's row
        if (warp != 0) return;
    }
    __syncwarp();
    if (lane == 0 && stats != nullptr) {
        atomicAdd(stats + 0, whole_row ? kExperts : candidates);
        if (whole_row) atomicAdd(stats + 1, 1);
    }
    // The reference's top-8 over the exact values.  (A selection of its own that gave taken, NaN and left-out experts one and
    // the same key chose expert 0 again and again once fewer than eight scores were numbers.)
    warp_top8(exact_row, bias, ids + static_cast<std::size_t>(token) * kTop, weights + static_cast<std::size_t>(token) * kTop,
              routed_scale);
}

}  // namespace

// Below this the fused decode kernel serves the block (up to 8 rows); the exact-order logits kernels took 50 µs at
// 9 - 31 rows where this router takes 20.
int router_fast_min_rows() { return 9; }

cudaError_t launch_router_fast(p92b_plan* plan, const std::uint16_t* x, const std::uint16_t* router_w, const float* bias,
                               int rows, float routed_scale, cudaStream_t stream, bool pdl) {
    static const bool disabled = std::getenv("P92B_EXACT_LOGITS") != nullptr;
    const int hidden = plan->hidden;
    if (disabled || rows < router_fast_min_rows() || hidden % 64 != 0 || hidden > 8192 ||
        (reinterpret_cast<std::uintptr_t>(x) & 15U) != 0U || (reinterpret_cast<std::uintptr_t>(router_w) & 15U) != 0U) {
        return cudaErrorNotSupported;
    }
    CUtensorMap map_x, map_w;
    cudaError_t st = make_operand_map(&map_x, x, static_cast<std::size_t>(rows), static_cast<std::size_t>(hidden) * 2, kTokTile);
    // the expert tile that brings the fewest bytes into the busiest SM
    const int token_tiles = (rows + kTokTile - 1) / kTokTile;
    int expert_tile = 64;
    int least = 0;
    for (int n = 64; n <= 256; n *= 2) {
        const int cost = (token_tiles * (kExperts / n) + plan->sm_count - 1) / plan->sm_count * (kStageA + n * kKBytes);
        if (least == 0 || cost < least) { least = cost; expert_tile = n; }
    }
    if (st == cudaSuccess) st = make_operand_map(&map_w, router_w, kExperts, static_cast<std::size_t>(hidden) * 2, expert_tile);
    if (st != cudaSuccess) return cudaErrorNotSupported;
    if ((st = ensure_dynamic_smem<logits_tc_kernel<64>>(Logits<64>::kSmem)) != cudaSuccess) return st;
    if ((st = ensure_dynamic_smem<logits_tc_kernel<128>>(Logits<128>::kSmem)) != cudaSuccess) return st;
    if ((st = ensure_dynamic_smem<logits_tc_kernel<256>>(Logits<256>::kSmem)) != cudaSuccess) return st;
    const bool in_registers = hidden == 32 * kChunksInRegisters;
    // small batches: K split over blocks of the logits kernel, and a block of eight warps per token in the repair
    const bool may_split = plan->logit_partials != nullptr && plan->max_rows >= rows && std::getenv("P92B_ROUTER_NO_SPLIT") == nullptr;
    const bool small = rows <= kRouterWideRows && may_split;
    const int k_blocks = hidden * 2 / kKBytes;
    // as many slices as fill the chip: 8 up to 512 rows, 4 up to 1,024, 2 up to 2,304 (512 rows, 16 blocks: 12 us)
    const int tiles = token_tiles * (kExperts / expert_tile);
    const int wanted = may_split && rows <= kRouterSplitRows
                           ? std::max(1, std::min({kRouterSplits, plan->sm_count / tiles, kRouterPartialRows / rows})) : 1;
    const int per_split = (k_blocks + wanted - 1) / wanted;
    const int splits = (k_blocks + per_split - 1) / per_split;                    // no empty slice
    constexpr int kWide = 8;
    const int repair_warps = small ? kWide : kRepairWarps;
    const std::size_t repair_smem = static_cast<std::size_t>(repair_warps) * (in_registers ? 0 : hidden) * 2 +
                                    static_cast<std::size_t>(repair_warps) * kExperts * (4 + 2);
    if (small) {
        st = in_registers ? ensure_dynamic_smem<route_repair_kernel<80, kWide>>(static_cast<int>(repair_smem))
                          : ensure_dynamic_smem<route_repair_kernel<0, kWide>>(static_cast<int>(repair_smem));
    } else {
        st = in_registers ? ensure_dynamic_smem<route_repair_kernel<80, 1>>(static_cast<int>(repair_smem))
                          : ensure_dynamic_smem<route_repair_kernel<0, 1>>(static_cast<int>(repair_smem));
    }
    if (st != cudaSuccess) return st;
    float* norms = plan->w_norms;
    float* approx_out = splits > 1 ? plan->logit_partials : plan->logits;
    const auto kernel = expert_tile == 64 ? logits_tc_kernel<64> : expert_tile == 128 ? logits_tc_kernel<128> : logits_tc_kernel<256>;
    const int smem = expert_tile == 64 ? Logits<64>::kSmem : expert_tile == 128 ? Logits<128>::kSmem : Logits<256>::kSmem;
    st = launch_kernel(kernel, dim3(token_tiles, kExperts / expert_tile, splits), dim3(kLogitThreads), smem, stream, pdl, map_x, map_w, approx_out, rows, hidden, plan->status, router_w, norms,
                       in_registers ? plan->w_chains : nullptr);
    if (st != cudaSuccess) return st;
    const float* partials = splits > 1 ? plan->logit_partials : nullptr;
    if (small) {
        st = launch_kernel(in_registers ? route_repair_kernel<80, kWide> : route_repair_kernel<0, kWide>, dim3(rows),
                           dim3(kWide * 32), repair_smem, stream, pdl, x, router_w, bias,
                           static_cast<const float*>(norms), plan->logits, plan->ids, plan->route_weights, rows, hidden,
                           routed_scale, plan->router_stats, partials, splits,
                           static_cast<const std::uint16_t*>(plan->w_chains));
    } else {
        st = launch_kernel(in_registers ? route_repair_kernel<80, 1> : route_repair_kernel<0, 1>,
                           dim3((rows + kRepairWarps - 1) / kRepairWarps), dim3(kRepairWarps * 32), repair_smem, stream, pdl, x,
                           router_w, bias, static_cast<const float*>(norms), plan->logits, plan->ids,
                           plan->route_weights, rows, hidden, routed_scale, plan->router_stats, partials, splits,
                           static_cast<const std::uint16_t*>(plan->w_chains));
    }
    plan->last_launches += 2;
    return st;
}

}  // namespace p92b
