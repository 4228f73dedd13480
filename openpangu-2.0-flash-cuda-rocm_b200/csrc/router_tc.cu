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
//   2. route_repair_chains_kernel (route_repair_kernel for hidden sizes other than 2,560)   eight, four or one warp per token
//                            by batch: corrected scores from the approximate logits, the approximate 8th best, the
//                            candidate set = every expert whose exact score may be among the eight best, the
//                            candidates' logits recomputed in the reference's exact order, and the reference's
//                            top-8 (cuda/nvfp4_ops.cu:357-433: higher corrected score first, ties to the lower id,
//                            weights from the uncorrected sigmoid, renormalised) taken over the exact values.
//
// Why that is exact.  Let delta_e bound |approximate - exact| of expert e's corrected score, a8 be the approximate 8th best
// and reach the largest delta of the approximately best experts (score >= a8, eight at least).  An expert is left out if its
// approximate score is < a8 - (reach + delta_e); its exact score is then < a8 - reach, while each of the approximately
// best has exact score >= a8 - reach: eight experts beat it, it is not in the exact top-8.  (Its own bound twice is not
// enough: an expert with a small router row was left out for experts with large ones whose exact scores were lower.)
// Hence the exact top-8 is a subset of the candidates, and selecting among exactly recomputed candidates gives the
// reference's ids and weights bit for bit.  delta_e = 0.25 * kLogitBound * ||x_t|| * ||w_e|| + 4e-6: the sigmoid's slope is
// at most 1/4; both the reference chain and the tensor-core sum differ from the true dot product by at most (number of
// sequential roundings) * (2^-24 rounded, 2^-23 cut off) * sum|x_i w_i| <= that * ||x|| ||w||, with hidden / 32 + 5 roundings in
// the reference's order and hidden / 16 steps in the tensor core's; kLogitBound = 2^-14 is 2.5 times their sum at 2,560
// columns and 1.6 times at 4,096 (twice as much is allowed above); 4e-6 covers the fast-math sigmoid's own error on both sides.  A token whose candidate set
// would exceed 24 experts or has fewer than eight, that holds a non-finite logit, or for which a bound is no finite
// number (squares that overflow), has its whole row recomputed exactly instead.
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
constexpr int kChainSteps = 80;                           // hidden / 32
__device__ __forceinline__ void row_norm(const std::uint16_t* __restrict__ w, float* __restrict__ norms,
                                         std::uint16_t* __restrict__ w_chains, int e, int hidden) {
    const int lane = threadIdx.x & 31;
    float s = 0.0F;
    if (w_chains != nullptr) {
        const std::uint16_t* row = w + static_cast<std::size_t>(e) * hidden + lane;
        uint4* to = reinterpret_cast<uint4*>(w_chains + static_cast<std::size_t>(e) * hidden) + lane;
#pragma unroll 5
        for (int c = 0; c < kChainSteps / 8; ++c) {
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
                                                                     std::uint16_t* __restrict__ w_chains,
                                                                     uint4* __restrict__ chunk_counts, int chunk_vectors,
                                                                     uint4* __restrict__ span_counts, int span_vectors) {
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
        // the expert counts that the repair kernel adds to
        const int block_index = static_cast<int>((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
        const int blocks = static_cast<int>(gridDim.x * gridDim.y * gridDim.z);
        for (int i = block_index * 128 + static_cast<int>(threadIdx.x) - 64; i < chunk_vectors + span_vectors; i += blocks * 128) {
            (i < chunk_vectors ? chunk_counts[i] : span_counts[i - chunk_vectors]) = make_uint4(0U, 0U, 0U, 0U);
        }
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

// Approximate logits of one token as a lane holds them: experts lane, lane + 32, ..., lane + 224.  `partials` (splits > 1): they
// arrive as `splits` slices of partial sums ([splits][rows][256]); all loads of the slices are issued before the first sum,
// one round trip and not one per slice, and the sums go to the logits buffer if `store`.
__device__ __forceinline__ void load_approximate(float* __restrict__ lg, const float* __restrict__ partials, int splits, int rows,
                                                 int token, bool store, float (&approx)[8]) {
    const int lane = threadIdx.x & 31;
    if (splits > 1) {
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
            if (store) lg[lane + 32 * i] = sum;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) approx[i] = lg[lane + 32 * i];
    }
}

// The candidates of one token, member[i] a ballot over experts 32 i .. 32 i + 31: approximate corrected score no further below
// the approximate 8th best than the two bounds allow.  All 256 if that cannot decide it (*whole_row): a logit or a bound that is
// no finite number, fewer than eight candidates (a NaN in the bias, or fewer than eight experts that -infinity does not
// mask) or more than a warp takes.
__device__ __forceinline__ int find_candidates(const float (&approx)[8], const float* __restrict__ bias, const float* __restrict__ w_norms,
                                               float x_norm, unsigned (&member)[8], bool* whole_row) {
    const int lane = threadIdx.x & 31;
    bool finite = true;
    float score[8], delta[8];
    std::uint32_t key[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = lane + 32 * i;
        score[i] = 1.0F / (1.0F + expf(-approx[i])) + bias[e];
        delta[i] = 0.25F * kLogitBound * x_norm * w_norms[e] + 4.0e-6F;
        finite = finite && fabsf(approx[i]) <= 3.0e38F && delta[i] <= 3.0e38F;
        const std::uint32_t bits = __float_as_uint(score[i]);
        key[i] = score[i] != score[i] ? 0U : (bits & 0x80000000U ? ~bits : bits | 0x80000000U);
    }
    finite = __all_sync(0xffffffffU, finite);
    // The eighth best: every lane orders its own eight, then eight rounds look at the heads.  Lanes that share a maximum give it
    // up together: the eighth then comes out lower and the candidates are more, never fewer.
#define P92B_ORDER(a, b)                                    \
    {                                                       \
        const std::uint32_t hi = max(key[a], key[b]);       \
        key[b] = min(key[a], key[b]);                       \
        key[a] = hi;                                        \
    }
    P92B_ORDER(0, 1) P92B_ORDER(2, 3) P92B_ORDER(4, 5) P92B_ORDER(6, 7)
    P92B_ORDER(0, 2) P92B_ORDER(1, 3) P92B_ORDER(4, 6) P92B_ORDER(5, 7)
    P92B_ORDER(1, 2) P92B_ORDER(5, 6)
    P92B_ORDER(0, 4) P92B_ORDER(1, 5) P92B_ORDER(2, 6) P92B_ORDER(3, 7)
    P92B_ORDER(2, 4) P92B_ORDER(3, 5)
    P92B_ORDER(1, 2) P92B_ORDER(3, 4) P92B_ORDER(5, 6)
#undef P92B_ORDER
    std::uint32_t top = 0U;
#pragma unroll 2
    for (int round = 0; round < kTop; ++round) {
        top = __reduce_max_sync(0xffffffffU, key[0]);
        if (key[0] == top) {
#pragma unroll
            for (int i = 0; i < 7; ++i) key[i] = key[i + 1];
            key[7] = 0U;
        }
    }
    const float eighth = __uint_as_float(top & 0x80000000U ? top & 0x7fffffffU : ~top);       // image 0: a NaN, nothing is within reach
    float reach = 0.0F;
#pragma unroll
    for (int i = 0; i < 8; ++i) reach = score[i] >= eighth ? fmaxf(reach, delta[i]) : reach;
    reach = __uint_as_float(__reduce_max_sync(0xffffffffU, __float_as_uint(reach)));         // (not negative: ordered as its bits)
    int candidates = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        member[i] = __ballot_sync(0xffffffffU, score[i] >= eighth - (reach + delta[i]));
        candidates += __popc(member[i]);
    }
    *whole_row = !finite || candidates > kMaxCandidates || candidates < kTop;
    if (*whole_row) {
#pragma unroll
        for (int i = 0; i < 8; ++i) member[i] = 0xffffffffU;
        candidates = kExperts;
    }
    return candidates;
}

// The members in order of their ids, as a list in shared memory.
__device__ __forceinline__ void list_candidates(const unsigned (&member)[8], std::uint16_t* cand) {
    const int lane = threadIdx.x & 31;
    int before = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if ((member[i] >> lane) & 1U) cand[before + __popc(member[i] & ((1U << lane) - 1U))] = static_cast<std::uint16_t>(lane + 32 * i);
        before += __popc(member[i]);
    }
    __syncwarp();
}

// The token's experts, which lanes 0..7 have just written, into the counts of its chunk of 32 tokens and of its span of 512
// (null: not wanted).
__device__ __forceinline__ void count_experts(std::int32_t* chunk_hist, std::int32_t* span_hist, int token, const std::int32_t* ids) {
    const int lane = threadIdx.x & 31;
    if (chunk_hist != nullptr && lane < kTop) {
        const int e = *reinterpret_cast<const volatile std::int32_t*>(ids + lane) & (kExperts - 1);
        atomicAdd(chunk_hist + static_cast<std::size_t>(token >> 5) * kExperts + e, 1);
        atomicAdd(span_hist + static_cast<std::size_t>(token >> 9) * kExperts + e, 1);
    }
}

// Logits that were not recomputed: a NaN, picked behind every number.
__device__ __forceinline__ void clear_exact_row(float* exact_row, int first, int threads) {
    for (int e = first; e < kExperts; e += threads) exact_row[e] = __uint_as_float(0x7fc00000U);
}

// Two chains at once: a.x = fmaf(x.x, w.x, a.x) and the same for y, rounded (and denormals flushed) as fmaf in this file.
__device__ __forceinline__ void fma_pair(float2& a, float2 x, float2 w) {
    unsigned long long acc = *reinterpret_cast<unsigned long long*>(&a);
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %0;"
        : "+l"(acc)
        : "l"(*reinterpret_cast<const unsigned long long*>(&x)), "l"(*reinterpret_cast<const unsigned long long*>(&w)));
    a = *reinterpret_cast<float2*>(&acc);
}

// The repair for hidden = 2,560.  The token row lies in shared memory in chain order (row_norm): piece (c, lane) of 16 bytes is
// eight steps of a lane's chain, for the token as for a router row.
// WPT (warps per token) = 1: a warp does everything for its token, four tokens per block - the form for more than a few hundred
// tokens.  The exact logits go four candidates at a time (there are 8.16 on average): four independent chains as two pairs,
// the router rows of the next step in flight, and a tree over the 32 lanes that halves the number of values with every step
// instead of repeating itself per candidate.  It waits for router rows more than it computes, so registers are worth warps:
// with five blocks per SM whole calls of 3,807 and 16,384 rows take 385 and 1,116 us, with eight candidates and four blocks
// 390 and 1,128, with six or seven blocks no less.  (Two candidates at a time from a token row in registers, all 256 exact
// logits in the selection: 96 us at 16,384 tokens, 80 with eight at a time; 15 at 512, now 11; 12 at 64, now 9.6.)
// WPT = 8 or 4: one token per block; its warps bring the row in together, each build the candidate list (the same list) and
// then share the candidates out, one chain at a time; warp 0 finishes.
template <int WPT>
__global__ void __launch_bounds__((WPT > 1 ? WPT : kRepairWarps) * 32, WPT == 8 ? 2 : WPT == 4 ? 4 : 5) route_repair_chains_kernel(
    const std::uint16_t* __restrict__ x, const float* __restrict__ bias, const float* __restrict__ w_norms, float* __restrict__ logits,
    std::int32_t* __restrict__ ids, float* __restrict__ weights, int rows, float routed_scale, int* __restrict__ stats,
    const float* __restrict__ partials, int splits, const std::uint16_t* __restrict__ w_chains, std::int32_t* __restrict__ chunk_hist,
    std::int32_t* __restrict__ span_hist) {
    constexpr int kHidden = 32 * kChainSteps;
    constexpr int kPieces = kChainSteps / 8;                  // of 16 bytes, per lane
    constexpr int kBatch = 4;                                 // candidates at a time
    constexpr int kWarps = WPT > 1 ? WPT : kRepairWarps;
    constexpr int kTokens = WPT > 1 ? 1 : kRepairWarps;             // per block
    __shared__ uint4 x_chains[kTokens][kPieces * 32];
    __shared__ float exact_rows[kTokens][kExperts];
    __shared__ std::uint16_t cand_lists[kWarps][kExperts];
    __shared__ float square_sums[kWarps];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int token = WPT > 1 ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) * kRepairWarps + warp;
    if (token >= rows) return;                     // WPT > 1: the grid is exactly `rows` blocks
    uint4* const x_row = x_chains[WPT > 1 ? 0 : warp];
    float* const exact_row = exact_rows[WPT > 1 ? 0 : warp];
    std::uint16_t* const cand = cand_lists[warp];
    float* const lg = logits + static_cast<std::size_t>(token) * kExperts;
    std::int32_t* const my_ids = ids + static_cast<std::size_t>(token) * kTop;
    float* const my_weights = weights + static_cast<std::size_t>(token) * kTop;
    float approx[8];
    float square = 0.0F;
    {
        const std::uint16_t* xg = x + static_cast<std::size_t>(token) * kHidden + lane;
#pragma unroll 5
        for (int c = WPT > 1 ? warp : 0; c < kPieces; c += WPT > 1 ? WPT : 1) {
            std::uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __ldg(xg + 32 * (8 * c + i));
#pragma unroll
            for (int i = 0; i < 8; ++i) square = fmaf(__uint_as_float(v[i] << 16), __uint_as_float(v[i] << 16), square);
            x_row[32 * c + lane] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
        }
    }
    load_approximate(lg, partials, splits, rows, token, WPT == 1 || warp == 0, approx);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) square += __shfl_xor_sync(0xffffffffU, square, off);
    if constexpr (WPT > 1) {
        if (lane == 0) square_sums[warp] = square;
        __syncthreads();                            // the row and its parts of the norm
        square = 0.0F;
#pragma unroll
        for (int v = 0; v < WPT; ++v) square += square_sums[v];
    }
    const float x_norm = sqrtf(square) * 1.0001F;
    unsigned member[8];
    bool whole_row;
    const int n_cand = find_candidates(approx, bias, w_norms, x_norm, member, &whole_row);
    list_candidates(member, cand);

    const uint4* const w_lane = reinterpret_cast<const uint4*>(w_chains) + lane;
    float mine = 0.0F;                              // lane i < n_cand <= 32: exact logit of candidate i
    if constexpr (WPT > 1) {
#pragma unroll 1
        for (int i = warp; i < n_cand; i += WPT) {
            const int e = cand[i];
            const uint4* w = w_lane + e * (kPieces * 32);
            uint4 q[kPieces];
#pragma unroll
            for (int c = 0; c < kPieces; ++c) q[c] = __ldg(w + 32 * c);
            float value = 0.0F;
#pragma unroll
            for (int c = 0; c < kPieces; ++c) {
                const uint4 xq = x_row[32 * c + lane];
                const std::uint32_t xs[4] = {xq.x, xq.y, xq.z, xq.w}, ws[4] = {q[c].x, q[c].y, q[c].z, q[c].w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    value = fmaf(__uint_as_float(xs[k] << 16), __uint_as_float(ws[k] << 16), value);
                    value = fmaf(__uint_as_float(xs[k] & 0xffff0000U), __uint_as_float(ws[k] & 0xffff0000U), value);
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) value += __shfl_down_sync(0xffffffffU, value, off);
            if (lane == 0) {
                exact_row[e] = value;
                lg[e] = value;
            }
        }
        __syncthreads();                                        // every warp's results are in the block's row
        if (warp != 0) return;
        if (lane < n_cand && !whole_row) mine = exact_row[cand[lane]];
    } else {
#pragma unroll 1
        for (int first = 0; first < n_cand; first += kBatch) {
            int at[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) at[k] = cand[min(first + k, n_cand - 1)] * (kPieces * 32);
            float2 acc[kBatch / 2];
#pragma unroll
            for (int m = 0; m < kBatch / 2; ++m) acc[m] = make_float2(0.0F, 0.0F);
            // a step of eight columns per lane; two sets of registers, the loads of one under way while the other is used
            uint4 even[kBatch], odd[kBatch];
            auto request = [&](uint4 (&q)[kBatch], int c) {
#pragma unroll
                for (int k = 0; k < kBatch; ++k) q[k] = __ldg(w_lane + at[k] + 32 * c);
            };
            auto add = [&](const uint4 (&q)[kBatch], int c) {
                const uint4 xq = x_row[32 * c + lane];
                const std::uint32_t xs[4] = {xq.x, xq.y, xq.z, xq.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float lo = __uint_as_float(xs[k] << 16), hi = __uint_as_float(xs[k] & 0xffff0000U);
#pragma unroll
                    for (int m = 0; m < kBatch / 2; ++m) {
                        const std::uint32_t wa = k == 0 ? q[2 * m].x : k == 1 ? q[2 * m].y : k == 2 ? q[2 * m].z : q[2 * m].w;
                        const std::uint32_t wb = k == 0 ? q[2 * m + 1].x : k == 1 ? q[2 * m + 1].y : k == 2 ? q[2 * m + 1].z : q[2 * m + 1].w;
                        fma_pair(acc[m], make_float2(lo, lo), make_float2(__uint_as_float(wa << 16), __uint_as_float(wb << 16)));
                        fma_pair(acc[m], make_float2(hi, hi), make_float2(__uint_as_float(wa & 0xffff0000U), __uint_as_float(wb & 0xffff0000U)));
                    }
                }
            };
            static_assert(kPieces % 2 == 0, "steps in pairs");
            request(even, 0);
#pragma unroll 1
            for (int c = 0; c < kPieces; c += 2) {
                request(odd, c + 1);
                add(even, c);
                if (c + 2 < kPieces) request(even, c + 2);
                add(odd, c + 1);
            }
            // The reference's tree over the 32 chains (lane l takes lane l + 16's sum, then l + 8's, ...), for the batch at once: a
            // lane hands half of its values to its partner and goes on with the other half, so that after the steps of 16 and 8
            // lanes it is left with candidate lane / 8.  An addition's two operands are the tree's, in either order.
            float v[kBatch] = {acc[0].x, acc[0].y, acc[1].x, acc[1].y};
#pragma unroll
            for (int half = kBatch / 2; half >= 1; half >>= 1) {
                const int off = half * (32 / kBatch);
                const bool upper = (lane & off) != 0;
#pragma unroll
                for (int m = 0; m < half; ++m) {
                    const float got = __shfl_xor_sync(0xffffffffU, upper ? v[m] : v[m + half], off);
                    v[m] = (upper ? v[m + half] : v[m]) + got;
                }
            }
            float value = v[0];
#pragma unroll
            for (int off = 16 / kBatch; off > 0; off >>= 1) value += __shfl_xor_sync(0xffffffffU, value, off);
            const int k = first + lane / (32 / kBatch);
            if (lane % (32 / kBatch) == 0 && k < n_cand) {
                exact_row[cand[k]] = value;
                lg[cand[k]] = value;
            }
            const float of_mine = __shfl_sync(0xffffffffU, value, lane % kBatch * (32 / kBatch));
            if (lane >= first && lane < first + kBatch) mine = of_mine;
        }
        __syncwarp();
    }
    if (lane == 0 && stats != nullptr) {
        atomicAdd(stats + 0, n_cand);
        if (whole_row) atomicAdd(stats + 1, 1);
    }
    // The reference's top-8 over the exact values.
    if (whole_row) {
        warp_top8(exact_row, bias, my_ids, my_weights, routed_scale);
        count_experts(chunk_hist, span_hist, token, my_ids);
        return;
    }
    // One candidate per lane, words as in warp_top8: nine rounds, a lane gives its word up when it is the maximum.
    const int my_e = lane < n_cand ? cand[lane] : 0;
    std::uint32_t word = 0U;
    if (lane < n_cand) {
        const float corrected = 1.0F / (1.0F + expf(-mine)) + bias[my_e];
        const std::uint32_t bits = __float_as_uint(corrected);
        const std::uint32_t image = corrected != corrected ? 0U : (bits & 0x80000000U ? ~bits : bits | 0x80000000U);
        word = (image & 0xffffff00U) | static_cast<std::uint32_t>(kExperts - 1 - my_e);
    }
    std::uint32_t of_slot = 0U;                    // lane k keeps the word of slot k, lane 8 the ninth
#pragma unroll 3
    for (int slot = 0; slot <= kTop; ++slot) {
        const std::uint32_t top = __reduce_max_sync(0xffffffffU, word);
        if (word == top) word = 0U;
        if (lane == slot) of_slot = top;
    }
    if (top8_is_close(of_slot)) {
        clear_exact_row(exact_row, lane, 32);
        __syncwarp();
        if (lane < n_cand) exact_row[my_e] = mine;
        __syncwarp();
        warp_top8_by_id(exact_row, bias, my_ids, my_weights, routed_scale);
    } else {
        warp_top8_write(of_slot, exact_row, my_ids, my_weights, routed_scale);
    }
    count_experts(chunk_hist, span_hist, token, my_ids);
}

// Any other hidden size: the token row in shared memory as it is, router rows read in place, one chain at a time.
template <int WPT>
__global__ void __launch_bounds__((WPT > 1 ? WPT : kRepairWarps) * 32) route_repair_kernel(
    const std::uint16_t* __restrict__ x, const std::uint16_t* __restrict__ w, const float* __restrict__ bias,
    const float* __restrict__ w_norms, float* __restrict__ logits, std::int32_t* __restrict__ ids,
    float* __restrict__ weights, int rows, int hidden, float routed_scale, int* __restrict__ stats,
    const float* __restrict__ partials, int splits, std::int32_t* __restrict__ chunk_hist,
    std::int32_t* __restrict__ span_hist) {
    extern __shared__ __align__(16) std::uint16_t repair_smem[];
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kWarps = WPT > 1 ? WPT : kRepairWarps;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int token = WPT > 1 ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) * kRepairWarps + warp;
    if (token >= rows) return;                     // WPT > 1: the grid is exactly `rows` blocks
    // per warp: the token row, then 256 exact logits, then the candidate list
    std::uint16_t* x_row = repair_smem + static_cast<std::size_t>(warp) * hidden;
    std::uint8_t* tail = reinterpret_cast<std::uint8_t*>(repair_smem + static_cast<std::size_t>(kWarps) * hidden);
    float* exact_row = reinterpret_cast<float*>(tail) + (WPT > 1 ? 0 : warp) * kExperts;      // WPT > 1: one row per block
    std::uint16_t* cand = reinterpret_cast<std::uint16_t*>(tail + kWarps * kExperts * 4) + warp * kExperts;
    float square = 0.0F;
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
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) square += __shfl_xor_sync(0xffffffffU, square, off);
    const float x_norm = sqrtf(square) * (hidden > 4096 ? 2.0002F : 1.0001F);          // (kLogitBound holds up to 4,096 columns)
    __syncwarp();
    float* lg = logits + static_cast<std::size_t>(token) * kExperts;
    float approx[8];
    load_approximate(lg, partials, splits, rows, token, WPT == 1 || warp == 0, approx);
    unsigned member[8];
    bool whole_row;
    const int n_cand = find_candidates(approx, bias, w_norms, x_norm, member, &whole_row);
    list_candidates(member, cand);
    if constexpr (WPT > 1) {
        clear_exact_row(exact_row, threadIdx.x, WPT * 32);
        __syncthreads();                               // before any warp stores a result into the shared row
    } else {
        clear_exact_row(exact_row, lane, 32);
        __syncwarp();
    }
    // this warp's share of the candidates: all of them (WPT = 1) or every WPT-th, starting with its own number
#pragma unroll 1
    for (int i = WPT > 1 ? warp : 0; i < n_cand; i += WPT) {
        const int e = cand[i];
        const float value = exact_logit(x_row, w + static_cast<std::size_t>(e) * hidden, hidden, lane);
        if (lane == 0) {
            exact_row[e] = value;
            lg[e] = value;
        }
    }
    if constexpr (WPT > 1) {
        __syncthreads();                                        // every warp's results are in the block's row
        if (warp != 0) return;
    }
    __syncwarp();
    if (lane == 0 && stats != nullptr) {
        atomicAdd(stats + 0, n_cand);
        if (whole_row) atomicAdd(stats + 1, 1);
    }
    // The reference's top-8 over the exact values.  (A selection of its own that gave taken, NaN and left-out experts one and
    // the same key chose expert 0 again and again once fewer than eight scores were numbers.)
    warp_top8(exact_row, bias, ids + static_cast<std::size_t>(token) * kTop, weights + static_cast<std::size_t>(token) * kTop,
              routed_scale);
    count_experts(chunk_hist, span_hist, token, ids + static_cast<std::size_t>(token) * kTop);
}

}  // namespace

// Below this the fused decode kernel serves the block (up to 8 rows); the exact-order logits kernels took 50 µs at
// 9 - 31 rows where this router takes 20.
int router_fast_min_rows() { return 9; }

cudaError_t launch_router_fast(p92b_plan* plan, const std::uint16_t* x, const std::uint16_t* router_w, const float* bias,
                               int rows, float routed_scale, cudaStream_t stream, bool pdl, bool count_experts) {
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
    const bool chain_order = hidden == 32 * kChainSteps;
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
    const std::size_t repair_smem = chain_order ? 0 : static_cast<std::size_t>(repair_warps) * (hidden * 2 + kExperts * (4 + 2));
    if (!chain_order) {
        st = small ? ensure_dynamic_smem<route_repair_kernel<kWide>>(static_cast<int>(repair_smem))
                   : ensure_dynamic_smem<route_repair_kernel<1>>(static_cast<int>(repair_smem));
        if (st != cudaSuccess) return st;
    }
    float* norms = plan->w_norms;
    float* approx_out = splits > 1 ? plan->logit_partials : plan->logits;
    const auto kernel = expert_tile == 64 ? logits_tc_kernel<64> : expert_tile == 128 ? logits_tc_kernel<128> : logits_tc_kernel<256>;
    const int smem = expert_tile == 64 ? Logits<64>::kSmem : expert_tile == 128 ? Logits<128>::kSmem : Logits<256>::kSmem;
    st = launch_kernel(kernel, dim3(token_tiles, kExperts / expert_tile, splits), dim3(kLogitThreads), smem, stream, pdl, map_x, map_w, approx_out, rows, hidden, plan->status, router_w, norms,
                       chain_order ? plan->w_chains : nullptr, reinterpret_cast<uint4*>(plan->chunk_hist),
                       count_experts ? (rows + 31) / 32 * kExperts / 4 : 0, reinterpret_cast<uint4*>(plan->span_hist),
                       count_experts ? (rows + 511) / 512 * kExperts / 4 : 0);
    if (st != cudaSuccess) return st;
    const float* partials = splits > 1 ? plan->logit_partials : nullptr;
    std::int32_t* chunk_hist = count_experts ? plan->chunk_hist : nullptr;
    // between the two, four warps per token up to what the chip holds at a time
    const bool medium = chain_order && !small && rows <= 4 * plan->sm_count;
    const dim3 repair_grid(small || medium ? rows : (rows + kRepairWarps - 1) / kRepairWarps), repair_block(repair_warps * 32);
    if (chain_order) {
        st = launch_kernel(small ? route_repair_chains_kernel<kWide> : medium ? route_repair_chains_kernel<4> : route_repair_chains_kernel<1>,
                           repair_grid, repair_block, 0, stream, pdl, x, bias, static_cast<const float*>(norms), plan->logits, plan->ids,
                           plan->route_weights, rows, routed_scale, plan->router_stats, partials, splits,
                           static_cast<const std::uint16_t*>(plan->w_chains), chunk_hist, plan->span_hist);
    } else {
        st = launch_kernel(small ? route_repair_kernel<kWide> : route_repair_kernel<1>, repair_grid, repair_block, repair_smem, stream,
                           pdl, x, router_w, bias, static_cast<const float*>(norms), plan->logits, plan->ids, plan->route_weights, rows,
                           hidden, routed_scale, plan->router_stats, partials, splits, chunk_hist, plan->span_hist);
    }
    plan->last_launches += 2;
    return st;
}

}  // namespace p92b
