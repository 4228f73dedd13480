// The dense MLP for a few rows (decode, verify step): two kernels that stream the weights through every SM.
//
// With one matrix triple and a few tokens the work is 3 x 9216 x 2560 FP4 weights, 40 MB or 6 us of HBM time, and the
// grouped kernels (expert_tc.cu) leave most of the chip idle on it: 72 gate/up tiles and 20 down tiles on 148 SMs, with a
// list kernel and a one-block quantiser in front (28.3 us for four rows).  Here
//   gate/up  a block owns half a tile, one box of 64 gate and 64 up rows (144 blocks), requests its weights before it
//            waits for the kernel upstream, and quantises the token rows itself while they arrive: the rows are the
//            same 20 KB for every block, so no kernel and no round trip through global memory is needed for them;
//   down     a block owns one 128-row tile and a part of K (20 tiles x 7 parts); its FP32 sums go to scratch and the
//            last block of a tile to arrive adds the parts in their order, so the result does not depend on timing.
// The shared memory of the two together fits one SM: a down block starts beside a gate/up block and has its weights in
// flight when the gate/up rows appear.
#include "p92b_common.cuh"
#include "tc_ptx.cuh"

#include <algorithm>

namespace p92b {

using namespace ptx;

namespace {

constexpr int kRowsMax = 32;                                 // that the kernels are built for
constexpr int kPartsMax = 8;                                 // of K, down product
constexpr int kTile = 128;
constexpr int kKB = 128;                                     // bytes of a K block per row: 256 values
constexpr int kSlab = kChunkScaleBytes;
constexpr int kWeightBytes = kChunkBox + kSlab;              // one box and its scales
constexpr int kTmemColumns = 128;                            // 32 accumulator columns, two buffers of 2 x 16 scale columns
constexpr int kQuantWarps = 16;
constexpr int kGuThreads = 64 + 32 * kQuantWarps;
constexpr int kDownThreads = 64 + 128;

struct DenseParams {
    BankView bank;
    int entry;
    int rows;
    const std::uint16_t* x;      // [rows][hidden]
    std::uint8_t* hq;            // [rows][inter / 2]
    std::uint8_t* hs;            // their scales, 128x4 tiled
    std::uint16_t* out;          // [rows][hidden]
    float* partial;              // [tile][part][row][128]
    unsigned* parts_done;        // [tile], zero between calls
    std::int32_t* status;
    float quant_scale;
    int hidden, inter;
    int parts;
};

// Gate/up: the ring is five stages - 13 MB in flight over the chip - so that a down block fits beside.
struct GateUp {
    static constexpr int kStages = 5;
    static constexpr int kRing = kStages * kWeightBytes;
    static constexpr int kBarriers = 2 * kStages + 2;
    static int smem_bytes(int n, int hidden) {
        return kRing + hidden / 2 * n + hidden / 64 * 512 + kBarriers * 8 + 16 + 1024;
    }
};

template <int N>
struct Down {
    static constexpr int kStages = N == 16 ? 4 : 3;
    static constexpr int kOffSfW = kChunkBox;
    static constexpr int kOffT = kWeightBytes;
    static constexpr int kOffSfT = kOffT + N * kKB;
    static constexpr int kStageBytes = kOffSfT + kSlab;
    static constexpr int kBarriers = 3 * kStages + 1;
    static constexpr int kSmem = kStages * kStageBytes + kBarriers * 8 + 16 + 1024;
};

// One K block: scale factors to TMEM, four products of K = 64.
__device__ __forceinline__ void issue_k_block(std::uint32_t accum, std::uint32_t sf, std::uint32_t w, std::uint32_t w_sf,
                                              std::uint32_t t, std::uint32_t t_sf, std::uint32_t idesc, bool first) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        tc_copy_sf(sf + k * 4, desc_scale_atom(w_sf + k * 512));
        tc_copy_sf(sf + 16 + k * 4, desc_scale_atom(t_sf + k * 512));
    }
    const std::uint64_t a = desc_k_major_sw128(w);
    const std::uint64_t b = desc_k_major_sw128(t);
#pragma unroll
    for (int k = 0; k < 4; ++k) mma_nvf4(accum, a + 2 * k, b + 2 * k, idesc, sf + k * 4, sf + 16 + k * 4, !first || k > 0);
}

template <int N>
__global__ void __launch_bounds__(kGuThreads, 1) dense_gate_up_kernel(const DenseParams p) {
    using C = GateUp;
    extern __shared__ std::uint8_t smem_raw[];
    const std::uint32_t base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    std::uint8_t* const base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const int k_blocks = p.hidden / 256;
    const std::uint32_t tokens = base + C::kRing;                               // [K block][N rows][128 bytes], swizzled
    const std::uint32_t token_sf = tokens + k_blocks * N * kKB;                 // [K block][4 tiles of 512 bytes]
    const std::uint32_t bars = token_sf + k_blocks * kSlab;
    auto weight_bar = [&](int s) { return bars + 8U * s; };
    auto empty_bar = [&](int s) { return bars + 8U * (C::kStages + s); };
    const std::uint32_t token_bar = bars + 8U * (2 * C::kStages);
    const std::uint32_t accum_full = token_bar + 8U;
    volatile std::uint32_t* tmem_slot = reinterpret_cast<volatile std::uint32_t*>(base_ptr + (accum_full + 8U - base));
    volatile std::uint32_t* abort_ptr = tmem_slot + 1;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(weight_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(token_bar, kQuantWarps);
        mbar_init(accum_full, 1);
        *abort_ptr = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(accum_full + 8U, kTmemColumns);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const std::uint32_t tmem = *tmem_slot;
    auto give_up = [&]() {
        *abort_ptr = 1;
        atomicCAS(p.status, kStatusOk, kStatusWaitExpired);
    };

    if (warp == 0) {
        if (elect_one()) {
            // chunk (tile, K block): this block's box and scale slab of it
            const std::uint8_t* chunks = p.bank.g13 +
                (static_cast<std::size_t>(p.entry) * (p.inter / kTile) + (blockIdx.x >> 1)) * k_blocks * kChunkBytes;
            const int half = blockIdx.x & 1;
            int issued = 0;
            for (; issued < k_blocks; ++issued) {
                const int s = issued % C::kStages;
                if (issued >= C::kStages && !mbar_wait(empty_bar(s), (issued / C::kStages - 1) & 1)) { give_up(); break; }
                const std::uint8_t* chunk = chunks + static_cast<std::size_t>(issued) * kChunkBytes;
                mbar_arrive_expect_tx(weight_bar(s), kWeightBytes);
                bulk_load(base + s * kWeightBytes, chunk + half * kChunkBox, kChunkBox, weight_bar(s));
                bulk_load(base + s * kWeightBytes + kChunkBox, chunk + kChunkScaleOffset + half * kSlab, kSlab, weight_bar(s));
            }
            if (*abort_ptr) {       // copies still in flight land before the block ends
                for (int i = max(0, issued - C::kStages); i < issued; ++i) mbar_wait(weight_bar(i % C::kStages), (i / C::kStages) & 1);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr std::uint32_t idesc = idesc_nvf4(kTile, N);
            bool ok = mbar_wait(token_bar, 0);
            for (int kb = 0; kb < k_blocks && ok; ++kb) {
                const int s = kb % C::kStages;
                ok = mbar_wait(weight_bar(s), (kb / C::kStages) & 1);
                if (!ok) break;
                tc_fence_after();
                const std::uint32_t st = base + s * kWeightBytes;
                issue_k_block(tmem, tmem + 32 + (kb & 1) * 32, st, st + kChunkBox, tokens + kb * N * kKB, token_sf + kb * kSlab, idesc, kb == 0);
                tc_commit(empty_bar(s));
            }
            if (ok) tc_commit(accum_full); else give_up();
        }
    } else {
        // token rows -> NVFP4 in the operand's shared-memory image (cuda/nvfp4_ops.cu:818-841; 16-byte pieces XOR-swizzled by
        // the row, scales 128x4 tiled); columns beyond the last row hold whatever was there and nothing reads them
        const float alpha_g = __ldg(p.bank.alpha + p.entry * 3 + 0);
        const float alpha_u = __ldg(p.bank.alpha + p.entry * 3 + 1);
        pdl_wait();
        const int blocks = p.hidden / 16;
#pragma unroll 2
        for (int i = threadIdx.x - 64; i < p.rows * blocks; i += 32 * kQuantWarps) {
            const int row = i / blocks;
            const int b = i - row * blocks;
            const uint4* src = reinterpret_cast<const uint4*>(p.x + static_cast<std::size_t>(row) * p.hidden + b * 16);
            const uint4 lo = __ldg(src), hi = __ldg(src + 1);
            const std::uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            float v[16];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                v[2 * k] = __uint_as_float(words[k] << 16);
                v[2 * k + 1] = __uint_as_float(words[k] & 0xffff0000U);
            }
            std::uint8_t scale_bits;
            const uint2 packed = quantize_block16(v, p.quant_scale, &scale_bits);
            const int kb = b >> 4, piece = (b & 15) >> 1;
            *reinterpret_cast<uint2*>(base_ptr + (tokens - base) + kb * N * kKB + row * kKB + ((piece ^ (row & 7)) * 16) + (b & 1) * 8) = packed;
            base_ptr[(token_sf - base) + kb * kSlab + ((b & 15) >> 2) * 512 + row * 16 + (b & 3)] = scale_bits;
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(token_bar);
        if (warp < 6) {
            const bool done = mbar_wait(accum_full, 0);
            if (!done) give_up();
            tc_fence_after();
            if (__all_sync(0xffffffffU, done)) {
                // lanes 0..15 of a quarter hold the gate sums of 16 intermediate rows, lanes 16..31 their up sums: of a
                // pair of tokens the lower half finishes the even one, the upper half the odd one
                const int quarter = warp & 3;
                const int row = blockIdx.x * (kTile / 2) + quarter * 16 + (lane & 15);
                const int sf_col = row >> 4;
                const bool upper = (lane & 16) != 0;
#pragma unroll 1
                for (int c0 = 0; c0 < p.rows; c0 += 16) {
                    std::uint32_t d[16];
                    tmem_load16(tmem + (static_cast<std::uint32_t>(quarter * 32) << 16) + c0, d);
                    tmem_load_wait();
#pragma unroll
                    for (int n = 0; n < 16; n += 2) {
                        if (c0 + n >= p.rows) break;                              // warp uniform
                        const std::uint32_t got = __shfl_xor_sync(0xffffffffU, upper ? d[n] : d[n + 1], 16);
                        const std::uint32_t g = upper ? got : d[n];
                        const std::uint32_t u = upper ? d[n + 1] : got;
                        const float gv = bf16_bits_to_float(float_to_bf16_bits(__uint_as_float(g) * alpha_g));
                        const float uv = bf16_bits_to_float(float_to_bf16_bits(__uint_as_float(u) * alpha_u));
                        const float h = bf16_bits_to_float(float_to_bf16_bits((gv / (1.0F + expf(-gv))) * uv));
                        const std::uint32_t amax_bits =
                            __reduce_max_sync(upper ? 0xffff0000U : 0x0000ffffU, __float_as_uint(h) & 0x7fffffffU);
                        const __nv_fp8_e4m3 scale(__uint_as_float(amax_bits) * (p.quant_scale / 6.0F));
                        const float decoded = static_cast<float>(scale);
                        const float multiplier = decoded == 0.0F ? 0.0F : p.quant_scale / decoded;
                        const float q = h * multiplier;
                        const float q_next = __shfl_xor_sync(0xffffffffU, q, 1);
                        const int token = c0 + n + (upper ? 1 : 0);
                        if (token >= p.rows) continue;                            // the last round of an odd row count
                        if ((lane & 1) == 0) {
                            p.hq[static_cast<std::size_t>(token) * (p.inter / 2) + (row >> 1)] =
                                static_cast<std::uint8_t>(__nv_fp4x2_e2m1(make_float2(q, q_next)).__x);
                        }
                        if ((lane & 15) == 0) p.hs[static_cast<std::size_t>(sf_col >> 2) * 512 + token * 16 + (sf_col & 3)] = scale.__x;
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemColumns);
    }
}

template <int N>
__global__ void __launch_bounds__(kDownThreads, 1) dense_down_kernel(const __grid_constant__ CUtensorMap map_h, const DenseParams p) {
    using C = Down<N>;
    extern __shared__ std::uint8_t smem_raw[];
    __shared__ unsigned arrived;
    const std::uint32_t base = (smem_u32(smem_raw) + 1023U) & ~1023U;
    const std::uint32_t bars = base + C::kStages * C::kStageBytes;
    auto weight_bar = [&](int s) { return bars + 8U * s; };
    auto token_bar = [&](int s) { return bars + 8U * (C::kStages + s); };
    auto empty_bar = [&](int s) { return bars + 8U * (2 * C::kStages + s); };
    const std::uint32_t accum_full = bars + 8U * (3 * C::kStages);
    volatile std::uint32_t* tmem_slot = reinterpret_cast<volatile std::uint32_t*>(smem_raw + (accum_full + 8U - smem_u32(smem_raw)));
    volatile std::uint32_t* abort_ptr = tmem_slot + 1;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int k_blocks = p.inter / 256;
    const int tile = blockIdx.x / p.parts;
    const int part = blockIdx.x - tile * p.parts;
    const int first = part * k_blocks / p.parts;
    const int count = (part + 1) * k_blocks / p.parts - first;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(weight_bar(s), 1);
            mbar_init(token_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(accum_full, 1);
        *abort_ptr = 0;
        fence_mbar_init();
        prefetch_tensormap(&map_h);
    }
    if (warp == 1) {
        tmem_alloc(accum_full + 8U, kTmemColumns);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const std::uint32_t tmem = *tmem_slot;
    auto give_up = [&]() {
        *abort_ptr = 1;
        atomicCAS(p.status, kStatusOk, kStatusWaitExpired);
    };

    if (warp == 0) {
        if (elect_one()) {
            const std::uint8_t* chunks = p.bank.g2 +
                (static_cast<std::size_t>(p.entry) * (p.hidden / kTile) + tile) * (k_blocks / 2) * kChunkBytes;
            auto load_weights = [&](int i) {
                const int s = i % C::kStages, kb = first + i;
                const std::uint8_t* chunk = chunks + static_cast<std::size_t>(kb >> 1) * kChunkBytes;
                mbar_arrive_expect_tx(weight_bar(s), kWeightBytes);
                bulk_load(base + s * C::kStageBytes, chunk + (kb & 1) * kChunkBox, kChunkBox, weight_bar(s));
                bulk_load(base + s * C::kStageBytes + C::kOffSfW, chunk + kChunkScaleOffset + (kb & 1) * kSlab, kSlab, weight_bar(s));
            };
            auto load_tokens = [&](int i) {
                const int s = i % C::kStages, kb = first + i;
                mbar_arrive_expect_tx(token_bar(s), N * kKB + kSlab);
                tma_load_2d(base + s * C::kStageBytes + C::kOffT, &map_h, token_bar(s), kb * kKB, 0);
                bulk_load(base + s * C::kStageBytes + C::kOffSfT, p.hs + static_cast<std::size_t>(kb) * kSlab, kSlab, token_bar(s));
            };
            // the weights do not depend on the kernel upstream, the SwiGLU rows do
            const int ahead = min(C::kStages, count);
            for (int i = 0; i < ahead; ++i) load_weights(i);
            pdl_wait();
            for (int i = 0; i < ahead; ++i) load_tokens(i);
            int issued = ahead;
            for (; issued < count; ++issued) {
                if (!mbar_wait(empty_bar(issued % C::kStages), (issued / C::kStages - 1) & 1)) { give_up(); break; }
                load_weights(issued);
                load_tokens(issued);
            }
            if (*abort_ptr) {       // copies still in flight land before the block ends
                for (int i = max(0, issued - C::kStages); i < issued; ++i) {
                    mbar_wait(weight_bar(i % C::kStages), (i / C::kStages) & 1);
                    mbar_wait(token_bar(i % C::kStages), (i / C::kStages) & 1);
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr std::uint32_t idesc = idesc_nvf4(kTile, N);
            bool ok = true;
            for (int i = 0; i < count && ok; ++i) {
                const int s = i % C::kStages;
                ok = mbar_wait(weight_bar(s), (i / C::kStages) & 1) && mbar_wait(token_bar(s), (i / C::kStages) & 1);
                if (!ok) break;
                tc_fence_after();
                const std::uint32_t st = base + s * C::kStageBytes;
                issue_k_block(tmem, tmem + 32 + (i & 1) * 32, st, st + C::kOffSfW, st + C::kOffT, st + C::kOffSfT, idesc, i == 0);
                tc_commit(empty_bar(s));
            }
            if (ok) tc_commit(accum_full); else give_up();
        }
    } else {
        const float alpha = __ldg(p.bank.alpha + p.entry * 3 + 2);
        const bool done = mbar_wait(accum_full, 0);
        if (!done) give_up();
        tc_fence_after();
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                     // of the tile
        std::uint16_t* out = p.out + static_cast<std::size_t>(tile) * kTile + row;
        float* mine = p.partial + (static_cast<std::size_t>(tile) * p.parts + part) * p.rows * kTile + row;
        if (__all_sync(0xffffffffU, done)) {
#pragma unroll 1
            for (int c0 = 0; c0 < p.rows; c0 += 16) {
                std::uint32_t d[16];
                tmem_load16(tmem + (static_cast<std::uint32_t>(quarter * 32) << 16) + c0, d);
                tmem_load_wait();
#pragma unroll
                for (int n = 0; n < 16; ++n) {
                    if (c0 + n >= p.rows) break;
                    if (p.parts == 1) out[static_cast<std::size_t>(c0 + n) * p.hidden] = float_to_bf16_bits(__uint_as_float(d[n]) * alpha);
                    else __stcg(mine + (c0 + n) * kTile, __uint_as_float(d[n]));
                }
            }
        }
        if (p.parts > 1) {
            // every block counts, also one that gave up: the counter has to be back at zero for the next call
            __threadfence();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (threadIdx.x == 64) arrived = atomicInc(p.parts_done + tile, static_cast<unsigned>(p.parts - 1));
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (arrived == static_cast<unsigned>(p.parts - 1)) {
                __threadfence();
                const float* all = p.partial + static_cast<std::size_t>(tile) * p.parts * p.rows * kTile + row;
#pragma unroll 4
                for (int n = 0; n < p.rows; ++n) {
                    // all requests before the first sum: a loop over the parts pays a round trip to the L2 for each
                    float part_sum[kPartsMax];
#pragma unroll
                    for (int q = 0; q < kPartsMax; ++q) {
                        part_sum[q] = q < p.parts ? __ldcg(all + (static_cast<std::size_t>(q) * p.rows + n) * kTile) : 0.0F;
                    }
                    float sum = part_sum[0];
#pragma unroll
                    for (int q = 1; q < kPartsMax; ++q) sum = q < p.parts ? sum + part_sum[q] : sum;
                    out[static_cast<std::size_t>(n) * p.hidden] = float_to_bf16_bits(sum * alpha);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemColumns);
    }
}

template <int N>
cudaError_t launch_both(const p92b_plan* plan, const DenseParams& p, cudaStream_t stream, bool pdl) {
    const int gu_smem = GateUp::smem_bytes(N, p.hidden);
    if (cudaError_t st = ensure_dynamic_smem<dense_gate_up_kernel<N>>(227 * 1024); st != cudaSuccess) return st;
    if (cudaError_t st = ensure_dynamic_smem<dense_down_kernel<N>>(Down<N>::kSmem); st != cudaSuccess) return st;
    const cudaError_t st = launch_kernel(dense_gate_up_kernel<N>, dim3(p.inter / (kTile / 2)), dim3(kGuThreads), gu_smem, stream, pdl, p);
    if (st != cudaSuccess) return st;
    return launch_kernel(dense_down_kernel<N>, dim3(p.hidden / kTile * p.parts), dim3(kDownThreads), Down<N>::kSmem, stream, pdl,
                         plan->map_h[N == 16 ? 0 : 1], p);
}

}  // namespace

// The token rows of a block have to fit its shared memory (hidden 4,096 at most), and the rows be few: quantising in every
// block and adding up the parts cost 0.5 to 1 us per row, while the grouped kernels (expert_tc.cu) take nearly the same time
// from 1 to 32 rows.  What those lose, idle SMs, grows with the intermediate size - until the blocks here need a second round.
// Us a layer, few rows / grouped, at the last row count for the former and the first for the latter (hidden x intermediate):
// 2560 x 9216: 18 rows 23.9 / 24.1, 19 rows 24.8 / 24.2; 2048 x 8192: 17 rows 21.6 / 21.6, 18 rows 22.1 / 21.7;
// 1024 x 4096: 13 rows 15.5 / 16.4, 15 rows 16.9 / 16.5; 4096 x 4096: 13 rows 20.2 / 20.4, 14 rows 21.2 / 20.5;
// 2560 x 1024: 10 rows 14.4 / 14.8, 11 rows 15.0 / 14.8; 512 x 1536: 10 rows 12.2 / 13.2, 11 rows 13.3 / 13.2;
// 4096 x 14336, two rounds: 10 rows 35.1 / 35.3, 11 rows 36.1 / 35.4.
bool dense_few_rows_applies(const p92b_plan* plan, int rows) {
    const bool one_round = plan->intermediate / (kTile / 2) <= plan->sm_count;
    const int most = one_round ? std::min(kRowsMax, 9 + plan->intermediate / 1024) : 10;
    return rows <= most && plan->hidden <= 4096 && plan->hidden % 256 == 0 && plan->intermediate % 512 == 0;
}

cudaError_t launch_dense_few_rows(p92b_plan* plan, const p92b_bank* bank, const std::uint16_t* x, std::uint16_t* out, int rows,
                                  cudaStream_t stream, bool pdl) {
    DenseParams p {};
    p.bank = bank->view;
    p.entry = bank->view.local_experts;
    p.rows = rows;
    p.x = x;
    p.hq = plan->hq_pp;
    p.hs = plan->hs_sw;
    p.out = out;
    p.parts_done = plan->dense_parts_done;
    p.status = plan->status;
    p.quant_scale = 1.0F;
    p.hidden = plan->hidden;
    p.inter = plan->intermediate;
    // parts of K: as many blocks as there are SMs (20 tiles: 7 parts), at least one K block each.  The sums lie in the
    // grouped kernels' output rows, which this call does not use: (257 * 127 or fewer, at least 1,152) rows x hidden
    // BF16 values hold 8 parts x 32 rows x hidden FP32 values.
    p.parts = std::max(1, std::min({kPartsMax, plan->sm_count / (plan->hidden / kTile), plan->intermediate / 256}));
    p.partial = reinterpret_cast<float*>(plan->mixed_pp);
    if (static_cast<std::size_t>(p.parts) * rows * 4 > plan->pp_rows * 2) return cudaErrorInvalidValue;
    plan->last_launches += 2;
    return rows <= 16 ? launch_both<16>(plan, p, stream, pdl) : launch_both<32>(plan, p, stream, pdl);
}

}  // namespace p92b
