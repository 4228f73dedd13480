// Router: BF16 logits in the reference's two FP32 summation orders, and the
// sigmoid + correction-bias top-8 with renormalised weights.
//
// Bit-exactness contract.  Expert ids must equal the reference's, so the logits
// reproduce its FP32 fmaf chains and reduction trees value for value:
//   T == 1 (cuda/nvfp4_ops.cu:161-176): thread t of 256 sums columns t, t+256, ...;
//           warp shuffle-down tree; tree over the 8 warp sums (block_sum, :38-51).
//   T  > 1 (cuda/nvfp4_ops.cu:178-207): lane l of a warp sums columns l, l+32, ...;
//           warp shuffle-down tree.
// The score is written as the reference writes it, 1/(1+expf(-x)), and this
// file is compiled with --use_fast_math like the reference (CMakeLists.txt:98)
// so expf and the divisions lower to the same hardware approximations.
// Selection is pure comparison with ties to the lower id, which is order
// independent, so the top-8 itself is free to use a warp-per-token layout.
#include "p92b_common.cuh"

#include <cstdlib>
#include "tc_ptx.cuh"

#include <cfloat>

namespace p92b {

using ptx::pdl_launch_dependents;
using ptx::pdl_wait;

namespace {

// ---- T == 1 order ---------------------------------------------------------
// One block of 256 threads per expert row; thread t owns columns t + 256 j.
// The 5 KB row is one fully coalesced pass (ten 512-byte warp requests).
__global__ void __launch_bounds__(256) logits_gemv_kernel(const std::uint16_t* __restrict__ x,
                                                          const std::uint16_t* __restrict__ w,
                                                          float* __restrict__ out, int rows,
                                                          int columns) {
    const int row = blockIdx.x;
    if (row >= rows) return;
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float warp_sums[8];
    const std::uint16_t* wr = w + static_cast<std::size_t>(row) * columns;
    float value = 0.0F;
    for (int c = threadIdx.x; c < columns; c += 256) {
        value = fmaf(bf16_bits_to_float(x[c]), bf16_bits_to_float(wr[c]), value);
    }
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_down_sync(0xffffffffU, value, offset);
    if (lane == 0) warp_sums[warp] = value;
    __syncthreads();
    if (warp == 0) {
        value = lane < 8 ? warp_sums[lane] : 0.0F;
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_down_sync(0xffffffffU, value, offset);
        if (lane == 0) out[row] = value;
    }
}

// ---- T > 1 order ----------------------------------------------------------
// A warp owns a TE x TT tile of (expert, token) outputs; lane l accumulates the
// columns l, l+32, ... of every output in the tile (the reference's per-lane
// chain), so one pass over K yields TE*TT fmaf per TE+TT shared-memory reads,
// and the final shuffle-down tree is the reference's.  K is staged through
// shared memory in ascending chunks, which keeps each chain's order.
template <int TE, int TT, int WE, int WT>
__global__ void __launch_bounds__(WE* WT * 32) logits_rows_kernel(
    const std::uint16_t* __restrict__ x, const std::uint16_t* __restrict__ w,
    float* __restrict__ out, int batch_rows, int rows, int columns, int kc) {
    constexpr int BE = TE * WE;             // experts per block
    constexpr int BT = TT * WT;             // tokens per block
    constexpr int THREADS = WE * WT * 32;
    extern __shared__ __align__(16) std::uint16_t staged[];
    std::uint16_t* ws = staged;                                 // [BE][kc]
    std::uint16_t* xs = staged + static_cast<std::size_t>(BE) * kc;   // [BT][kc]
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int we = warp % WE;
    const int wt = warp / WE;
    const int e0 = blockIdx.x * BE;
    const int t0 = blockIdx.y * BT;
    const int kc8 = kc / 8;
    float acc[TE][TT];
#pragma unroll
    for (int i = 0; i < TE; ++i)
#pragma unroll
        for (int j = 0; j < TT; ++j) acc[i][j] = 0.0F;

    pdl_wait();                // and no early start for the next kernel, as in the large form below
    for (int k0 = 0; k0 < columns; k0 += kc) {
        if (k0 != 0) __syncthreads();
        // 16-byte coalesced staging; rows beyond the edge are zero filled
        for (int idx = threadIdx.x; idx < BE * kc8; idx += THREADS) {
            const int r = idx / kc8;
            const int c8 = idx - r * kc8;
            uint4 v = make_uint4(0U, 0U, 0U, 0U);
            if (e0 + r < rows) {
                v = *reinterpret_cast<const uint4*>(w + static_cast<std::size_t>(e0 + r) * columns + k0 + c8 * 8);
            }
            *reinterpret_cast<uint4*>(ws + static_cast<std::size_t>(r) * kc + c8 * 8) = v;
        }
        for (int idx = threadIdx.x; idx < BT * kc8; idx += THREADS) {
            const int r = idx / kc8;
            const int c8 = idx - r * kc8;
            uint4 v = make_uint4(0U, 0U, 0U, 0U);
            if (t0 + r < batch_rows) {
                v = *reinterpret_cast<const uint4*>(x + static_cast<std::size_t>(t0 + r) * columns + k0 + c8 * 8);
            }
            *reinterpret_cast<uint4*>(xs + static_cast<std::size_t>(r) * kc + c8 * 8) = v;
        }
        __syncthreads();
#pragma unroll 4
        for (int j = 0; j < kc / 32; ++j) {
            float wv[TE];
            float xv[TT];
#pragma unroll
            for (int i = 0; i < TE; ++i) wv[i] = bf16_bits_to_float(ws[static_cast<std::size_t>(we * TE + i) * kc + j * 32 + lane]);
#pragma unroll
            for (int i = 0; i < TT; ++i) xv[i] = bf16_bits_to_float(xs[static_cast<std::size_t>(wt * TT + i) * kc + j * 32 + lane]);
#pragma unroll
            for (int i = 0; i < TE; ++i)
#pragma unroll
                for (int t = 0; t < TT; ++t) acc[i][t] = fmaf(xv[t], wv[i], acc[i][t]);
        }
    }
#pragma unroll
    for (int i = 0; i < TE; ++i) {
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            float value = acc[i][t];
#pragma unroll
            for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_down_sync(0xffffffffU, value, offset);
            const int e = e0 + we * TE + i;
            const int tok = t0 + wt * TT + t;
            if (lane == 0 && e < rows && tok < batch_rows) out[static_cast<std::size_t>(tok) * rows + e] = value;
        }
    }
}

// ---- T > 1 order, up to eight tokens ----------------------------------------
// A block takes two experts and all tokens, four warps: (expert, half of the tokens).  Both expert rows and the token rows
// arrive by asynchronous 16-byte copies that are all in flight at once; with loads into registers on the way to shared
// memory, 64 blocks took 15.4 us for four tokens.  The chains are the ones above.
template <int TT>
__global__ void __launch_bounds__(128) logits_few_rows_kernel(const std::uint16_t* __restrict__ x, const std::uint16_t* __restrict__ w,
                                                              float* __restrict__ out, int batch_rows, int rows, int columns) {
    extern __shared__ __align__(16) std::uint16_t staged[];            // [2 experts + 2 TT tokens][columns]
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int pieces = columns / 8;
    const int e0 = blockIdx.x * 2;
    pdl_launch_dependents();
    pdl_wait();
    const int staged_rows = 2 + min(batch_rows, 2 * TT);
    for (int r = warp; r < staged_rows; r += 4) {
        const std::uint16_t* src = r < 2 ? w + static_cast<std::size_t>(min(e0 + r, rows - 1)) * columns
                                         : x + static_cast<std::size_t>(r - 2) * columns;
        for (int piece = lane; piece < pieces; piece += 32) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                         ::"r"(static_cast<std::uint32_t>(__cvta_generic_to_shared(staged + static_cast<std::size_t>(r) * columns + piece * 8))),
                         "l"(src + piece * 8) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int e = e0 + (warp & 1);
    const int t0 = (warp >> 1) * TT;
    if (e >= rows || t0 >= batch_rows) return;
    const std::uint16_t* wr = staged + static_cast<std::size_t>(warp & 1) * columns + lane;
    const std::uint16_t* xr = staged + static_cast<std::size_t>(2 + t0) * columns + lane;
    float acc[TT];
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[t] = 0.0F;
#pragma unroll 8
    for (int c = 0; c < columns; c += 32) {
        const float wv = bf16_bits_to_float(wr[c]);
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            // rows beyond the batch were not staged: what lies there goes into sums that nobody reads
            acc[t] = fmaf(bf16_bits_to_float(xr[static_cast<std::size_t>(t) * columns + c]), wv, acc[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < TT; ++t) {
        float value = acc[t];
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_down_sync(0xffffffffU, value, offset);
        if (lane == 0 && t0 + t < batch_rows) out[static_cast<std::size_t>(t0 + t) * rows + e] = value;
    }
}

// ---- T > 1 order, large batches ----------------------------------------------
// Same per-lane chains as above, organised for throughput: a block of four warps computes 16 experts x
// 16 tokens, a warp 8 x 8 of them.  K advances in chunks of 256 columns that sit TRANSPOSED in shared
// memory - element (row, column l + 32 j) at [row][l][j] - so that a lane fetches its eight j-values of
// a row with one 16-byte read.  A chunk arrives by asynchronous 16-byte copies issued a whole chunk ahead
// (no registers; loading into registers instead left the global latency exposed: 274 µs against 230 µs
// at T=4096; one 512-byte bulk copy of the TMA unit per row was slower too: 242 µs against 199 µs), and is
// transposed inside shared memory with 16-byte reads, byte permutes and 8-byte
// stores laid out so that every bank is hit exactly twice per instruction, the minimum for 256 bytes.
// Two buffers of each image, one block synchronisation per chunk.  The fmaf order of every
// chain is still j ascending; the multiply uses the two-wide FP32 fused multiply-add of sm_100, each half
// of which is an ordinary round-to-nearest fmaf.
__device__ __forceinline__ void async_copy16(std::uint32_t dst_smem, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;          // 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst_smem), "l"(src), "r"(bytes) : "memory");
}

template <int MIN_BLOCKS>
__global__ void __launch_bounds__(128, MIN_BLOCKS) logits_rows_large_kernel(const std::uint16_t* __restrict__ x,
                                                                           const std::uint16_t* __restrict__ w,
                                                                           float* __restrict__ out, int batch_rows, int rows,
                                                                           int columns) {
    constexpr int TE = 8, TT = 8, WE = 2, WT = 2, KC = 256;
    constexpr int BE = TE * WE, BT = TT * WT, ROWS = BE + BT;      // 16 expert rows + 16 token rows
    constexpr int ROW_WORDS = 32 * 4 + 4;                           // 512 bytes + 16 bytes of padding
    static_assert(ROWS == 32, "one transposition unit per thread: 32 rows x 2 j-quads x 2 lane halves = 128 threads");
    extern __shared__ __align__(16) std::uint8_t large_smem[];
    std::uint32_t (*raw)[ROWS][ROW_WORDS] = reinterpret_cast<std::uint32_t (*)[ROWS][ROW_WORDS]>(large_smem);
    std::uint32_t (*tile)[ROWS][ROW_WORDS] =
        reinterpret_cast<std::uint32_t (*)[ROWS][ROW_WORDS]>(large_smem + 2 * ROWS * ROW_WORDS * 4);
    // No early start for the next kernel: blocks here are small enough for three to share an SM, so blocks that come in while
    // these compute take the places of idle SMs and the work ends up unevenly spread (128 rows of 4,096 columns, 256 tokens,
    // call after call: 30.5 us with the trigger up front, 21.9 with it behind the products, 18.4 without; 256 rows of 2,560
    // columns: 23.3, 20.5 and 18.0).
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int we = warp % WE, wt = warp / WE;
    const int e0 = blockIdx.x * BE, t0 = blockIdx.y * BT;
    float2 acc[TE][TT / 2];
#pragma unroll
    for (int i = 0; i < TE; ++i)
#pragma unroll
        for (int j = 0; j < TT / 2; ++j) acc[i][j] = make_float2(0.0F, 0.0F);

    // global -> raw image, asynchronously: 32 rows x 32 pieces of 16 bytes, eight per thread, consecutive
    // threads on consecutive pieces of a row
    auto fetch = [&](int k0, int buffer) {
#pragma unroll
        for (int q = 0; q < ROWS * 32 / 128; ++q) {
            const int idx = threadIdx.x + q * 128;
            const int r = idx >> 5, piece = idx & 31;
            const bool is_w = r < BE;
            const int src_row = is_w ? e0 + r : t0 + (r - BE);
            const bool ok = is_w ? src_row < rows : src_row < batch_rows;
            const std::uint16_t* src = (is_w ? w : x) + static_cast<std::size_t>(ok ? src_row : 0) * columns + k0 + piece * 8;
            async_copy16(static_cast<std::uint32_t>(__cvta_generic_to_shared(&raw[buffer][r][piece * 4])), src, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // raw image -> transposed image.  A thread takes, for one row, four j-values (j = 4q .. 4q+3) of sixteen
    // neighbouring lanes: eight 16-byte reads, byte permutes, sixteen 8-byte stores whose lanes are spread
    // over sixteen rows and both j-quads, so every bank is hit exactly twice per instruction.
    const int s_row = (warp >> 1) * 16 + (lane >> 4) * 8 + (lane & 7);
    const int s_q = (lane >> 3) & 1;
    const int s_side = warp & 1;
    auto transpose = [&](int buffer) {
        const uint4* src = reinterpret_cast<const uint4*>(&raw[buffer][s_row][(128 * s_q + 16 * s_side) / 2]);
        std::uint32_t* row = &tile[buffer][s_row][0];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 p0 = src[h], p1 = src[4 + h], p2 = src[8 + h], p3 = src[12 + h];     // j = 4q .. 4q+3: 64 bytes apart
            const std::uint32_t words[4][4] = {{p0.x, p0.y, p0.z, p0.w}, {p1.x, p1.y, p1.z, p1.w},
                                               {p2.x, p2.y, p2.z, p2.w}, {p3.x, p3.y, p3.z, p3.w}};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned select = (i & 1) ? 0x7632U : 0x5410U;       // the high or the low BF16 of both words
                const int l = 16 * s_side + 8 * h + i;
                uint2 v;
                v.x = __byte_perm(words[0][i >> 1], words[1][i >> 1], select);     // j = 4q, 4q+1
                v.y = __byte_perm(words[2][i >> 1], words[3][i >> 1], select);     // j = 4q+2, 4q+3
                *reinterpret_cast<uint2*>(row + l * 4 + 2 * s_q) = v;
            }
        }
    };
    fetch(0, 0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (KC < columns) fetch(KC, 1);
    transpose(0);
    int buffer = 0;
    for (int k0 = 0; k0 < columns; k0 += KC) {
        // chunk k0 is transposed in tile[buffer] (by every thread: not yet visible), chunk k0 + KC is arriving in raw[buffer ^ 1]
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (k0 + KC < columns) {
            if (k0 + 2 * KC < columns) fetch(k0 + 2 * KC, buffer);   // raw[buffer] was transposed before the barrier
            transpose(buffer ^ 1);                                    // tile[buffer ^ 1] was last read before the barrier
        }
        uint4 wv[TE], xv[TT];
#pragma unroll
        for (int i = 0; i < TE; ++i) wv[i] = *reinterpret_cast<const uint4*>(&tile[buffer][we * TE + i][lane * 4]);
#pragma unroll
        for (int i = 0; i < TT; ++i) xv[i] = *reinterpret_cast<const uint4*>(&tile[buffer][BE + wt * TT + i][lane * 4]);
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            float wf[TE], xf[TT];
#pragma unroll
            for (int i = 0; i < TE; ++i) {
                const std::uint32_t word = jj < 2 ? wv[i].x : jj < 4 ? wv[i].y : jj < 6 ? wv[i].z : wv[i].w;
                wf[i] = __uint_as_float((jj & 1) ? (word & 0xffff0000U) : (word << 16));
            }
#pragma unroll
            for (int i = 0; i < TT; ++i) {
                const std::uint32_t word = jj < 2 ? xv[i].x : jj < 4 ? xv[i].y : jj < 6 ? xv[i].z : xv[i].w;
                xf[i] = __uint_as_float((jj & 1) ? (word & 0xffff0000U) : (word << 16));
            }
#pragma unroll
            for (int i = 0; i < TE; ++i) {
                const float2 w2 = make_float2(wf[i], wf[i]);
#pragma unroll
                for (int t = 0; t < TT / 2; ++t) acc[i][t] = __ffma2_rn(make_float2(xf[2 * t], xf[2 * t + 1]), w2, acc[i][t]);
            }
        }
        buffer ^= 1;
    }
#pragma unroll
    for (int i = 0; i < TE; ++i) {
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            float value = (t & 1) ? acc[i][t / 2].y : acc[i][t / 2].x;
#pragma unroll
            for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_down_sync(0xffffffffU, value, offset);
            const int e = e0 + we * TE + i;
            const int tok = t0 + wt * TT + t;
            if (lane == 0 && e < rows && tok < batch_rows) out[static_cast<std::size_t>(tok) * rows + e] = value;
        }
    }
}

// ---- top-8 ----------------------------------------------------------------
// One warp per token; lane l holds experts l, l+32, ..., l+224 in registers.
// Eight rounds of (local best, warp butterfly arg-max) with the reference's
// total order: higher corrected score first, equal scores -> lower id
// (cuda/nvfp4_ops.cu:391-392,411-412).  Weights are the uncorrected sigmoid of
// the winners, summed in slot order and scaled by routed_scale/total (:420,425-432).
__global__ void __launch_bounds__(128) router_top8_kernel(const float* __restrict__ logits,
                                                          const float* __restrict__ bias,
                                                          std::int32_t* __restrict__ ids,
                                                          float* __restrict__ weights, int rows,
                                                          float routed_scale) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= rows) return;
    warp_top8(logits + static_cast<std::size_t>(row) * kExperts, bias, ids + static_cast<std::size_t>(row) * 8,
              weights + static_cast<std::size_t>(row) * 8, routed_scale);
}

}  // namespace

cudaError_t launch_router_logits(const std::uint16_t* x, const std::uint16_t* w, float* out,
                                 int batch_rows, int rows, int columns, bool gemv_order,
                                 cudaStream_t stream, bool pdl) {
    if (x == nullptr || w == nullptr || out == nullptr || batch_rows <= 0 || rows <= 0 ||
        columns <= 0 || columns % 128 != 0) {
        return cudaErrorInvalidValue;
    }
    if (gemv_order) {
        if (batch_rows != 1) return cudaErrorInvalidValue;
        return launch_kernel(logits_gemv_kernel, dim3(rows), dim3(256), 0, stream, pdl, x, w, out, rows, columns);
    }
    if (!aligned_to(16, x, w)) return cudaErrorInvalidValue;         // the forms below copy 16 bytes at a time
    if (batch_rows <= 8) {
        // decode: the whole K extent of two expert rows and of every token in shared memory
        if (static_cast<std::size_t>(12) * columns * 2 > 200 * 1024) return cudaErrorInvalidValue;
        const dim3 grid((rows + 1) / 2);
        const std::size_t row_bytes = static_cast<std::size_t>(columns) * 2;
        if (batch_rows <= 4) {
            if (cudaError_t st = ensure_dynamic_smem<logits_few_rows_kernel<2>>(200 * 1024); st != cudaSuccess) return st;
            return launch_kernel(logits_few_rows_kernel<2>, grid, dim3(128), 6 * row_bytes, stream, pdl, x, w, out, batch_rows, rows, columns);
        }
        if (cudaError_t st = ensure_dynamic_smem<logits_few_rows_kernel<4>>(200 * 1024); st != cudaSuccess) return st;
        return launch_kernel(logits_few_rows_kernel<4>, grid, dim3(128), 10 * row_bytes, stream, pdl, x, w, out, batch_rows, rows, columns);
    } else if (columns % 256 == 0) {
        // 16 experts x 16 tokens per block of four warps.  (Measured at T=4096 with the chunk copied asynchronously
        // into shared memory and transposed there: 230 µs with this block shape, 237 - 296 µs with three others.)
        dim3 grid((rows + 15) / 16, (batch_rows + 15) / 16);
        constexpr std::size_t smem = 4 * 32 * (32 * 4 + 4) * 4;     // raw and transposed images of 32 padded rows, two of each
        if (cudaError_t st = ensure_dynamic_smem<logits_rows_large_kernel<3>>(static_cast<int>(smem)); st != cudaSuccess) return st;
        return launch_kernel(logits_rows_large_kernel<3>, grid, dim3(128), smem, stream, pdl, x, w, out, batch_rows, rows,
                             columns);
    } else {
        constexpr int TE = 8, TT = 8, WE = 2, WT = 4;
        constexpr int KC = 128;
        const std::size_t smem = static_cast<std::size_t>(TE * WE + TT * WT) * KC * 2;
        dim3 grid((rows + TE * WE - 1) / (TE * WE), (batch_rows + TT * WT - 1) / (TT * WT));
        return launch_kernel(logits_rows_kernel<TE, TT, WE, WT>, grid, dim3(WE * WT * 32), smem, stream, pdl, x, w, out,
                             batch_rows, rows, columns, KC);
    }
}

cudaError_t launch_router_top8(const float* logits, const float* bias, std::int32_t* ids,
                               float* weights, int rows, float routed_scale, cudaStream_t stream, bool pdl) {
    if (logits == nullptr || bias == nullptr || ids == nullptr || weights == nullptr || rows <= 0) {
        return cudaErrorInvalidValue;
    }
    return launch_kernel(router_top8_kernel, dim3((rows + 3) / 4), dim3(128), 0, stream, pdl, logits, bias, ids, weights,
                         rows, routed_scale);
}

}  // namespace p92b
