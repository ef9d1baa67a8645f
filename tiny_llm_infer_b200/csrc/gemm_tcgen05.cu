// y[M, N] = x[M, K] . W[N, K]^T in bfloat16 with float32 accumulation on the fifth-generation
// tensor cores (tcgen05), for the many-row products of a prefill step, with the SwiGLU of
// the feed-forward optionally fused into the epilogue.
//
// The reference calls cublasHgemm for these products and runs SwiGLU as a kernel of its own
// over the [tokens, 2 x intermediate] result (kernels/src/matmul_kernel_cuda.cu:83-91,
// kernels/src/swiglu_kernel_cuda.cu:7-27).
//
// The kernel is persistent: one block per SM walks over 128 x 256 tiles of y (row tiles
// fastest, so that blocks running at the same time share a slab of W in L2).  Warp 0 is the
// producer: one thread issues TMA loads (cp.async.bulk.tensor, 128-byte swizzle) of a
// 128 x 64 slab of x and a 256 x 64 slab of W into a ring of four shared-memory stages and arms
// an mbarrier per stage with the expected byte count.  Warp 1 owns the tensor memory (all 512
// float32 columns of the SM's TMEM: two accumulators of 128 x 256) and issues the MMAs: one
// thread, four tcgen05.mma (128 x 256 x 16) per stage, shared-memory descriptors advanced by
// 32 bytes inside the swizzle atom; a tcgen05.commit hands the stage back to the producer when
// the tensor core has read it, another one hands the finished accumulator to the epilogue.
// Warps 2 to 5 are the epilogue: each thread owns one row of the tile, reads its accumulator
// row from TMEM 32 columns at a time (tcgen05.ld), writes bfloat16 to global memory and gives
// the accumulator back; meanwhile the MMAs of the next tile fill the other accumulator.  In
// SwiGLU mode the W slab is made of 128 gate rows and the 128 up rows that belong to them
// (two TMA boxes), so that columns j and 128 + j of the accumulator are gate and up of the
// same output: the epilogue writes silu(gate) * up, and the [tokens, 2 x intermediate] matrix
// never exists.
//
// Every wait on an mbarrier is bounded: when a limit runs out the block records a code in
// the error word the caller passed, stops issuing work, still waits (bounded) for the copies
// it has in flight, frees its tensor memory and returns.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace tllm {

constexpr int kBM = 128, kBN = 256, kBK = 64;
constexpr int kStageBBytes = kBN * kBK * 2;
constexpr int kGemmThreads = 192;
constexpr uint32_t kTmemCols = 512;

// act(gate) of the gated epilogue with the fast intrinsics: silu g / (1 + e^-g), the tanh form of GELU
// written the same way, 0.5 g (1 + tanh(u)) = g / (1 + e^-2u) with u = sqrt(2/pi) (g + 0.044715 g^3), or ReLU.
template <int ACT>
__device__ __forceinline__ float fast_gate_act(float g) {
    if (ACT == kActRelu) return fmaxf(g, 0.0f);
    if (ACT == kActGeluTanh) {
        const float u2 = 1.5957691216057308f * (g + 0.044715f * g * g * g);
        return __fdividef(g, 1.0f + __expf(-u2));
    }
    return __fdividef(g, 1.0f + __expf(-g));
}

// A gated unit's output the same way (`gated_unit` in common.cuh).
template <int ACT>
__device__ __forceinline__ float fast_gated_unit(float g, float u, const GateConst& c) {
    if (ACT == kActClampedSwish) {
        g = fminf(g, c.limit);
        u = fminf(fmaxf(u, -c.limit), c.limit);
        return __fdividef(g, 1.0f + __expf(-c.slope * g)) * (u + 1.0f);
    }
    return fast_gate_act<ACT>(g) * u;
}

// An activation on every output of a plain product (ACT: a GateAct code, or kActNone for none): silu and the
// tanh GELU as above, the exact GELU 0.5 g (1 + erf(g / sqrt 2)) with the library's erff.
constexpr int kActNone = -1;
template <int ACT>
__device__ __forceinline__ float unary_act(float g) {
    if (ACT == kActGeluErf) return 0.5f * g * (1.0f + erff(g * 0.7071067811865476f));
    if (ACT == kActNone) return g;
    if (ACT == kActTanh) return tanhf(g);
    if (ACT == kActRelu2) { const float r = fmaxf(g, 0.0f); return r * r; }
    return fast_gate_act<ACT>(g);
}

__device__ __forceinline__ void store_bf16x8(bf16* p, const float* v) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}

// Write 32 values of one output row starting at column col0 (vector stores where the row allows).
__device__ __forceinline__ void store_row32(bf16* row_ptr, int col0, int cols, const float* v) {
    if (col0 + 32 <= cols && (cols % 8) == 0) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) store_bf16x8(row_ptr + col0 + i, v + i);
    } else {
        for (int i = 0; i < 32; ++i)
            if (col0 + i < cols) row_ptr[col0 + i] = __float2bfloat16_rn(v[i]);
    }
}

// SWIGLU: W holds `half_n` gate rows and as many up rows, a column tile is 128 outputs and y is
// [M, half_n]; stacked ([gate; up]: the tile's gate and up rows are two boxes, accumulator columns
// 0..127 and 128..255) or interleaved by eight (eight gate rows, their eight up rows, ...: the
// tile is 256 neighbouring rows and a gate's up is eight columns further).  Otherwise a column
// tile is 256 outputs of N and y is [M, N].
// MT: row tiles of 128 per block.  MT = 1: two accumulators of 128 x 256 take turns, the
// epilogue of a tile overlaps the MMAs of the next, four stages of 48 KB.  MT = 2: the block
// owns 256 rows, both accumulators belong to one tile, every slab of W fetched from L2 feeds
// twice as many MMAs (32 KB of shared-memory fill per 128 x 256 x 64 instead of 48 KB), three
// stages of 64 KB; the epilogue is not overlapped.
template <bool SWIGLU, int MT, int ACT>
__global__ void __launch_bounds__(kGemmThreads)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    bf16* __restrict__ y, int M, int N, int K, int half_n, int interleaved, int tiles_m,
                    int tiles_n, int* __restrict__ error_word, const GateConst gc) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[4], empty_bar[4], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    // the dynamic window is not guaranteed to start on a 1024-byte boundary: round up
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    constexpr int kStages = MT == 1 ? 4 : 3, kNumBuf = MT == 1 ? 2 : 1;
    constexpr int kRows = kBM * MT, kStageABytes = kRows * kBK * 2, kStageBytes = kStageABytes + kStageBBytes;
    constexpr int kOutRowBytes = 64 * 2 + 16;                 // staging row of 64 outputs, padded
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* stage_out = tiles + (size_t)kStages * kStageBytes + (size_t)(warp & 3) * 32 * kOutRowBytes;
    const int k_blocks = (K + kBK - 1) / kBK;
    const int total_tiles = tiles_m * tiles_n;
    const int out_cols = SWIGLU ? half_n : N;
    constexpr int kColTile = SWIGLU ? 128 : kBN;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);             // one arrival per epilogue warp
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {   // this warp owns the tensor memory from allocation to release
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         cvta_shared(&tmem_base_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* aborted = &abort_flag;

    if (warp == 0) {
        // ------------------------------------------------------------ producer (one thread)
        if (lane == 0) {
            int it = 0;                               // k-blocks issued so far, over all tiles
            for (int t = blockIdx.x; t < total_tiles && !*aborted; t += gridDim.x) {
                const int tile_m = t % tiles_m, tile_n = t / tiles_m;
                const int a_row = tile_m * kRows;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % kStages;
                    if (it >= kStages && !mbar_wait(&empty_bar[s], ((it / kStages) - 1) & 1)) {
                        atomicExch(error_word, 1);
                        *aborted = 1;
                    }
                    if (*aborted) break;
                    unsigned char* a_dst = tiles + (size_t)s * kStageBytes;
                    unsigned char* b_dst = a_dst + kStageABytes;
                    mbar_expect_tx(&full_bar[s], kStageBytes);
                    tma_load_2d(a_dst, &map_x, kb * kBK, a_row, &full_bar[s]);
                    if (SWIGLU && !interleaved) {
                        tma_load_2d(b_dst, &map_w, kb * kBK, tile_n * 128, &full_bar[s]);
                        tma_load_2d(b_dst + kStageBBytes / 2, &map_w, kb * kBK, half_n + tile_n * 128, &full_bar[s]);
                    } else {
                        tma_load_2d(b_dst, &map_w, kb * kBK, tile_n * kBN, &full_bar[s]);
                        tma_load_2d(b_dst + kStageBBytes / 2, &map_w, kb * kBK, tile_n * kBN + 128, &full_bar[s]);
                    }
                }
            }
            // on an abort: do not leave the block while copies into its shared memory are in flight
            if (*aborted) {
                const int first = it > kStages ? it - kStages : 0;
                for (int i = first; i < it; ++i) mbar_wait(&full_bar[i % kStages], (i / kStages) & 1);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (one thread)
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc_bf16(kBM, kBN);
            int it = 0, local = 0;
            for (int t = blockIdx.x; t < total_tiles && !*aborted; t += gridDim.x, ++local) {
                const int buf = local % kNumBuf;
                if (local >= kNumBuf && !mbar_wait(&acc_empty[buf], ((local / kNumBuf) - 1) & 1)) {
                    atomicExch(error_word, 4);
                    *aborted = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t tmem_acc = tmem_base + buf * kBN;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % kStages;
                    if (!mbar_wait(&full_bar[s], (it / kStages) & 1)) {
                        atomicExch(error_word, 2);
                        *aborted = 1;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t a_addr = cvta_shared(tiles + (size_t)s * kStageBytes);
                    const uint32_t b_addr = a_addr + kStageABytes;
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k) {
                        const uint64_t b_desc = smem_desc_sw128(b_addr + k * 32);
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt) {
                            const uint64_t a_desc = smem_desc_sw128(a_addr + mt * (kBM * kBK * 2) + k * 32);
                            umma_bf16(tmem_acc + mt * kBN, a_desc, b_desc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        }
                    }
                    umma_commit(&empty_bar[s]);      // the stage is free once these MMAs have read it
                }
                umma_commit(&acc_full[buf]);         // the accumulator is complete once all MMAs are done
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (four warps, one row per thread)
        const int quad = warp & 3;                   // a warp may read TMEM lanes 32 * (warp % 4) .. + 31
        int local = 0;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++local) {
            const int buf = local % kNumBuf;
            const int tile_m = t % tiles_m, tile_n = t / tiles_m;
            const int row_base = tile_m * kRows;
            if (!warp_wait(&acc_full[buf], (local / kNumBuf) & 1, aborted, error_word, 3)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
            for (int mt = 0; mt < MT; ++mt) {
                const int row0 = row_base + mt * kBM + quad * 32;                // first row of this warp
                const uint32_t lane_addr = tmem_base + (buf + mt) * kBN + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
                for (int c = 0; c < kColTile; c += 64) {                          // 64 output columns at a time
                    float v[64];
                    if (SWIGLU && interleaved) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {             // 64 accumulator columns: 32 outputs
                            uint32_t r0[32], r1[32];
                            tmem_ld32_issue(lane_addr + 2 * c + 64 * h, r0);
                            tmem_ld32_issue(lane_addr + 2 * c + 64 * h + 32, r1);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                const int gi = 16 * (i >> 3) + (i & 7);
                                const float g0 = __uint_as_float(r0[gi]), g1 = __uint_as_float(r1[gi]);
                                v[32 * h + i] = fast_gated_unit<ACT>(g0, __uint_as_float(r0[gi + 8]), gc);
                                v[32 * h + 16 + i] = fast_gated_unit<ACT>(g1, __uint_as_float(r1[gi + 8]), gc);
                            }
                        }
                    } else if (SWIGLU) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t gr[32], ur[32];
                            tmem_ld32_issue(lane_addr + c + 32 * h, gr);
                            tmem_ld32_issue(lane_addr + 128 + c + 32 * h, ur);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                const float g = __uint_as_float(gr[i]);
                                v[32 * h + i] = fast_gated_unit<ACT>(g, __uint_as_float(ur[i]), gc);
                            }
                        }
                    } else {
                        uint32_t r0[32], r1[32];
                        tmem_ld32_issue(lane_addr + c, r0);
                        tmem_ld32_issue(lane_addr + c + 32, r1);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            v[i] = unary_act<ACT>(__uint_as_float(r0[i]));
                            v[32 + i] = unary_act<ACT>(__uint_as_float(r1[i]));
                        }
                    }
                    // through the warp's staging tile, so that a store instruction writes whole
                    // 128-byte lines (4 rows x 128 bytes) instead of 16 bytes in each of 32 rows
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 64; i += 8) store_bf16x8(reinterpret_cast<bf16*>(stage_out + lane * kOutRowBytes) + i, v + i);
                    __syncwarp();
                    const int col0 = tile_n * kColTile + c;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int piece = lane + 32 * j, r = piece >> 3, p16 = piece & 7;
                        const int row = row0 + r, col = col0 + p16 * 8;
                        if (row < M && col < out_cols) {
                            const uint4 val = *reinterpret_cast<const uint4*>(stage_out + r * kOutRowBytes + p16 * 16);
                            bf16* dst = y + (size_t)row * out_cols + col;
                            if (col + 8 <= out_cols && (out_cols % 8) == 0) {
                                *reinterpret_cast<uint4*>(dst) = val;
                            } else {
                                const bf16* e = reinterpret_cast<const bf16*>(&val);
                                for (int i = 0; i < 8; ++i)
                                    if (col + i < out_cols) dst[i] = e[i];
                            }
                        }
                    }
                }
            }
            // the accumulator may be overwritten once all four warps have read it
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols)
                     : "memory");
    }
}

// ---------------------------------------------------------------- the experts of a mixture
// y[r] = x[r] . W_e^T for the rows r of every expert e, x the plan's rows one after the other, w the experts' matrices
// stacked ([experts * w_rows, K]).  The weights are the MMA's A operand (128 weight rows: the M of the instruction) and an
// expert's rows its B operand, so the instruction's N follows the expert's rows in steps of sixteen: an accumulator is
// [128 weight rows x n rows], a tile of few rows costs little, and every weight comes from HBM once as long as its expert
// has no more rows than a tile of the plan.
//
// What bounds it: with few rows per expert the weights' way from HBM (64 experts of 2048 x 4096, gate|up + down: 138 + 69 us
// for 8 tokens that reach 25 experts, 6.0 TB/s; 330 + 165 us for 256 tokens, 6.5 TB/s), with many what the blocks fetch
// from L2 (425 + 224 us for 8192 rows, 0.97 PFLOP/s).  Two weight slabs per block halve the fetches of the rows: 441 instead of
// 530 us with 8192 rows, 140 instead of 155 with 32.  Tiles of 256 rows leave no second accumulator beside the first (450 us),
// boxes of 16 and 32 rows instead of 64 cost the copy engine more than they save (567, 501 us).  Issued from a branch for
// one lane, the MMAs of a stage took longer than HBM takes to deliver it (180 instead of 155 us with 32 rows).
// The form with the rows as A operand, padded to 128 per tile, took 465 + 233 us for 8192 rows; few rows ran on
// mma.sync tiles (336 + 162 us for 8 tokens), and on mma.sync fragments straight from HBM they take 146 + 95 us.
//
// Warps as in the dense kernel: one producer thread, one MMA warp, four epilogue warps.  An epilogue thread owns one
// weight row (an output column) and reads sixteen rows' sums at a time; for gated units, whose gate and up rows are
// interleaved by eight, the lanes eight apart exchange sums, each then making the outputs of every second row.
struct MoeTiles {
    const int *tile_expert, *tile_row0, *n_tiles, *offsets;
};
constexpr int kMoeStages = 9, kMoeBoxRows = 64;

// The MMA warp runs its loop whole: the descriptors are made by all its lanes (in uniform registers) and one lane issues.
__device__ __forceinline__ void umma_bf16_if(uint32_t issue, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(issue)
        : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t issue, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(cvta_shared(bar)),
        "r"(issue)
        : "memory");
}

// SLABS: weight tiles of 128 rows per block.  MODE 0: the product, as TOut.  1: act(gate) * up.  2: act(product).
// ACT: a GateAct code.
template <int SLABS, int MODE, int ACT, typename TOut>
__global__ void __launch_bounds__(kGemmThreads)
moe_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, TOut* __restrict__ y,
                   int w_rows, int K, int tiles_n, int tile_rows, int stages, int* __restrict__ error_word,
                   const MoeTiles lists, const GateConst gc) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kMoeStages], empty_bar[kMoeStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    constexpr int kSlab = kBM * kBK * 2, kABytes = SLABS * kSlab;
    const int stage_bytes = kABytes + tile_rows * kBK * 2;
    constexpr int kAccCols = 128, kAccTile = SLABS * kAccCols;       // of tensor memory; two tiles' accumulators take turns
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_blocks = (K + kBK - 1) / kBK;
    const int total = *lists.n_tiles * tiles_n;             // an expert's weight tiles one after the other
    const int out_cols = MODE == 1 ? w_rows / 2 : w_rows;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMoeStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(cvta_shared(&tmem_base_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* aborted = &abort_flag;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0, issued = 0;
            uint32_t phase = 1;                              // of empty_bar: the first round of the ring waits for nothing
            for (int t = blockIdx.x; t < total && !*aborted; t += gridDim.x) {
                const int tile = t / tiles_n, e = lists.tile_expert[tile], row0 = lists.tile_row0[tile];
                const int rows = min(tile_rows, lists.offsets[e + 1] - row0), boxes = (rows + kMoeBoxRows - 1) / kMoeBoxRows;
                const int w_row = e * w_rows + (t - tile * tiles_n) * SLABS * kBM;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (issued >= stages && !mbar_wait(&empty_bar[s], phase)) {
                        atomicExch(error_word, 1);
                        *aborted = 1;
                    }
                    if (*aborted) break;
                    unsigned char* a_dst = tiles + (size_t)s * stage_bytes;
                    mbar_expect_tx(&full_bar[s], kABytes + boxes * kMoeBoxRows * kBK * 2);
                    tma_load_2d(a_dst, &map_w, kb * kBK, w_row, &full_bar[s]);
                    for (int b = 0; b < boxes; ++b)
                        tma_load_2d(a_dst + kABytes + b * kMoeBoxRows * kBK * 2, &map_x, kb * kBK, row0 + b * kMoeBoxRows, &full_bar[s]);
                    ++issued;
                    if (++s == stages) { s = 0; phase ^= 1; }
                }
            }
            // on an abort: do not leave the block while copies into its shared memory are in flight
            if (*aborted) {
                const int first = issued > stages ? issued - stages : 0;
                for (int i = first; i < issued; ++i) mbar_wait(&full_bar[i % stages], (i / stages) & 1);
            }
        }
    } else if (warp == 1) {
        const uint32_t issue = lane == 0;
        const uint64_t desc0 = smem_desc_sw128(cvta_shared(tiles));     // a stage and a step inside it only add to its address
        int s = 0, local = 0;
        uint32_t phase = 0;
        for (int t = blockIdx.x; t < total && !*aborted; t += gridDim.x, ++local) {
            const int tile = t / tiles_n;
            const int rows = min(tile_rows, lists.offsets[lists.tile_expert[tile] + 1] - lists.tile_row0[tile]);
            const uint32_t idesc = instr_desc_bf16(kBM, (rows + 15) & ~15);
            const int buf = local & 1;
            if (local >= 2 && !mbar_wait(&acc_empty[buf], ((local >> 1) - 1) & 1)) {
                if (issue) atomicExch(error_word, 4);
                *aborted = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t tmem_acc = tmem_base + buf * kAccTile;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!mbar_wait(&full_bar[s], phase)) {
                    if (issue) atomicExch(error_word, 2);
                    *aborted = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint64_t a_desc = desc0 + (uint32_t)(s * stage_bytes >> 4), b_desc = a_desc + (kABytes >> 4);
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k)
#pragma unroll
                    for (int m = 0; m < SLABS; ++m)
                        umma_bf16_if(issue, tmem_acc + m * kAccCols, a_desc + (m * kSlab + k * 32) / 16, b_desc + k * 2, idesc,
                                     (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit_if(issue, &empty_bar[s]);
                if (++s == stages) { s = 0; phase ^= 1; }
            }
            umma_commit_if(issue, &acc_full[buf]);
        }
    } else {
        const int quad = warp & 3;
        int local = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++local) {
            const int tile = t / tiles_n, row0 = lists.tile_row0[tile];
            const int rows = min(tile_rows, lists.offsets[lists.tile_expert[tile] + 1] - row0);
            const int buf = local & 1;
            if (!warp_wait(&acc_full[buf], (local >> 1) & 1, aborted, error_word, 3)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
            for (int m = 0; m < SLABS; ++m) {
                const int w0 = ((t - tile * tiles_n) * SLABS + m) * kBM + quad * 32;       // first weight row of this warp
                const uint32_t lane_addr = tmem_base + buf * kAccTile + m * kAccCols + ((uint32_t)(quad * 32) << 16);
                const int col = MODE == 1 ? w0 / 2 + (lane >> 4) * 8 + (lane & 7) : w0 + lane;
                const bool is_up = MODE == 1 && (lane & 8);
#pragma unroll 1
                for (int c = 0; c < rows; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(lane_addr + c, r);
                    tmem_ld_wait();
                    TOut* dst = y + (size_t)(row0 + c) * out_cols + col;
                    if (MODE == 1) {
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            const float mine = __uint_as_float(is_up ? r[i + 1] : r[i]);
                            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(is_up ? r[i] : r[i + 1]), 8);
                            const float v = gated_unit(is_up ? other : mine, is_up ? mine : other, ACT, gc);
                            const int row = i + (is_up ? 1 : 0);
                            if (c + row < rows && col < out_cols) dst[(size_t)row * out_cols] = from_f32<TOut>(v);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float v = MODE == 2 ? gate_act(__uint_as_float(r[i]), ACT) : __uint_as_float(r[i]);
                            if (c + i < rows && col < out_cols) dst[(size_t)i * out_cols] = from_f32<TOut>(v);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// ---------------------------------------------------------------------------------- host side
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// Tensor map of a row-major [rows, k] bfloat16 matrix for boxes of `box_rows` x 64 with 128-byte swizzle.
static bool make_map(CUtensorMap* map, const void* base, long long rows, long long k, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int sm_count() {
    static int n = [] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        return v;
    }();
    return n;
}

template <bool SWIGLU, int MT, int ACT = (SWIGLU ? (int)kActSilu : kActNone)>
static int launch_tcgen05(const CUtensorMap& mx, const CUtensorMap& mw, void* y, int M, int N, int K, int half_n,
                          int interleaved, int* error_word, cudaStream_t stream, const GateConst gc = GateConst{0.0f, 0.0f}) {
    const size_t smem = (size_t)(MT == 1 ? 4 : 3) * (kBM * MT * kBK * 2 + kStageBBytes) + 1024 + 4 * 32 * (64 * 2 + 16);
    static OncePerDevice configured;
    if (configured.first()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel<SWIGLU, MT, ACT>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { set_error("gemm_tcgen05: %s", cudaGetErrorString(e)); return (int)e; }
        configured.done();
    }
    const int out_cols = SWIGLU ? half_n : N;
    const int col_tile = SWIGLU ? 128 : kBN;
    const int tiles_n = (out_cols + col_tile - 1) / col_tile;
    const int tiles_m = (M + kBM * MT - 1) / (kBM * MT);
    const int total = tiles_m * tiles_n;
    const int grid = total < sm_count() ? total : sm_count();
    gemm_tcgen05_kernel<SWIGLU, MT, ACT><<<grid, kGemmThreads, smem, stream>>>(mx, mw, (bf16*)y, M, N, K, half_n, interleaved,
                                                                      tiles_m, tiles_n, error_word, gc);
    return finish_launch("gemm_tcgen05");
}

template <int SLABS, int MODE, int ACT, typename TOut>
static int launch_moe_tcgen05(const CUtensorMap& mx, const CUtensorMap& mw, void* y, int w_rows, int K, int tile_rows,
                              int max_tiles, const MoeTiles& lists, GateConst gc, int* error_word, cudaStream_t stream) {
    constexpr size_t kMost = 226 * 1024 - 512;              // of 227 KB; the barriers and the alignment of the ring take the rest
    const size_t stage = (size_t)(SLABS * kBM + tile_rows) * kBK * 2;
    int stages = (int)((kMost - 1024) / stage);
    if (stages > kMoeStages) stages = kMoeStages;
    static OncePerDevice configured;
    if (configured.first()) {
        cudaError_t e = cudaFuncSetAttribute(moe_tcgen05_kernel<SLABS, MODE, ACT, TOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost);
        if (e != cudaSuccess) { set_error("moe_tcgen05: %s", cudaGetErrorString(e)); return (int)e; }
        configured.done();
    }
    const int tiles_n = (w_rows + SLABS * kBM - 1) / (SLABS * kBM);
    const long long most = (long long)max_tiles * tiles_n;
    const int grid = most < sm_count() ? (int)most : sm_count();
    moe_tcgen05_kernel<SLABS, MODE, ACT, TOut><<<grid, kGemmThreads, stages * stage + 1024, stream>>>(
        mx, mw, (TOut*)y, w_rows, K, tiles_n, tile_rows, stages, error_word, lists, gc);
    return finish_launch("moe_tcgen05");
}

}  // namespace tllm

using namespace tllm;

// y = x . w^T (y is [M, N]) or, with bit 1 of `swiglu`, y = silu(x . gate^T) * (x . up^T) (y is
// [M, N / 2]) for w = [gate; up], or with bit 4 as well for gate and up rows interleaved by eight.
// Bits 8 and up: the activation (GateAct); limit, slope: constants of the clamped swish.
// Bit 2 keeps blocks of 128 rows.  x [M, K], w [N, K] bfloat16 row-major, K a multiple of 8,
// operands 16-byte aligned.  `error_word` is a device int the kernel sets to a non-zero code if
// one of its bounded waits ran out (the result is then invalid); the caller clears and reads it.
extern "C" int tllm_gemm_tcgen05(const void* x, const void* w, void* y, int M, int N, int K, int swiglu,
                                 float limit, float slope, int* error_word, cudaStream_t stream) {
    TLLM_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_tcgen05: bad sizes");
    TLLM_REQUIRE(K % 8 == 0, "gemm_tcgen05: K = %d is no multiple of 8", K);
    TLLM_REQUIRE(!(swiglu & 1) || N % 2 == 0, "gemm_tcgen05: SwiGLU needs an even number of weight rows");
    const int interleaved = (swiglu & 4) ? 1 : 0;
    TLLM_REQUIRE(!interleaved || ((swiglu & 1) && N % 16 == 0),
                 "gemm_tcgen05: interleaved gate and up rows come in sixteens, N = %d", N);
    TLLM_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0,
                 "gemm_tcgen05: operands must be 16-byte aligned");
    TLLM_REQUIRE(error_word != nullptr, "gemm_tcgen05: no error word");
    CUtensorMap mx, mw;
    const bool tall = M > 128 && !(swiglu & 2) ;          // blocks of 256 rows once there are that many
    TLLM_REQUIRE(make_map(&mx, x, M, K, tall ? 2 * kBM : kBM) && make_map(&mw, w, N, K, 128),
                 "gemm_tcgen05: cuTensorMapEncodeTiled failed or is not available");
    const int act = swiglu >> 8;                            // bits 8 and up: the activation (GateAct)
    if (swiglu & 16) {                                      // a plain product with an activation on every output
        TLLM_REQUIRE(!(swiglu & 1), "gemm_tcgen05: either a gated or a plain activation");
#define UNARY(A) (tall ? launch_tcgen05<false, 2, A>(mx, mw, y, M, N, K, 0, 0, error_word, stream)                \
                       : launch_tcgen05<false, 1, A>(mx, mw, y, M, N, K, 0, 0, error_word, stream))
        if (act == kActGeluErf) return UNARY(kActGeluErf);
        if (act == kActGeluTanh) return UNARY(kActGeluTanh);
        if (act == kActSilu) return UNARY(kActSilu);
        if (act == kActRelu2) return UNARY(kActRelu2);
        if (act == kActTanh) return UNARY(kActTanh);
#undef UNARY
        TLLM_REQUIRE(false, "gemm_tcgen05: unknown activation %d", act);
    }
    TLLM_REQUIRE(gated_act_ok(act, limit), "gemm_tcgen05: unknown activation %d", act);
    if ((swiglu & 1) && act == kActClampedSwish) {
        const GateConst gc{limit, slope};
        return tall ? launch_tcgen05<true, 2, kActClampedSwish>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream, gc)
                    : launch_tcgen05<true, 1, kActClampedSwish>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream, gc);
    }
    if ((swiglu & 1) && act == kActRelu)
        return tall ? launch_tcgen05<true, 2, kActRelu>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream)
                    : launch_tcgen05<true, 1, kActRelu>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream);
    if ((swiglu & 1) && act == kActGeluTanh)
        return tall ? launch_tcgen05<true, 2, kActGeluTanh>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream)
                    : launch_tcgen05<true, 1, kActGeluTanh>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream);
    if (swiglu & 1)
        return tall ? launch_tcgen05<true, 2>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream)
                    : launch_tcgen05<true, 1>(mx, mw, y, M, N, K, N / 2, interleaved, error_word, stream);
    return tall ? launch_tcgen05<false, 2>(mx, mw, y, M, N, K, 0, 0, error_word, stream)
                : launch_tcgen05<false, 1>(mx, mw, y, M, N, K, 0, 0, error_word, stream);
}

// The experts' products: x [rows, K] holds the experts' rows one after the other, w is [experts][n][K], and the plan's
// lists (device memory; at most max_tiles entries) cut every expert's rows into tiles of at most tile_rows (64 or 128).  flags: 1 gated (with 4: gate and up rows interleaved by eight, y is [rows, n / 2] bfloat16); 16 an activation on
// every output (y bfloat16); else the plain product, bfloat16 or with 32 float32.  Bits 8 and up: the activation
// (GateAct).
extern "C" int tllm_moe_tcgen05(const void* x, const void* w, void* y, int rows, int n, int K, int experts, int flags, int tile_rows,
                                const int* tile_expert, const int* tile_row0, const int* n_tiles, const int* offsets, int max_tiles,
                                float limit, float slope, int* error_word, cudaStream_t stream) {
    TLLM_REQUIRE(rows > 0 && n > 0 && K > 0 && experts > 0 && max_tiles > 0, "moe_tcgen05: bad sizes");
    TLLM_REQUIRE((long long)experts * n <= 0x7fffffff - 2 * kBM, "moe_tcgen05: %d experts of %d weight rows", experts, n);
    TLLM_REQUIRE(K % 8 == 0, "moe_tcgen05: K = %d is no multiple of 8", K);
    TLLM_REQUIRE(tile_rows == 64 || tile_rows == 128, "moe_tcgen05: tiles of %d rows", tile_rows);
    const bool gated = flags & 1;
    // One weight slab per block while that still gives every multiprocessor at most one block (4 rows of 64 experts:
    // 36 + 17 us instead of 40 + 19; 8 rows, 59 + 30 instead of 57 + 29, already take two).
    const int reached = rows < experts ? rows : experts;
    const bool two = (long long)reached * ((n + kBM - 1) / kBM) > sm_count();
    TLLM_REQUIRE(!gated || ((flags & 4) && n % 16 == 0), "moe_tcgen05: gate and up rows interleaved by eight, n = %d", n);
    TLLM_REQUIRE((long long)max_tiles * ((n + kBM - 1) / kBM) <= 0x7fffffff, "moe_tcgen05: too many tiles");
    TLLM_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15u) == 0,
                 "moe_tcgen05: operands must be 16-byte aligned");
    TLLM_REQUIRE(error_word && tile_expert && tile_row0 && n_tiles && offsets, "moe_tcgen05: missing list");
    CUtensorMap mx, mw;
    TLLM_REQUIRE(make_map(&mx, x, rows, K, kMoeBoxRows) && make_map(&mw, w, (long long)experts * n, K, two ? 2 * kBM : kBM),
                 "moe_tcgen05: cuTensorMapEncodeTiled failed or is not available");
    const MoeTiles lists{tile_expert, tile_row0, n_tiles, offsets};
    const GateConst gc{limit, slope};
    const int act = flags >> 8;
#define MOE(M, A, T)                                                                                                            \
    return two ? launch_moe_tcgen05<2, M, A, T>(mx, mw, y, n, K, tile_rows, max_tiles, lists, gc, error_word, stream)  \
               : launch_moe_tcgen05<1, M, A, T>(mx, mw, y, n, K, tile_rows, max_tiles, lists, gc, error_word, stream)
    if (flags & 16) {
        TLLM_REQUIRE(!gated, "moe_tcgen05: either a gated or a plain activation");
        if (act == kActRelu2) MOE(2, kActRelu2, bf16);
        if (act == kActTanh) MOE(2, kActTanh, bf16);
        if (act == kActSilu) MOE(2, kActSilu, bf16);
        if (act == kActGeluTanh) MOE(2, kActGeluTanh, bf16);
        if (act == kActGeluErf) MOE(2, kActGeluErf, bf16);
        TLLM_REQUIRE(false, "moe_tcgen05: unknown activation %d", act);
    }
    TLLM_REQUIRE(!gated || gated_act_ok(act, limit), "moe_tcgen05: unknown activation %d", act);
    if (gated && act == kActClampedSwish) MOE(1, kActClampedSwish, bf16);
    if (gated && act == kActRelu) MOE(1, kActRelu, bf16);
    if (gated && act == kActGeluTanh) MOE(1, kActGeluTanh, bf16);
    if (gated) MOE(1, kActSilu, bf16);
    if (flags & 32) MOE(0, kActSilu, float);
    MOE(0, kActSilu, bf16);
#undef MOE
}
