// y[M, N] = x[M, K] . W[N, K]^T, float32 in and out, on the fifth-generation tensor cores (tcgen05).
//
// The tensor cores have no float32 product, so every operand goes in as the sum of three bfloat16 numbers, which holds its 24
// bits: x = x0 + x1 + x2, w likewise, and of the nine products the six down to 2^-18 of the largest are made (what is left out is
// below 2^-26).  The tensor core cuts its float32 sums off instead of rounding them, so x0 w0 has an accumulator of its own, the
// five small products another, and after every 128 terms both are added to float32 sums in registers, rounded to nearest: the
// result is closer to 64 bits than the library's sum over k in order (2-norms at K = 1024: 1.4e-7 and 5.7e-7, at 12288 2.1e-7 and
// 2.0e-6).
//
// Warps 0 to 7 fetch both operands as float32 (each thread eight pieces of eight numbers, the next slab's loads on their way
// while the present one is split), split them and write the six bfloat16 slabs of 128 x 64 in the 128-byte swizzle; one thread of
// warp 16 issues 24 MMAs (128 x 128 x 16) per slab of 64; warps 8 to 15 add the accumulators up, two sets of which take turns.
// Sums that are no finite numbers are made again at the end from the operands as they are, so that infinities, overflows and numbers
// that bfloat16 cannot hold come out as a float32 product has them.  Below some 2^-110 an operand's last part loses bits.
// No scratch and no second copy of a weight exists.  Work for few tiles is cut over K, the shares' sums added in their order by a
// second kernel.
//
// What bounds it: a slab takes 1.65 us, of which the MMAs are 0.8 at the tensor core's rate; they read shared memory at its full
// width while the splitters write 96 KB a slab into it, and the splitters' loads are one slab ahead at most (a piece's load issued as
// soon as the piece is split was slower, 2.1 us: the threads then wait on loads between their stores).  2048 x 24576 x 4096: 2.22 ms,
// 186 TFLOP/s; the library's kernel 6.95 ms.  Smaller sizes: ops.f32_tcgen05_pays.
#include "common.cuh"
#include "mma_tiles.cuh"
#include "tcgen05.cuh"

namespace tllm {

constexpr int kFTile = 128, kFK = 64, kFStages = 2, kFPart = kFTile * kFK * 2, kFStage = 6 * kFPart;
constexpr int kFSplitters = 256, kFAdders = 256, kFThreads = kFSplitters + kFAdders + 32;
constexpr float kFLargest = 3.402823466e38f; // the largest finite number
constexpr int kFTogether = 2;                // slabs whose products meet in one pair of accumulators (128 terms)

__global__ void __launch_bounds__(kFThreads, 1)
gemm_f32_tcgen05_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, int tiles_m,
                        int tiles, int splits, int slabs_each, int* __restrict__ error_word) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kFStages], empty_bar[kFStages], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag, odd_flag;
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int all_slabs = (K + kFK - 1) / kFK, units = tiles * splits;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kFStages; ++s) {
            mbar_init(&full_bar[s], kFSplitters / 32);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kFAdders / 32);
        }
        mbar_init(&drained, 1);
        abort_flag = odd_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(cvta_shared(&tmem_base_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base_slot;
    volatile int* aborted = &abort_flag;
    // unit u: tile u % tiles (rows of x fastest), share u / tiles of its slabs
    auto slabs_of = [&](int u) { return min(slabs_each, all_slabs - u / tiles * slabs_each); };

    if (warp < 8) {
        // ------------------------------------------------------------ fetch and split
        const int piece = threadIdx.x & 7, row0 = threadIdx.x >> 3;                    // rows row0 + 32 i
        float4 v[8][2];                                                                // four pieces of x, four of w
        auto fetch = [&](int u, int slab) {
            const int tile = u % tiles, m0 = tile % tiles_m * kFTile, n0 = tile / tiles_m * kFTile;
            const int k = (u / tiles * slabs_each + slab) * kFK + piece * 8;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const bool is_x = i < 4;
                const int r = (is_x ? m0 : n0) + row0 + 32 * (i & 3);
                const float* p = (is_x ? x : w) + (size_t)r * K + k;
                const bool in = r < (is_x ? M : N);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    v[i][h] = in && k + 4 * h < K ? *reinterpret_cast<const float4*>(p + 4 * h) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        };
        int it = 0;
        bool alive = true;
        if ((int)blockIdx.x < units) fetch(blockIdx.x, 0);
        for (int u = blockIdx.x; u < units && alive; u += gridDim.x) {
            const int slabs = slabs_of(u);
            for (int slab = 0; slab < slabs; ++slab, ++it) {
                const int s = it % kFStages;
                if (it >= kFStages && !warp_wait(&empty_bar[s], ((it / kFStages) - 1) & 1, aborted, error_word, 11)) { alive = false; break; }
                unsigned char* stage = ring + s * kFStage;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint4 p[3];
                    split3(v[i][0].x, v[i][0].y, p[0].x, p[1].x, p[2].x);
                    split3(v[i][0].z, v[i][0].w, p[0].y, p[1].y, p[2].y);
                    split3(v[i][1].x, v[i][1].y, p[0].z, p[1].z, p[2].z);
                    split3(v[i][1].z, v[i][1].w, p[0].w, p[1].w, p[2].w);
                    const int r = row0 + 32 * (i & 3);
                    unsigned char* to = stage + (i < 4 ? 0 : 3 * kFPart) + r * 128 + ((piece ^ (r & 7)) << 4);
#pragma unroll
                    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(to + q * kFPart) = p[q];
                }
                if (slab + 1 < slabs) fetch(u, slab + 1);
                else if (u + (int)gridDim.x < units) fetch(u + gridDim.x, 0);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");         // the tensor core reads what these threads wrote
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_bar[s]);
            }
        }
    } else if (warp == 16) {
        // ------------------------------------------------------------ MMA issuer (one thread)
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc_bf16(kFTile, kFTile);
            constexpr int kLeft[6] = {2, 0, 1, 1, 0, 0}, kRight[6] = {0, 2, 1, 0, 1, 0};
            int it = 0, group = 0;
            const auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
                if (!mbar_wait(bar, parity)) {
                    atomicExch(error_word, code);
                    *aborted = 1;
                }
                return !*aborted;
            };
            for (int u = blockIdx.x; u < units && !*aborted; u += gridDim.x) {
                const int slabs = slabs_of(u);
                for (int slab = 0; slab < slabs && !*aborted; slab += kFTogether, ++group) {
                    const int buf = group & 1;
                    if (group >= 2 && !wait(&acc_empty[buf], ((group >> 1) - 1) & 1, 14)) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    for (int j = slab; j < min(slab + kFTogether, slabs); ++j, ++it) {
                        const int s = it % kFStages;
                        if (!wait(&full_bar[s], (it / kFStages) & 1, 12)) break;
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        const uint32_t a = cvta_shared(ring + s * kFStage), b = a + 3 * kFPart;
#pragma unroll
                        for (int q = 0; q < 6; ++q)
#pragma unroll
                            for (int k = 0; k < kFK / 16; ++k)
                                umma_bf16(tmem + buf * 256 + (q < 5 ? 128 : 0), smem_desc_sw128(a + kLeft[q] * kFPart + k * 32),
                                          smem_desc_sw128(b + kRight[q] * kFPart + k * 32), idesc, j > slab || k > 0 || (q > 0 && q < 5) ? 1u : 0u);
                        umma_commit(&empty_bar[s]);
                    }
                    umma_commit(&acc_full[buf]);
                }
            }
            if (*aborted) {                          // do not leave while products are in flight
                umma_commit(&drained);
                mbar_wait(&drained, 0);
            }
        }
    } else {
        // ------------------------------------------------------------ add the accumulators up (a row and 64 columns per thread)
        const int quad = warp & 3, half = (warp >> 2) & 1;
        int group = 0;
        bool alive = true, odd = false;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int slabs = slabs_of(u);
            float sum[64];
#pragma unroll
            for (int i = 0; i < 64; ++i) sum[i] = 0.0f;
            for (int slab = 0; slab < slabs; slab += kFTogether, ++group) {
                const int buf = group & 1;
                if (!warp_wait(&acc_full[buf], (group >> 1) & 1, aborted, error_word, 13)) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t from = tmem + buf * 256 + half * 64 + ((uint32_t)(quad * 32) << 16);
#pragma unroll
                for (int c = 0; c < 64; c += 16)
#pragma unroll
                    for (int part = 1; part >= 0; --part) {                            // the small products first
                        uint32_t r[16];
                        tmem_ld16(from + part * 128 + c, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(r[i]);
                    }
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[buf]);
            }
            if (!alive) break;
            const int tile = u % tiles, row = tile % tiles_m * kFTile + quad * 32 + lane, col0 = tile / tiles_m * kFTile + half * 64;
            if (row < M) {
                float* dst = y + ((size_t)(u / tiles) * M + row) * N + col0;
                float largest = 0.0f;                // NaN where any sum is an infinity or no number
#pragma unroll
                for (int i = 0; i < 64; ++i) largest = fmaf(sum[i], 0.0f, largest);
                odd |= largest != largest;
#pragma unroll
                for (int i = 0; i < 64; i += 4)
                    if (col0 + i < N) *reinterpret_cast<float4*>(dst + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
            }
        }
        if (odd) odd_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (odd_flag && !abort_flag) {
        // A sum that is no finite number is made again from the float32 operands, a thread each, over its share of K in order: an
        // infinity's second part is no number and its product with a part of zero neither, and a number beyond the largest
        // bfloat16 goes in as an infinity.  Given up once it is no number, which it then stays.
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int tile = u % tiles, m0 = tile % tiles_m * kFTile, n0 = tile / tiles_m * kFTile;
            const int k0 = u / tiles * slabs_each * kFK, k1 = min(K, k0 + slabs_of(u) * kFK);
            for (int i = threadIdx.x; i < kFTile * kFTile; i += kFThreads) {
                const int row = m0 + i / kFTile, col = n0 + i % kFTile;
                if (row >= M || col >= N) continue;
                float* at = y + ((size_t)(u / tiles) * M + row) * N + col;
                if (fabsf(*at) <= kFLargest) continue;
                float sum = 0.0f;
                for (int k = k0; k < k1 && sum == sum; k += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(x + (size_t)row * K + k);
                    const float4 b = *reinterpret_cast<const float4*>(w + (size_t)col * K + k);
                    sum = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
                }
                *at = sum;
            }
        }
    }
    if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
}

// y[i] = the shares' sums in their order, four numbers per thread.
__global__ void gemm_f32_shares_kernel(const float* __restrict__ shares, float* __restrict__ y, size_t n, int splits) {
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += (size_t)gridDim.x * blockDim.x * 4) {
        float4 s = *reinterpret_cast<const float4*>(shares + i);
        for (int k = 1; k < splits; ++k) {
            const float4 v = *reinterpret_cast<const float4*>(shares + k * n + i);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        *reinterpret_cast<float4*>(y + i) = s;
    }
}

}  // namespace tllm

using namespace tllm;

// x [M, K], w [N, K], y [M, N] float32 row-major, K and N multiples of 4, operands 16-byte aligned.  splits: shares of K (each of
// at least one slab of 64); with more than one, shares is float[splits * M * N].  error_word as in tllm_gemm_tcgen05.
extern "C" int tllm_gemm_f32_tcgen05(const float* x, const float* w, float* y, int M, int N, int K, int splits, float* shares,
                                     int* error_word, cudaStream_t stream) {
    TLLM_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32_tcgen05: bad sizes");
    TLLM_REQUIRE(K % 4 == 0 && N % 4 == 0, "gemm_f32_tcgen05: K = %d, N = %d are no multiples of 4", K, N);
    TLLM_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y) |
                   reinterpret_cast<uintptr_t>(shares)) & 15u) == 0, "gemm_f32_tcgen05: operands must be 16-byte aligned");
    const int slabs = (K + kFK - 1) / kFK;
    TLLM_REQUIRE(splits >= 1 && splits <= slabs && (splits == 1 || shares != nullptr), "gemm_f32_tcgen05: %d shares of %d slabs", splits, slabs);
    TLLM_REQUIRE(error_word != nullptr, "gemm_f32_tcgen05: no error word");
    const int each = (slabs + splits - 1) / splits, used = (slabs + each - 1) / each;        // shares that have any
    const long long tiles_m = (M + kFTile - 1) / kFTile, tiles = tiles_m * ((N + kFTile - 1) / kFTile);
    TLLM_REQUIRE(tiles * used <= 0x7fffffff, "gemm_f32_tcgen05: too many tiles");
    constexpr int kBytes = kFStages * kFStage + 1024;
    static OncePerDevice configured;
    if (configured.first()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
        if (e != cudaSuccess) { set_error("gemm_f32_tcgen05: %s", cudaGetErrorString(e)); return (int)e; }
        configured.done();
    }
    const int sms = sm_count_cached() > 0 ? sm_count_cached() : 148;
    const int grid = tiles * used < sms ? (int)(tiles * used) : sms;
    gemm_f32_tcgen05_kernel<<<grid, kFThreads, kBytes, stream>>>(x, w, used > 1 ? shares : y, M, N, K, (int)tiles_m, (int)tiles, used, each, error_word);
    if (int rc = finish_launch("gemm_f32_tcgen05")) return rc;
    if (used == 1) return 0;
    const size_t n = (size_t)M * N;
    const size_t blocks = (n / 4 + 255) / 256;
    gemm_f32_shares_kernel<<<(int)(blocks < 8u * sms ? blocks : 8u * sms), 256, 0, stream>>>(shares, y, n, used);
    return finish_launch("gemm_f32_shares");
}
