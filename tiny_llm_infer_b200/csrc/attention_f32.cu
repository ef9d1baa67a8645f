// Attention of prompt portions over the paged cache in true float32: tiles of 64 query rows and 64 keys, an online softmax
// between two matrix products on the float32 pipe.  Head widths 64 and 128.
//
// The general kernel (attention_general.cu) gives every (token, head) a block that reads all its keys and values again, a dot
// product per warp and key with a reduction for each: two prompts of 300 tokens with 16 heads on 8 of 128 took 250 us, this
// 76.  Here a thread owns 8 rows x 4 keys of the scores and 8 rows x HD / 16 columns of the output, so that a value read
// from shared memory serves four to eight products (packed, two per instruction; a score's even and odd elements are summed
// apart).  What bounds it is that pipe and the shared memory's reads, about equally, and with few tiles the longest block.
//
// Keys and values come by 16-byte cp.async; the next key tile is on its way while the present scores become weights and meet
// the values, the next value tile while the next scores are made.
#include "common.cuh"

namespace tllm {

constexpr int kTM = 64, kTN = 64, kF32Threads = 128;

__device__ __forceinline__ void f32_cp16(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0));
}

template <int HD>
struct F32Layout {
    static constexpr int kRow = HD + 4, kPRow = kTM + 4;        // padded rows: neighbouring rows' pieces lie in different banks
    static constexpr int kQ = 0, kK = kTM * kRow, kV = kK + kTN * kRow, kP = kV + kTN * HD, kFloats = kP + kTN * kPRow;
};

template <int HD>
__global__ void __launch_bounds__(kF32Threads)
paged_attention_f32_kernel(const float* q, const float* cache, const int* __restrict__ seg_info, const int* __restrict__ tiles,
                           const int* __restrict__ block_table, int max_pages, int page_size, int q_heads, int kv_heads, int window,
                           float scale, float* __restrict__ out) {
    using L = F32Layout<HD>;
    constexpr int kCols = HD / 64;                              // runs of four output columns per thread
    extern __shared__ __align__(16) float sm[];
    float *q_s = sm + L::kQ, *k_s = sm + L::kK, *v_s = sm + L::kV, *p_s = sm + L::kP;
    const int seg = tiles[2 * blockIdx.y], q_off = tiles[2 * blockIdx.y + 1], head = blockIdx.x;
    const int slot = seg_info[4 * seg], start = seg_info[4 * seg + 1], len = seg_info[4 * seg + 2], pos0 = seg_info[4 * seg + 3];
    const int rows_here = min(kTM, len - q_off), first_pos = pos0 + q_off, last_pos = first_pos + rows_here - 1;
    if (rows_here <= 0) return;
    if (slot < 0) {                                             // rows of no request, as in the general kernel
        for (int i = threadIdx.x; i < rows_here * HD; i += kF32Threads)
            out[((size_t)(start + q_off + i / HD) * q_heads + head) * HD + i % HD] = 0.0f;
        return;
    }
    const int g = head / (q_heads / kv_heads);
    const int* table = block_table + (size_t)slot * max_pages;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;     // keys tx + 16 i, rows 8 ty + r
    auto first_key = [&](int pos) { return window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0; };
    const int lo_all = first_key(first_pos), kt_first = lo_all / kTN, kt_last = last_pos / kTN;

    auto copy = [&](float* dst, int stride, int kt, int plane) {
        constexpr int kPieces = HD / 4;
        for (int i = threadIdx.x; i < kTN * kPieces; i += kF32Threads) {
            const int r = i / kPieces, c = (i % kPieces) * 4, key = kt * kTN + r;
            const int page = (key <= last_pos && key >= lo_all) ? table[key / page_size] : -1;
            const size_t row = (((size_t)(page < 0 ? 0 : page) * 2 + plane) * kv_heads + g) * page_size + key % page_size;
            f32_cp16(dst + r * stride + c, page < 0 ? cache : cache + row * HD + c, page >= 0);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    for (int i = threadIdx.x; i < kTM * (HD / 4); i += kF32Threads) {
        const int r = i / (HD / 4), c = (i % (HD / 4)) * 4;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < rows_here) x = *reinterpret_cast<const float4*>(q + ((size_t)(start + q_off + r) * q_heads + head) * HD + c);
        x.x *= scale; x.y *= scale; x.z *= scale; x.w *= scale;
        *reinterpret_cast<float4*>(q_s + r * L::kRow + c) = x;
    }
    copy(k_s, L::kRow, kt_first, 0);
    copy(v_s, HD, kt_first, 1);

    float m[8], l[8];
    float2 o[8][2 * kCols];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.0f;
#pragma unroll
        for (int c = 0; c < 2 * kCols; ++c) o[r][c] = make_float2(0.0f, 0.0f);
    }
    for (int kt = kt_first; kt <= kt_last; ++kt) {
        const int key0 = kt * kTN;
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the keys; the values may still be coming
        __syncthreads();
        float2 s[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[r][i] = make_float2(0.0f, 0.0f);
#pragma unroll 2
        for (int d = 0; d < HD; d += 4) {
            float4 k4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) k4[i] = *reinterpret_cast<const float4*>(k_s + (tx + 16 * i) * L::kRow + d);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float4 q4 = *reinterpret_cast<const float4*>(q_s + (ty * 8 + r) * L::kRow + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[r][i] = __ffma2_rn(make_float2(q4.x, q4.y), make_float2(k4[i].x, k4[i].y), s[r][i]);
                    s[r][i] = __ffma2_rn(make_float2(q4.z, q4.w), make_float2(k4[i].z, k4[i].w), s[r][i]);
                }
            }
        }
        __syncthreads();                                        // the keys have been read
        if (kt < kt_last) copy(k_s, L::kRow, kt + 1, 0);
        else asm volatile("cp.async.commit_group;\n" ::);
        const bool whole = key0 + kTN - 1 <= first_pos && key0 >= first_key(last_pos);
        float p[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int pos = first_pos + ty * 8 + r, lo = first_key(pos);
            float top = -INFINITY;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = key0 + tx + 16 * i;
                p[r][i] = whole || (key <= pos && key >= lo) ? s[r][i].x + s[r][i].y : -INFINITY;
                top = fmaxf(top, p[r][i]);
            }
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[r], top), m_use = m_new == -INFINITY ? 0.0f : m_new;
            const float corr = expf(m[r] - m_use);              // exp(-inf) = 0 before the first key
            m[r] = m_new;
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                p[r][i] = expf(p[r][i] - m_use);
                sum += p[r][i];
            }
            l[r] = l[r] * corr + sum;                           // of this thread's keys; the sixteen meet at the end
            const float2 c2 = make_float2(corr, corr);
#pragma unroll
            for (int c = 0; c < 2 * kCols; ++c) o[r][c] = __fmul2_rn(o[r][c], c2);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float4*>(p_s + (tx + 16 * i) * L::kPRow + ty * 8 + 4 * h) =
                    make_float4(p[4 * h][i], p[4 * h + 1][i], p[4 * h + 2][i], p[4 * h + 3][i]);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the values; the next keys may still be coming
        __syncthreads();
        auto meet = [&](int j, int row0, int row1) {            // key j with the thread's rows that see it
            const float4 pa = *reinterpret_cast<const float4*>(p_s + j * L::kPRow + ty * 8);
            const float4 pb = *reinterpret_cast<const float4*>(p_s + j * L::kPRow + ty * 8 + 4);
            const float w[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                const float4 v4 = *reinterpret_cast<const float4*>(v_s + j * HD + 64 * c + 4 * tx);
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    if (r < row0 || r > row1) continue;
                    const float2 w2 = make_float2(w[r], w[r]);
                    o[r][2 * c] = __ffma2_rn(w2, make_float2(v4.x, v4.y), o[r][2 * c]);
                    o[r][2 * c + 1] = __ffma2_rn(w2, make_float2(v4.z, v4.w), o[r][2 * c + 1]);
                }
            }
        };
        if (whole) {
#pragma unroll 4
            for (int j = 0; j < kTN; ++j) meet(j, 0, 7);
        } else {
            // a key that a row does not see is left out, not weighted by zero: its value may be infinite or no number
            const int pos = first_pos + ty * 8, lo = first_key(pos);
            for (int j = max(0, lo - key0); j < kTN && key0 + j <= pos + 7; ++j) {
                const int key = key0 + j;
                meet(j, key - pos, window > 0 ? key + window - 1 - pos : 7);
            }
        }
        __syncthreads();                                        // values and weights have been read
        if (kt < kt_last) copy(v_s, HD, kt + 1, 1);
        else asm volatile("cp.async.commit_group;\n" ::);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], x);
        const int row = ty * 8 + r;
        if (row >= rows_here) continue;
        const float inv = 1.0f / l[r];
        float* dst = out + ((size_t)(start + q_off + row) * q_heads + head) * HD;
#pragma unroll
        for (int c = 0; c < kCols; ++c)
            *reinterpret_cast<float4*>(dst + 64 * c + 4 * tx) =
                make_float4(o[r][2 * c].x * inv, o[r][2 * c].y * inv, o[r][2 * c + 1].x * inv, o[r][2 * c + 1].y * inv);
    }
}

template <int HD>
static int launch_f32(const float* q, const float* cache, const int* seg_info, const int* tiles, int n_tiles, const int* block_table,
                      int max_pages, int page_size, int q_heads, int kv_heads, int window, float scale, float* out, cudaStream_t stream) {
    constexpr size_t smem = F32Layout<HD>::kFloats * sizeof(float);
    static OncePerDevice configured;
    if (configured.first()) {
        cudaError_t e = cudaFuncSetAttribute(paged_attention_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { set_error("paged_attention_f32: %s", cudaGetErrorString(e)); return (int)e; }
        configured.done();
    }
    paged_attention_f32_kernel<HD><<<dim3(q_heads, n_tiles), kF32Threads, smem, stream>>>(
        q, cache, seg_info, tiles, block_table, max_pages, page_size, q_heads, kv_heads, window, scale, out);
    return finish_launch("paged_attention_f32");
}

}  // namespace tllm

using namespace tllm;

// q, out [tokens, q_heads * head_dim], cache [pages, 2, kv_heads, page_size, head_dim], float32, 16-byte aligned; tiles
// int[n_tiles][2] = segment, offset of 64 query rows.
extern "C" int tllm_paged_attention_f32(const float* q, const float* cache, const int* seg_info, const int* tiles, int n_tiles,
                                        const int* block_table, int max_pages, int page_size, int q_heads, int kv_heads, int head_dim,
                                        int window, float scale, float* out, cudaStream_t stream) {
    TLLM_REQUIRE(q_heads > 0 && kv_heads > 0 && q_heads % kv_heads == 0, "paged_attention_f32: %d query heads over %d key/value heads", q_heads, kv_heads);
    TLLM_REQUIRE(head_dim == 64 || head_dim == 128, "paged_attention_f32: head_dim %d", head_dim);
    TLLM_REQUIRE(page_size > 0 && max_pages > 0 && n_tiles >= 0 && n_tiles <= 65535, "paged_attention_f32: bad sizes");
    TLLM_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0,
                 "paged_attention_f32: operands must be 16-byte aligned");
    if (n_tiles == 0) return 0;
    if (head_dim == 128)
        return launch_f32<128>(q, cache, seg_info, tiles, n_tiles, block_table, max_pages, page_size, q_heads, kv_heads, window, scale, out, stream);
    return launch_f32<64>(q, cache, seg_info, tiles, n_tiles, block_table, max_pages, page_size, q_heads, kv_heads, window, scale, out, stream);
}
