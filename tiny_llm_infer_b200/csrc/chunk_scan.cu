// The recurrences of delta_rule.cu over prompt portions, sixteen tokens at a time.
//
// The scan kernel there walks a portion token by token: a token's read-out and, with a correction, its update wait for the
// token before, some 550 cycles each (2048 tokens of 32 heads of 128 x 128: 577 us for the delta rule, a fifth of what the
// float32 pipe could do).  Inside a chunk of C = 16 tokens the same sums can be written without that chain.  With G_ij =
// the product of the decays of the tokens j + 1 .. i (per key channel, per head, or a constant per head) and S the state
// before the chunk,
//
//   x_i = (G_i,-1 k_i)^T S,   o_i = (G_i,-1 q_i)^T S + sum_{j <= i} Q_ij u_j,   S <- G_C,-1 S + sum_j (G_Cj k_j) u_j^T,
//   u_i = beta_i (v_i - x_i - sum_{j < i} A_ij u_j)   (the delta rule), or w_i v_i,
//   A_ij = k_i^T G_ij k_j,   Q_ij = q_i^T G_ij k_j,
//
// and the delta rule's u come from one triangular 16 x 16 matrix, u = T (v - x) with T = (1 + diag(beta) A)^-1 diag(beta),
// which the columns of a head share; its read-outs from Q T, o_i = .. + sum_j (Q T)_ij (v - x)_j.  So the state is read twice
// and written once per sixteen tokens, as small matrix products.  Every G is a product of decays, made by multiplying them up from
// either side; nothing is divided and no exponential of a sum is taken, so the results are as exact as the token's way.
//
//   chunk_pairs  one warp per (chunk, head): T and Q T, or Q, the decays from the chunk's start and the write weights
//                (chunk_scalar_pairs where the decays are per head: one warp per chunk and key head).
//   chunk_scan   one block per (portion, head, 32 or 16 columns): the state in the registers of four warps, its products on the
//                tensor cores with every float32 operand in three bfloat16 parts.
//
// The layout of the request's state is the scan kernel's (row r * per + il of column j at [il][j][r]).
#include "common.cuh"
#include "mma_tiles.cuh"

namespace tllm {

constexpr int kC = 16;                         // tokens of a chunk
constexpr int kPairFloats = 2 * kC * kC;       // T and Q T, or the scalars and Q, of one (chunk, head)

// What the sums need of a recurrence.  kDelta: decays per channel and the correction; kChannel: decays per channel, u = w v
// (w = 1 where `beta` is null); kHead: one decay per (token, head) in `beta`, w in `fgate`; kFixed: one decay per head in
// `fgate`, w = 1.
enum ChunkKind : int { kDelta = 0, kChannel = 1, kHead = 2, kFixed = 3 };

// Chunk c of a portion is entry first + c of the pairs, first = start / 16 + the portions that start before it (whatever
// their order in seg_info); entries that no chunk has stay unused.  Called by all threads of a block.
__device__ __forceinline__ int first_entry(const int* seg_info, int segments, int seg) {
    const int start = seg_info[4 * seg + 1];
    int before = 0;
    for (int base = 0; base < segments; base += blockDim.x) {
        const int s = base + threadIdx.x;
        const int at = s < segments ? seg_info[4 * s + 1] : 0x7fffffff;
        before += __syncthreads_count(at < start || (at == start && s < seg));
    }
    return start / kC + before;
}

__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }

// Sums over the warp of N values per lane (N = 16 or 32), by exchanging halves: value n ends in lane n (N = 16: in lanes
// n and n + 16).
template <int N>
__device__ __forceinline__ float halves_sum(float (&v)[N], int lane) {
#pragma unroll
    for (int half = N / 2; half > 0; half >>= 1) {
        const bool up = lane & half;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
        }
    }
    return N == 16 ? v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16) : v[0];
}

// The left operand of one step of sixteen terms from two tiles of accumulators.
__device__ __forceinline__ void split_left(const float (&t0)[4], const float (&t1)[4], uint32_t (&a)[3][4]) {
    split3(t0[0], t0[1], a[0][0], a[1][0], a[2][0]);
    split3(t0[2], t0[3], a[0][1], a[1][1], a[2][1]);
    split3(t1[0], t1[1], a[0][2], a[1][2], a[2][2]);
    split3(t1[2], t1[3], a[0][3], a[1][3], a[2][3]);
}

// d[k] = a[k / PER] . (tile k of the tiles in b, two to a b) over sixteen terms each, N products side by side: each is a chain of six
// dependent mma, and four or more chains keep the tensor pipe busy where one waits four times as long as it works.
template <int N, int PER, int NA, int NB>
__device__ __forceinline__ void products3(float (&d)[N][4], const uint32_t (&a)[NA][3][4], const uint32_t (&b)[NB][3][4]) {
    constexpr int kLeft[6] = {2, 0, 1, 1, 0, 0}, kRight[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
    for (int k = 0; k < N; ++k) d[k][0] = d[k][1] = d[k][2] = d[k][3] = 0.0f;
#pragma unroll
    for (int s = 0; s < 6; ++s)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t bt[2] = {b[k / 2][kRight[s]][2 * (k % 2)], b[k / 2][kRight[s]][2 * (k % 2) + 1]};
            mma_bf16_16816(d[k], a[k / PER][kLeft[s]], bt);
        }
}

// Decays per channel.  DK 128: a lane has four neighbouring channels; DK 64: the upper sixteen lanes carry zeros.
template <int DK, int KIND>
__global__ void __launch_bounds__(128)
chunk_pairs_kernel(const int* __restrict__ seg_info, int segments, const float* qn, const float* kn, const float* decay, const float* beta,
                   int heads, int kv_heads, float* pairs) {
    static_assert(KIND == kDelta || KIND == kChannel, "one decay per head: chunk_scalar_pairs_kernel");
    constexpr bool kCorr = KIND == kDelta;
    const int seg = blockIdx.y, slot = seg_info[4 * seg], start = seg_info[4 * seg + 1], len = seg_info[4 * seg + 2];
    const int first = first_entry(seg_info, segments, seg);
    const int lane = threadIdx.x & 31, head = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (head >= heads || slot < 0) return;
    const int kvh = head / (heads / kv_heads), col = lane & 15;                 // this lane's j
    const bool live = lane * 4 < DK;
    const float4 zero = make_float4(0, 0, 0, 0), one = make_float4(1, 1, 1, 1);
    for (int c0 = blockIdx.z * kC; c0 < len; c0 += gridDim.z * kC) {
        const int n = min(kC, len - c0);
        float* T = pairs + ((size_t)(first + c0 / kC) * heads + head) * kPairFloats;
        float* Q = T + kC * kC;
        auto at = [&](const float* p, int i, int h, int hs) -> float4 {
            return live ? *reinterpret_cast<const float4*>(p + ((size_t)(start + c0 + i) * hs + h) * DK + lane * 4) : zero;
        };
        const float w_own = col < n && beta != nullptr ? beta[(size_t)(start + c0 + col) * heads + head] : 1.0f;     // of token `col`
        float4 w[kC];                                               // k_j, decayed up to the token at hand
        float4 q4[4], g4[4];                                        // the next four tokens' q and decays
        float trow[kC];                                             // column `col` of T
#pragma unroll
        for (int i = 0; i < kC; ++i) w[i] = i < n ? at(kn, i, kvh, kv_heads) : zero;
#pragma unroll
        for (int i = 0; i < kC; ++i) {
            if (i % 4 == 0)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    q4[e] = i + e < n ? at(qn, i + e, kvh, kv_heads) : zero;
                    g4[e] = i + e < n ? at(decay, i + e, head, heads) : one;
                }
            const float4 k = w[i], q = q4[i % 4];                   // w[i] has no decay on it yet
            float s;                                                // lane j: Q_ij; with the correction lane 16 + j: A_ij
#pragma unroll
            for (int j = 0; j < i; ++j) w[j] = mul4(w[j], g4[i % 4]);
            if (kCorr) {
                float v[32];
#pragma unroll
                for (int j = 0; j < kC; ++j) {
                    v[j] = j <= i ? dot4(q, w[j]) : 0.0f;
                    v[16 + j] = j < i ? dot4(k, w[j]) : 0.0f;
                }
                s = halves_sum<32>(v, lane);
                // row i of T: beta_i (e_i - sum_j A_ij T_j), column `col` in both halves of the warp
                const float b = __shfl_sync(0xffffffffu, w_own, i);
                float acc = col == i ? 1.0f : 0.0f;
#pragma unroll
                for (int j = 0; j < i; ++j) acc = fmaf(-__shfl_sync(0xffffffffu, s, 16 + j), trow[j], acc);
                trow[i] = b * acc;
                float qt = 0.0f;                                    // row i of Q T
#pragma unroll
                for (int j = 0; j <= i; ++j) qt = fmaf(__shfl_sync(0xffffffffu, s, j), trow[j], qt);
                if (lane < 16) {
                    T[i * kC + col] = trow[i];
                    Q[i * kC + col] = qt;
                }
            } else {
                float v[16];
#pragma unroll
                for (int j = 0; j < kC; ++j) v[j] = j <= i ? dot4(q, w[j]) : 0.0f;
                s = halves_sum<16>(v, lane);
                if (lane == 0) T[i] = 1.0f;
                // of a later token nothing, not zero times its weight: that may be infinite or no number
                if (lane < 16) Q[i * kC + col] = col <= i ? s * w_own : 0.0f;
            }
        }
        if (!kCorr && lane < 16) T[kC + col] = w_own;               // row 1: what token j's values are multiplied by in the state
    }
}

// One decay per head: Q_ij = w_j d_ij q_i^T k_j, where the products of a chunk's queries and keys are the same for all heads of a
// key and d_ij is the product of the decays j + 1 .. i.  One warp per (chunk, key head): q and k straight from memory in the
// operands' layout, and their product on the tensor cores as in the scan below.  Bound by reading q and k (2048 tokens, 32 heads
// of 128: 67 MB).
template <int DK, int KIND>
__global__ void __launch_bounds__(128)
chunk_scalar_pairs_kernel(const int* __restrict__ seg_info, int segments, const float* qn, const float* kn, const float* beta,
                          const float* fgate, int heads, int kv_heads, float* pairs) {
    const int seg = blockIdx.y, slot = seg_info[4 * seg], start = seg_info[4 * seg + 1], len = seg_info[4 * seg + 2];
    const int first = first_entry(seg_info, segments, seg);
    const int lane = threadIdx.x & 31, kvh = blockIdx.x * 4 + (threadIdx.x >> 5), rep = heads / kv_heads;
    if (kvh >= kv_heads || slot < 0) return;
    const int row = lane >> 2, two = (lane & 3) * 2, col = lane & 15;
    for (int c0 = blockIdx.z * kC; c0 < len; c0 += gridDim.z * kC) {
        const int n = min(kC, len - c0);
        const size_t at = ((size_t)(start + c0) * kv_heads + kvh) * DK + two;
        auto load = [&](const float* p, int i, int ch) -> float2 {
            return i < n ? *reinterpret_cast<const float2*>(p + at + (size_t)i * kv_heads * DK + ch) : make_float2(0.0f, 0.0f);
        };
        float s[2][4];                                              // q_i^T k_j: rows i of the lane, row and row + 8; tiles of eight j
        constexpr int kAhead = 4;                                   // steps of sixteen channels whose loads are on their way at once
        float2 q[kAhead][4], k[kAhead][4];
#pragma unroll
        for (int ks = 0; ks < DK / 16; ++ks) {
            if (ks % kAhead == 0)
#pragma unroll
                for (int m = 0; m < kAhead; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        q[m][e] = load(qn, row + (e & 1) * 8, (ks + m) * 16 + (e >> 1) * 8);
                        k[m][e] = load(kn, row + (e >> 1) * 8, (ks + m) * 16 + (e & 1) * 8);
                    }
            uint32_t a[1][3][4], b[1][3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x = q[ks % kAhead][e], y = k[ks % kAhead][e];
                split3(x.x, x.y, a[0][0][e], a[0][1][e], a[0][2][e]);
                split3(y.x, y.y, b[0][0][e], b[0][1][e], b[0][2][e]);
            }
            float d[2][4];
            products3<2, 2>(d, a, b);
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[t][e] = ks == 0 ? d[t][e] : s[t][e] + d[t][e];
        }
        for (int h = 0; h < rep; ++h) {
            const int head = kvh * rep + h;
            float a_own = 1.0f, w_own = 1.0f;                       // token `col`'s decay and the weight of its values
            if (col < n) {
                const size_t t = (size_t)(start + c0 + col) * heads + head;
                if (KIND == kHead) { a_own = beta[t]; w_own = fgate[t]; }
                else a_own = fgate[head];
            }
            float d[2][4], since = 1.0f, after = 1.0f;              // of the lane's (i, j); from the chunk's start to `col`; after it
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) d[t][e] = 1.0f;
#pragma unroll
            for (int m = 0; m < kC; ++m) {
                const float a = __shfl_sync(0xffffffffu, a_own, m);
                if (m <= col) since *= a;
                else after *= a;
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (m > t * 8 + two + (e & 1) && m <= row + (e >> 1) * 8) d[t][e] *= a;
            }
            float* T = pairs + ((size_t)(first + c0 / kC) * heads + head) * kPairFloats;
            float* Q = T + kC * kC;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int j = t * 8 + two;
                const float w0 = __shfl_sync(0xffffffffu, w_own, j), w1 = __shfl_sync(0xffffffffu, w_own, j + 1);
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const int i = row + (e >> 1) * 8;
                    // of a later token nothing, not zero times its weight: that may be infinite or no number
                    *reinterpret_cast<float2*>(Q + i * kC + j) = make_float2(j <= i ? s[t][e] * d[t][e] * w0 : 0.0f, j + 1 <= i ? s[t][e + 1] * d[t][e + 1] * w1 : 0.0f);
                }
            }
            if (lane < 16) {                                        // row 0: the decays since the chunk's start; row 1: what token
                T[col] = since;                                     // j's values are multiplied by in the state
                T[kC + col] = w_own * after;
            }
        }
    }
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0));
}

// ---------------------------------------------------------------- the scan over the chunks
// All three products of a chunk (the read-outs S^T k and S^T q, the sums with T and Q T, the update u k^T) run on
// mma.sync m16n8k16 with every float32 operand as the exact-to-2^-24 sum of three bfloat16 parts: a product is six mma, the
// parts' products down to 2^-18 of the largest (what is left out is below 2^-26), smallest first, started from zero for every
// sixteen terms and then added to the running float32 sum, which keeps the tensor core's cut-off sums out of long chains.  The
// state lies transposed in the accumulators' layout ([columns][keys], 16 columns and DK / kParts keys per warp), which is at
// once the layout of the left operand of the read-outs; u comes out of T's product as the left operand of the update; so
// nothing but the warps' partial read-outs, which meet over the parts of the keys, passes through shared memory.
//
// Warps of their own split the tokens a chunk ahead, a thread per pair of channels of one operand; others fetch them.
//
// What bounds it: a chunk takes a block 2300 (one decay per head) to 3300 cycles (the delta rule), of which 880 to 1450 are mma (8.6
// cycles each and scheduler); the rest is the chain from the read-outs over the meeting of the parts and T to the update, and the
// splitting of the state.  Eight warps with half the keys each (273 to 296 us for the delta rule), the parts' meeting prefetched
// around (280) and operands split once by the pairs' kernel into 44 KB records per chunk and head (267, for 180 MB of scratch) did
// not shorten it.  Before, on the float32 pipe with a lane per 8 rows of 4 columns (two fused multiply-adds per instruction), and
// now, with the pairs: 2048 tokens of 32 heads of 128 x 128, delta rule 386 and 273 us, one decay per head 245 and 183; 16 heads 237
// and 204, 179 and 140; 64 heads of 128 x 64, 1023 tokens, one decay per head 140 and 108.  The error against 64 bits is no larger
// (products to 2^-26, sums of sixteen terms added in float32).
constexpr int kMatRow = 24;                    // bfloat16 elements of a row of T or Q in shared memory
constexpr float kLargest = 3.38e38f;           // beyond it the first part would be an infinity

// LIGHT: fewer helping warps and less fetched ahead, so that two blocks share a multiprocessor (recurrences of one decay per head).
template <int DK, int KIND, int COLS, bool LIGHT>
struct ChunkLayout {
    static constexpr bool kVec = KIND == kDelta || KIND == kChannel, kCorr = KIND == kDelta;
    static constexpr int kTiles = COLS / 16, kParts = 4 / kTiles, kKeys = DK / kParts;    // warps: column tiles x parts of the keys
    static constexpr int kArrays = kCorr ? 3 : 2, kMats = kCorr ? 2 : 1;
    static constexpr int kSplitters = (LIGHT ? 1 : kArrays) * DK / 2, kLoaders = LIGHT ? 32 : 64, kThreads = 128 + kSplitters + kLoaders;
    static constexpr int kSplit = kC * DK * 2, kMat = kC * kMatRow * 2;                  // bytes of one part of an operand
    static constexpr int kMatAt = kArrays * 3 * kSplit, kGamAt = kMatAt + kMats * 3 * kMat, kStage = kGamAt + (kVec ? DK * 4 : 0);
    static constexpr int kRaw = (kVec ? 3 : 2) * kC * DK * 4;
    static constexpr int kVRow = COLS + 4, kRing = kC * kVRow * 4 + kPairFloats * 4;
    static constexpr int kRaws = LIGHT ? 2 : 3;                                           // chunks fetched and not yet split
    static constexpr int kRawAt = 2 * kStage, kRingAt = kRawAt + kRaws * kRaw, kSumsAt = kRingAt + 4 * kRing;
    static constexpr int kBytes = kSumsAt + 4 * 16 * 32 * 4;
    static constexpr int kBlocks = kBytes <= 113 * 1024 ? 2 : 1;                         // per SM
};

template <int DK, int KIND, int COLS, bool LIGHT>
__global__ void __launch_bounds__(ChunkLayout<DK, KIND, COLS, LIGHT>::kThreads, ChunkLayout<DK, KIND, COLS, LIGHT>::kBlocks)
chunk_scan_kernel(const int* __restrict__ seg_info, const float* qn, const float* kn, const float* vv, const float* decay,
                  const float* pairs, float* state, long long state_stride, int segments, int heads, int kv_heads, int dv, float* o_raw) {
    using L = ChunkLayout<DK, KIND, COLS, LIGHT>;
    constexpr bool kVec = L::kVec, kCorr = L::kCorr;
    extern __shared__ __align__(16) unsigned char sm[];
    const int seg = blockIdx.y, groups = dv / COLS, head = blockIdx.x / groups, col0 = blockIdx.x % groups * COLS;
    const int slot = seg_info[4 * seg], start = seg_info[4 * seg + 1], len = seg_info[4 * seg + 2];
    const int first = first_entry(seg_info, segments, seg);
    if (slot < 0 || len <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kvh = head / (heads / kv_heads);
    const int chunks = (len + kC - 1) / kC;
    // byte of channel ch of token i in one part of an operand: 16-byte pieces, exchanged so that eight rows lie in eight banks
    auto at = [](int i, int piece) { return i * (DK * 2) + ((piece ^ (i & 7)) << 4); };

    if (warp >= 4 + L::kSplitters / 32) {                       // fetch the tokens two or three chunks ahead, split T and Q T
        const int me = threadIdx.x - 128 - L::kSplitters;
        auto issue = [&](int c) {                               // one group of copies a call, an empty one past the end
            if (c >= chunks) {
                asm volatile("cp.async.commit_group;\n" ::);
                return;
            }
            const int c0 = c * kC, n = min(kC, len - c0);
            float* raw = reinterpret_cast<float*>(sm + L::kRawAt + c % L::kRaws * L::kRaw);
            float* v = reinterpret_cast<float*>(sm + L::kRingAt + (c & 3) * L::kRing);
            constexpr int kPieces = DK / 4, kVPieces = COLS / 4;
            const int e = me % kPieces * 4, ve = me % kVPieces * 4;
            const float* q = qn + ((size_t)(start + c0) * kv_heads + kvh) * DK + e;
            const float* k = kn + ((size_t)(start + c0) * kv_heads + kvh) * DK + e;
            const float* g = kVec ? decay + ((size_t)(start + c0) * heads + head) * DK + e : nullptr;
            const float* x = vv + ((size_t)(start + c0) * heads + head) * dv + col0 + ve;
#pragma unroll
            for (int s = 0; s < kC * kPieces / L::kLoaders; ++s) {
                const int t = me / kPieces + s * (L::kLoaders / kPieces), from = t < n ? t : 0;
                cp16(raw + t * DK + e, q + (size_t)from * kv_heads * DK, t < n);
                cp16(raw + (kC + t) * DK + e, k + (size_t)from * kv_heads * DK, t < n);
                if (kVec) cp16(raw + (2 * kC + t) * DK + e, g + (size_t)from * heads * DK, t < n);
            }
#pragma unroll
            for (int s = 0; s < kC * kVPieces / L::kLoaders; ++s) {
                const int t = me / kVPieces + s * (L::kLoaders / kVPieces), from = t < n ? t : 0;
                cp16(v + t * L::kVRow + ve, x + (size_t)from * heads * dv, t < n);
            }
            const float* p = pairs + ((size_t)(first + c) * heads + head) * kPairFloats;
#pragma unroll
            for (int i = 0; i < kPairFloats / 4; i += L::kLoaders) cp16(v + kC * L::kVRow + (i + me) * 4, p + (i + me) * 4, true);
            asm volatile("cp.async.commit_group;\n" ::);
        };
        auto split_mats = [&](int c) {
            constexpr int kEach = L::kMats * kC * kC / 2 / L::kLoaders;
            const float* mats = reinterpret_cast<const float*>(sm + L::kRingAt + (c & 3) * L::kRing) + kC * L::kVRow + (kCorr ? 0 : kC * kC);
            unsigned char* to = sm + (c & 1) * L::kStage + L::kMatAt;
            float2 x[kEach];
#pragma unroll
            for (int s = 0; s < kEach; ++s) x[s] = *reinterpret_cast<const float2*>(mats + (me + s * L::kLoaders) * 2);
#pragma unroll
            for (int s = 0; s < kEach; ++s) {
                const int i = me + s * L::kLoaders, mat = i / (kC * kC / 2), row = i % (kC * kC / 2) / (kC / 2), e = i % (kC / 2) * 2;
                uint32_t h, m, l;
                split3(x[s].x, x[s].y, h, m, l);
                unsigned char* at_row = to + mat * 3 * L::kMat + (row * kMatRow + e) * 2;
                *reinterpret_cast<uint32_t*>(at_row) = h;
                *reinterpret_cast<uint32_t*>(at_row + L::kMat) = m;
                *reinterpret_cast<uint32_t*>(at_row + 2 * L::kMat) = l;
            }
        };
#pragma unroll
        for (int c = 0; c < L::kRaws - 1; ++c) issue(c);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(L::kRaws - 2) : "memory");
        __syncthreads();                                        // chunk 0 is here
        issue(L::kRaws - 1);
        for (int c = 0; c <= chunks; ++c) {
            if (c < chunks) split_mats(c);
            asm volatile("cp.async.wait_group %0;\n" ::"n"(L::kRaws - 2) : "memory");
            __syncthreads();                                    // chunk c is ready, chunk c + 1 here, chunk c - 1 done with
            issue(c + L::kRaws);
        }
        return;
    }
    if (warp >= 4) {                                            // split the tokens of chunk c while chunk c - 1 is consumed
        const int me = threadIdx.x - 128, ch = me % (DK / 2) * 2;
        // operand 0: q with the decays since the chunk's start on it, 1: k with those up to its end, 2: k as q
        __syncthreads();
        for (int c = 0; c <= chunks; ++c) {
            for (int array = me / (DK / 2); c < chunks && array < L::kArrays; array += L::kSplitters / (DK / 2)) {
                const int n = min(kC, len - c * kC);
                const float* raw = reinterpret_cast<const float*>(sm + L::kRawAt + c % L::kRaws * L::kRaw);
                const float* src = raw + (array == 0 ? 0 : kC * DK) + ch;
                unsigned char* stage = sm + (c & 1) * L::kStage;
                unsigned char* dst = stage + array * 3 * L::kSplit + (ch & 7) * 2;
                float2 p = make_float2(1.0f, 1.0f);
                // several tokens' loads before the first store: the chains of a token's three parts overlap
                constexpr int kBatch = 8;
                auto batch = [&](int first_token, int step) {
                    float2 x[kBatch], g[kBatch];
#pragma unroll
                    for (int s = 0; s < kBatch; ++s) {
                        x[s] = *reinterpret_cast<const float2*>(src + (first_token + s * step) * DK);
                        if (kVec) g[s] = *reinterpret_cast<const float2*>(raw + (2 * kC + first_token + s * step) * DK + ch);
                    }
                    uint32_t h[kBatch], m[kBatch], l[kBatch];
#pragma unroll
                    for (int s = 0; s < kBatch; ++s) {
                        if (kVec) {
                            if (first_token + s * step >= n) g[s] = make_float2(1.0f, 1.0f);
                            const float2 after = make_float2(p.x * g[s].x, p.y * g[s].y);
                            if (step > 0) p = after;
                            x[s].x *= p.x, x[s].y *= p.y;
                            p = after;
                        }
                        split3(x[s].x, x[s].y, h[s], m[s], l[s]);
                    }
#pragma unroll
                    for (int s = 0; s < kBatch; ++s) {
                        unsigned char* to = dst + at(first_token + s * step, ch >> 3);
                        *reinterpret_cast<uint32_t*>(to) = h[s];
                        *reinterpret_cast<uint32_t*>(to + L::kSplit) = m[s];
                        *reinterpret_cast<uint32_t*>(to + 2 * L::kSplit) = l[s];
                    }
                };
                if (kVec && array == 1) {
                    batch(kC - 1, -1);
                    batch(kC - 1 - kBatch, -1);
                } else {
                    batch(0, 1);
                    batch(kBatch, 1);
                    if (kVec && array == 0) *reinterpret_cast<float2*>(stage + L::kGamAt + ch * 4) = p;
                }
            }
            __syncthreads();
        }
        return;
    }
    const int tile = warp % L::kTiles, part = warp / L::kTiles, key0 = part * L::kKeys;
    const int row = lane >> 2, two = (lane & 3) * 2, mid = lane >> 3, mrow = lane & 7;
    const int mine = tile * 16 + row;                           // the lane's first column of the block's, the other is 8 further
    // row i of the state lies at [i % per][column][i / per]
    constexpr int kR = DK <= 64 ? 4 : 8, kPer = DK / kR;
    float* st_ptr = state + (long long)slot * state_stride + (size_t)head * DK * dv;
    auto state_at = [&](int t, int e) -> float& {
        const int i = key0 + t * 8 + two + (e & 1);
        return st_ptr[((size_t)(i % kPer) * dv + col0 + mine + (e >> 1) * 8) * kR + i / kPer];
    };
    float S[L::kKeys / 8][4];
#pragma unroll
    for (int t = 0; t < L::kKeys / 8; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[t][e] = state_at(t, e);
    float* sums = reinterpret_cast<float*>(sm + L::kSumsAt) + lane;                         // [warp][value][lane]

    __syncthreads();
    __syncthreads();                                            // the first chunk is ready
    for (int c = 0; c < chunks; ++c) {
        const int n = min(kC, len - c * kC);
        const uint32_t stage = smem_u32(sm + (c & 1) * L::kStage);
        const float* V = reinterpret_cast<const float*>(sm + L::kRingAt + (c & 3) * L::kRing);
        const float* T = V + kC * L::kVRow;                     // float32: T and Q T, or the scalars and Q
        // read-outs of the state before the chunk over this warp's keys: tiles of eight tokens of q, and of k
        constexpr int kRead = kCorr ? 2 : 1;                    // operands read out: q, and k
        constexpr int kAtOnce = L::kKeys / 16 >= 2 ? 2 : 1;     // steps of sixteen keys
        float x[2 * kRead][4];
#pragma unroll
        for (int ks = 0; ks < L::kKeys / 16; ks += kAtOnce) {
            uint32_t a[kAtOnce][3][4], b[kAtOnce * kRead][3][4];
            float d[2 * kAtOnce * kRead][4];
#pragma unroll
            for (int k = 0; k < kAtOnce; ++k) {
#pragma unroll
                for (int w = 0; w < kRead; ++w)
#pragma unroll
                    for (int s = 0; s < 3; ++s)
                        ldmatrix_x4(b[k * kRead + w][s], stage + ((w == 0 ? 0 : 2) * 3 + s) * L::kSplit + at((mid >> 1) * 8 + mrow, key0 / 8 + 2 * (ks + k) + (mid & 1)));
                split_left(S[2 * (ks + k)], S[2 * (ks + k) + 1], a[k]);
            }
            products3<2 * kAtOnce * kRead, 2 * kRead>(d, a, b);
#pragma unroll
            for (int k = 0; k < kAtOnce; ++k)
#pragma unroll
                for (int t = 0; t < 2 * kRead; ++t)
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[t][e] = ks + k == 0 ? d[t][e] : x[t][e] + d[k * 2 * kRead + t][e];
        }
        // the parts' sums meet, added in the parts' order by all of them; a warp needs those of k and its own tile of q
#pragma unroll
        for (int t = 0; t < 2 * kRead; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) sums[(warp * 16 + t * 4 + e) * 32] = x[t][e];
        asm volatile("bar.sync %0, %1;\n" ::"r"(2 + tile), "n"(L::kParts * 32) : "memory");
        float o[4], y[2][4], u[2][4];
        auto met = [&](int t, int e) {
            float v = sums[(tile * 16 + t * 4 + e) * 32];
#pragma unroll
            for (int p = 1; p < L::kParts; ++p) v += sums[((p * L::kTiles + tile) * 16 + t * 4 + e) * 32];
            return v;
        };
        const int mt = part & 1;                                // its tile of tokens to read out (parts 0 and 1)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = met(mt, e);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[t][e] = V[(t * 8 + two + (e & 1)) * L::kVRow + mine + (e >> 1) * 8];
                if (kCorr) y[t][e] -= met(2 + t, e);
            }
        // A later token's value must not reach an earlier read-out through its weight of zero: infinities and values that
        // are no numbers are left out of the products and brought in one by one.
        bool odd = false;
        float clean[2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool fine = fabsf(y[t][e]) <= kLargest;
                odd |= !fine;
                clean[t][e] = fine ? y[t][e] : 0.0f;
            }
        odd = __any_sync(0xffffffffu, odd);
        {
            uint32_t a[1][3][4], b[L::kMats][3][4];             // T's two tiles of tokens and this warp's of Q T, or that of Q
            const uint32_t mats = stage + L::kMatAt + (((mid >> 1) * 8 + mrow) * kMatRow + (mid & 1) * 8) * 2;
#pragma unroll
            for (int m = 0; m < L::kMats; ++m)
#pragma unroll
                for (int s = 0; s < 3; ++s) ldmatrix_x4(b[m][s], mats + (m * 3 + s) * L::kMat);
            if (mt) {
#pragma unroll
                for (int s = 0; s < 3; ++s) b[L::kMats - 1][s][0] = b[L::kMats - 1][s][2], b[L::kMats - 1][s][1] = b[L::kMats - 1][s][3];
            }
            split_left(clean[0], clean[1], a[0]);
            float d[kCorr ? 3 : 1][4];
            products3<kCorr ? 3 : 1, 3>(d, a, b);
            if (kCorr) {
#pragma unroll
                for (int e = 0; e < 4; ++e) u[0][e] = d[0][e], u[1][e] = d[kCorr ? 1 : 0][e];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = kCorr ? o[e] + d[kCorr ? 2 : 0][e] : fmaf(o[e], T[mt * 8 + two + (e & 1)], d[0][e]);
        }
        if (!kCorr) {
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) u[t][e] = T[kC + t * 8 + two + (e & 1)] * y[t][e];
        }
        if (odd) {
#pragma unroll
            for (int j = 0; j < kC; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {                   // the lane's two columns
                    const float yj = __shfl_sync(0xffffffffu, y[j / 8][2 * h + (j & 1)], (lane & ~3) | (j & 7) >> 1);
                    if (fabsf(yj) <= kLargest) continue;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
#pragma unroll
                        for (int t = 0; t < 2; ++t)
                            if (kCorr && t * 8 + two + e >= j) u[t][2 * h + e] = fmaf(T[(t * 8 + two + e) * kC + j], yj, u[t][2 * h + e]);
                        if (mt * 8 + two + e >= j) o[2 * h + e] = fmaf(T[kC * kC + (mt * 8 + two + e) * kC + j], yj, o[2 * h + e]);
                    }
                }
        }
        if (part < 2) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = mt * 8 + two + (e & 1);
                if (i < n) o_raw[((size_t)(start + c * kC + i) * heads + head) * dv + col0 + mine + (e >> 1) * 8] = o[e];
            }
        }
        // the state moves on
        uint32_t ua[1][3][4];
        split_left(u[0], u[1], ua[0]);
#pragma unroll
        for (int ks = 0; ks < L::kKeys / 16; ks += kAtOnce) {
            uint32_t b[kAtOnce][3][4];
            float d[2 * kAtOnce][4];
#pragma unroll
            for (int k = 0; k < kAtOnce; ++k)
#pragma unroll
                for (int s = 0; s < 3; ++s)
                    ldmatrix_x4_trans(b[k][s], stage + (3 + s) * L::kSplit + at((mid & 1) * 8 + mrow, key0 / 8 + 2 * (ks + k) + (mid >> 1)));
            products3<2 * kAtOnce, 2 * kAtOnce>(d, ua, b);
#pragma unroll
            for (int t = 0; t < 2 * kAtOnce; ++t) {
                float2 g;
                if (kVec) g = *reinterpret_cast<const float2*>(sm + (c & 1) * L::kStage + L::kGamAt + (key0 + (2 * ks + t) * 8 + two) * 4);
                else g.x = g.y = T[kC - 1];
                float (&St)[4] = S[2 * ks + t];
                St[0] = fmaf(St[0], g.x, d[t][0]), St[1] = fmaf(St[1], g.y, d[t][1]);
                St[2] = fmaf(St[2], g.x, d[t][2]), St[3] = fmaf(St[3], g.y, d[t][3]);
            }
        }
        __syncthreads();                                        // chunk c is done with, chunk c + 1 ready
    }
#pragma unroll
    for (int t = 0; t < L::kKeys / 8; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) state_at(t, e) = S[t][e];
}

template <int DK, int KIND, int COLS, bool LIGHT>
static int launch_chunk_scan(const int* seg_info, int segments, const float* qn, const float* kn, const float* vv, const float* decay,
                             const float* pairs, float* state, long long state_stride, int heads, int kv_heads, int dv, float* o_raw,
                             cudaStream_t stream) {
    using L = ChunkLayout<DK, KIND, COLS, LIGHT>;
    static OncePerDevice configured;
    if (configured.first()) {
        cudaError_t e = cudaFuncSetAttribute(chunk_scan_kernel<DK, KIND, COLS, LIGHT>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes);
        if (e != cudaSuccess) { set_error("chunk_scan: %s", cudaGetErrorString(e)); return (int)e; }
        configured.done();
    }
    chunk_scan_kernel<DK, KIND, COLS, LIGHT><<<dim3(heads * (dv / COLS), segments), L::kThreads, L::kBytes, stream>>>(
        seg_info, qn, kn, vv, decay, pairs, state, state_stride, segments, heads, kv_heads, dv, o_raw);
    return finish_launch("chunk_scan");
}

template <int DK, int KIND>
static int launch_chunks(const int* seg_info, int segments, int rows, const float* qn, const float* kn, const float* vv,
                         const float* decay, const float* beta, const float* fgate, float* pairs, float* state,
                         long long state_stride, int heads, int kv_heads, int dv, float* o_raw, cudaStream_t stream) {
    const int each = (rows / kC + segments) / segments;        // chunks of a portion on average: a block each
    if constexpr (KIND == kDelta || KIND == kChannel)
        chunk_pairs_kernel<DK, KIND><<<dim3((heads + 3) / 4, segments, each < 65535 ? each : 65535), 128, 0, stream>>>(
            seg_info, segments, qn, kn, decay, beta, heads, kv_heads, pairs);
    else
        chunk_scalar_pairs_kernel<DK, KIND><<<dim3((kv_heads + 3) / 4, segments, each < 65535 ? each : 65535), 128, 0, stream>>>(
            seg_info, segments, qn, kn, beta, fgate, heads, kv_heads, pairs);
    if (int rc = finish_launch("chunk_pairs")) return rc;
    // Blocks of 32 columns split a head's tokens half as often as blocks of 16, which are for grids that would leave a quarter of
    // the multiprocessors without a block.  Where there are more blocks than multiprocessors, the light form of the recurrences
    // with one decay per head holds two on each (three portions of 701 tokens, 32 heads of 128 x 128, constant decays: 189 us
    // with the pairs against 196; 64 heads, 2048 tokens 324 against 349; a single round of blocks, 32 heads, 202 against 183).
    const int sms = sm_count_cached() > 0 ? sm_count_cached() : 148;
    const long long blocks = (long long)segments * heads * (dv / 32);
#define CHUNK_LAUNCH(COLS, LIGHT) \
    return launch_chunk_scan<DK, KIND, COLS, LIGHT>(seg_info, segments, qn, kn, vv, decay, pairs, state, state_stride, heads, kv_heads, dv, o_raw, stream)
    if (dv % 32 != 0 || blocks * 4 < 3LL * sms) CHUNK_LAUNCH(16, false);
    if constexpr (KIND == kHead || KIND == kFixed) {
        if (blocks > sms) CHUNK_LAUNCH(32, true);
    }
    CHUNK_LAUNCH(32, false);
#undef CHUNK_LAUNCH
}

}  // namespace tllm

using namespace tllm;

// The recurrences of tllm_delta_scan by chunks: modes 0 (delta rule), 1 (decay per channel), 3 (decay per token and head), 5
// (constant decay per head), with that entry's operands.  pairs
// float[(rows / 16 + segments) * heads * 512].  qn, kn, vv, decay and pairs on 16-byte boundaries.
extern "C" int tllm_chunk_scan(const int* seg_info, int segments, int rows, const float* qn, const float* kn, const float* vv,
                               const float* decay, const float* beta, const float* fgate, float* pairs, float* state,
                               long long state_stride, int heads, int kv_heads, int dk, int dv, float* o_raw, int mode, cudaStream_t stream) {
    TLLM_REQUIRE(segments >= 0 && rows >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0, "chunk_scan: bad sizes");
    TLLM_REQUIRE((dk == 64 || dk == 128) && dv > 0 && dv % 16 == 0, "chunk_scan: keys of %d, values of %d", dk, dv);
    TLLM_REQUIRE(segments <= 65535, "chunk_scan: %d portions", segments);
    const auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    TLLM_REQUIRE(al(qn) && al(kn) && al(vv) && al(decay) && al(pairs), "chunk_scan: operands must be 16-byte aligned");
    TLLM_REQUIRE(seg_info != nullptr && pairs != nullptr, "chunk_scan: no portions");
    if (segments == 0 || rows == 0) return 0;
#define CHUNKS(K)                                                                                                                \
    return dk == 128 ? launch_chunks<128, K>(seg_info, segments, rows, qn, kn, vv, decay, beta, fgate, pairs, state, state_stride, \
                                             heads, kv_heads, dv, o_raw, stream)                                                  \
                     : launch_chunks<64, K>(seg_info, segments, rows, qn, kn, vv, decay, beta, fgate, pairs, state, state_stride,  \
                                            heads, kv_heads, dv, o_raw, stream)
    if (mode == 0) {
        TLLM_REQUIRE(decay != nullptr && beta != nullptr, "chunk_scan: the delta rule lacks an operand");
        CHUNKS(kDelta);
    }
    if (mode == 1) {
        TLLM_REQUIRE(decay != nullptr, "chunk_scan: no decays");
        CHUNKS(kChannel);
    }
    if (mode == 3) {
        TLLM_REQUIRE(beta != nullptr && fgate != nullptr, "chunk_scan: no decays or strengths");
        CHUNKS(kHead);
    }
    TLLM_REQUIRE(mode == 5 && fgate != nullptr, "chunk_scan: unknown recurrence %d", mode);
    CHUNKS(kFixed);
#undef CHUNKS
}
