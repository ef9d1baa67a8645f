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
// and written once per sixteen tokens, as small matrix products with sixteen independent sums each.  Every G is a product of
// decays, made by multiplying them up from either side; nothing is divided and no exponential of a sum is taken, so the
// results are as exact as the token's way.  All sums are float32.
//
//   chunk_pairs  one warp per (chunk, head): T and Q T, or Q, the decays from the chunk's start and the write weights.
//   chunk_scan   one block per (portion, head, 32 or 16 columns); a warp owns 2 NL columns, a lane 8 rows (4 where keys have
//                64 elements) of NL of them in registers.  The sums of a group of tokens meet over the sixteen lanes of a
//                column by exchanging halves.
//
// The layout of the request's state is the scan kernel's (row r * per + il of column j at [il][j][r]).
#include "common.cuh"

namespace tllm {

constexpr int kC = 16;                         // tokens of a chunk
constexpr int kPairFloats = 2 * kC * kC;       // T and Q T, or the scalars and Q, of one (chunk, head)
constexpr int kPad = 20;                       // floats of a row of either in shared memory

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

// DK 128: a lane has four neighbouring channels; DK 64: the upper sixteen lanes carry zeros.
template <int DK, int KIND>
__global__ void __launch_bounds__(128)
chunk_pairs_kernel(const int* __restrict__ seg_info, int segments, const float* qn, const float* kn, const float* decay, const float* beta,
                   const float* fgate, int heads, int kv_heads, float* pairs) {
    constexpr bool kVec = KIND == kDelta || KIND == kChannel, kCorr = KIND == kDelta;
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
        // scalars of token `col`: its decay and the weight of its values
        float a_own = 1.0f, w_own = 1.0f;
        if (col < n) {
            const size_t t = (size_t)(start + c0 + col) * heads + head;
            if (KIND == kDelta || KIND == kChannel) w_own = beta != nullptr ? beta[t] : 1.0f;
            if (KIND == kHead) { a_own = beta[t]; w_own = fgate[t]; }
            if (KIND == kFixed) a_own = fgate[head];
        }
        float4 w[kC];                                               // k_j, decayed up to the token at hand
        float4 q4[4], g4[4];                                        // the next four tokens' q and decays
        float trow[kC];                                             // column `col` of T
        float d = 1.0f, prefix = 1.0f;                              // scalar decays: of j up to i, and from the chunk's start
#pragma unroll
        for (int i = 0; i < kC; ++i) w[i] = i < n ? at(kn, i, kvh, kv_heads) : zero;
#pragma unroll
        for (int i = 0; i < kC; ++i) {
            if (i % 4 == 0)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    q4[e] = i + e < n ? at(qn, i + e, kvh, kv_heads) : zero;
                    if (kVec) g4[e] = i + e < n ? at(decay, i + e, head, heads) : one;
                }
            const float4 k = w[i], q = q4[i % 4];                   // w[i] has no decay on it yet
            float s;                                                // lane j: Q_ij; with the correction lane 16 + j: A_ij
            if (kVec) {
#pragma unroll
                for (int j = 0; j < i; ++j) w[j] = mul4(w[j], g4[i % 4]);
            }
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
                if (!kVec) {
                    const float a = __shfl_sync(0xffffffffu, a_own, i);
                    if (col < i) d *= a;                            // j < i: one more decay between j and i
                    prefix *= a;
                    s *= d;
                    if (lane == 0) T[i] = prefix;
                } else if (lane == 0) {
                    T[i] = 1.0f;
                }
                // of a later token nothing, not zero times its weight: that may be infinite or no number
                if (lane < 16) Q[i * kC + col] = col <= i ? s * w_own : 0.0f;
            }
        }
        // row 1: what token j's values are multiplied by in the state, its weight and the decays after it
        if (!kCorr && lane < 16) T[kC + col] = w_own * d;
    }
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0));
}
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// COLS columns per block (16 or 32), NL columns per lane (4 or 2).
template <int DK, int KIND, int COLS, int NL>
struct ChunkLayout {
    static constexpr bool kVec = KIND == kDelta || KIND == kChannel;
    static constexpr int kWarps = COLS / (2 * NL), kStages = kVec ? 3 : 2;
    static constexpr int kIssuers = (kVec ? COLS / 8 : kWarps) * 32;      // decays per channel: warps of their own prepare the tokens
    static constexpr int kThreads = kWarps * 32 + (kVec ? kIssuers : 0);
    static constexpr int kK = 0, kQ = kC * DK, kG = 2 * kC * DK, kV = kG + (kVec ? kC * DK : 0), kT = kV + kC * COLS, kQm = kT + kC * kPad;
    static constexpr int kGam = kQm + kC * kPad, kStage = kGam + (kVec ? DK : 0);
    static constexpr int kX = kStages * kStage, kU = kX + kC * COLS, kFloats = kU + kC * COLS;
};

template <int DK, int KIND, int COLS, int NL>
__global__ void __launch_bounds__(ChunkLayout<DK, KIND, COLS, NL>::kThreads, 512 / ChunkLayout<DK, KIND, COLS, NL>::kThreads)
chunk_scan_kernel(const int* __restrict__ seg_info, const float* qn, const float* kn, const float* vv, const float* decay,
                  const float* pairs, float* state, long long state_stride, int segments, int heads, int kv_heads, int dv, float* o_raw) {
    using L = ChunkLayout<DK, KIND, COLS, NL>;
    constexpr bool kVec = L::kVec, kCorr = KIND == kDelta;
    constexpr int kH = DK / 64, kPairs = 2 * kH, kIssuers = L::kIssuers;           // a lane's runs of four rows
    constexpr int kWide = 2 * NL, kGroup = kC / NL;                                // columns of a warp; tokens whose sums meet at once
    extern __shared__ __align__(16) float sm[];
    const int seg = blockIdx.y, groups = dv / COLS, head = blockIdx.x / groups, col0 = blockIdx.x % groups * COLS;
    const int slot = seg_info[4 * seg], start = seg_info[4 * seg + 1], len = seg_info[4 * seg + 2];
    const int first = first_entry(seg_info, segments, seg);
    if (slot < 0 || len <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane & 15, cg = (lane >> 4) * NL;
    const int kvh = head / (heads / kv_heads), mine = warp * kWide + cg;                      // first of the lane's columns
    float* xs = sm + L::kX + warp * kC * kWide;
    float* us = sm + L::kU + warp * kC * kWide;

    const int me = kVec ? (int)threadIdx.x - L::kWarps * 32 : threadIdx.x;         // among the threads that copy
    auto issue = [&](int c0, int st) {
        const int n = min(kC, len - c0);
        float* s = sm + st * L::kStage;
        for (int i = me; i < kC * DK / 4; i += kIssuers) {
            const int t = i / (DK / 4), e = (i % (DK / 4)) * 4;
            const bool in = t < n;
            const size_t row = (size_t)(start + c0 + (in ? t : 0));
            cp16(s + L::kK + t * DK + e, kn + (row * kv_heads + kvh) * DK + e, in);
            cp16(s + L::kQ + t * DK + e, qn + (row * kv_heads + kvh) * DK + e, in);
            if (kVec) cp16(s + L::kG + t * DK + e, decay + (row * heads + head) * DK + e, in);
        }
        for (int i = me; i < kC * COLS / 4; i += kIssuers) {
            const int t = i / (COLS / 4), e = (i % (COLS / 4)) * 4;
            const bool in = t < n;
            cp16(s + L::kV + t * COLS + e, vv + ((size_t)(start + c0 + (in ? t : 0)) * heads + head) * dv + col0 + e, in);
        }
        const float* p = pairs + ((size_t)(first + c0 / kC) * heads + head) * kPairFloats;
        for (int i = me; i < kPairFloats / 4; i += kIssuers) {
            const int t = (i & 63) / 4, e = (i & 3) * 4;
            cp16(s + (i < 64 ? L::kT : L::kQm) + t * kPad + e, p + i * 4, true);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };

    // Decays per channel: q and (for the correction) k take on the decays since the chunk's start, and g's place the k's with
    // the decays up to its end; a thread has a channel of all sixteen tokens.  Warps of their own do it, a chunk ahead.
    auto prepare = [&](int c0, int st) {
        const int n = min(kC, len - c0);
        float* s = sm + st * L::kStage;
        for (int ch = me; ch < DK; ch += kIssuers) {
            float k[kC], g[kC], q[kC], p = 1.0f;
#pragma unroll
            for (int i = 0; i < kC; ++i) {
                k[i] = s[L::kK + i * DK + ch];
                g[i] = s[L::kG + i * DK + ch];
                q[i] = s[L::kQ + i * DK + ch];
            }
#pragma unroll
            for (int i = 0; i < kC; ++i) {
                if (i >= n) g[i] = 1.0f;
                p *= g[i];
                s[L::kQ + i * DK + ch] = q[i] * p;
                if (kCorr) s[L::kK + i * DK + ch] = k[i] * p;
            }
            s[L::kGam + ch] = p;
            p = 1.0f;
#pragma unroll
            for (int i = kC - 1; i >= 0; --i) {
                s[L::kG + i * DK + ch] = k[i] * p;
                p *= g[i];
            }
        }
    };
    if (kVec && warp >= L::kWarps) {
        issue(0, 0);
        if (kC < len) issue(kC, 1);
        for (int c0 = 0, st = 0; c0 < len + kC; c0 += kC, st = st == 2 ? 0 : st + 1) {     // prepares c0 while c0 - kC is consumed
            if (c0 < len) {
                if (c0 + kC < len) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                asm volatile("bar.sync 1, %0;\n" ::"n"(kIssuers) : "memory");             // the copies of all of these warps
                prepare(c0, st);
            }
            __syncthreads();                                    // c0 - kC is done with: its stage, the one after next, is free
            if (c0 + 2 * kC < len) issue(c0 + 2 * kC, st == 0 ? 2 : st - 1);
        }
        return;
    }
    if (!kVec) issue(0, 0);
    // the lane's rows: 64 h + 4 r + e; row i of the state lies at [i % per][column][i / per]
    constexpr int kR = DK <= 64 ? 4 : 8, kPer = DK / kR;
    float* st_ptr = state + (long long)slot * state_stride + (size_t)head * DK * dv;
    auto state_at = [&](int h, int e, int c) -> float& {
        const int i = 64 * h + 4 * r + e;
        return st_ptr[((size_t)(i % kPer) * dv + col0 + mine + c) * kR + i / kPer];
    };
    float2 S[NL][kPairs];
#pragma unroll
    for (int c = 0; c < NL; ++c)
#pragma unroll
        for (int h = 0; h < kH; ++h) {
            S[c][2 * h] = make_float2(state_at(h, 0, c), state_at(h, 1, c));
            S[c][2 * h + 1] = make_float2(state_at(h, 2, c), state_at(h, 3, c));
        }

    if (kVec) __syncthreads();                                  // the first chunk is ready
    for (int c0 = 0, st = 0; c0 < len; c0 += kC, st = st == L::kStages - 1 ? 0 : st + 1) {
        const int n = min(kC, len - c0);
        if (!kVec) {
            if (c0 + kC < len) {
                issue(c0 + kC, st ^ 1);
                asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            }
            __syncthreads();
        }
        float* s = sm + st * L::kStage;
        // sums against the state before the chunk, kGroup tokens at a time; token kGroup g + r / NL of column r % NL ends here
        float xk[NL], xq[NL];
#pragma unroll
        for (int g = 0; g < NL; ++g) {
            constexpr int kSums = kCorr ? 2 : 1;
            float v[kSums][16];
#pragma unroll
            for (int t = 0; t < kGroup; ++t) {
                float2 acc[kSums][NL];
#pragma unroll
                for (int h = 0; h < kH; ++h) {
                    const int off = (kGroup * g + t) * DK + 64 * h + 4 * r;
                    const float4 q4 = *reinterpret_cast<const float4*>(s + L::kQ + off);
                    float4 k4;
                    if (kCorr) k4 = *reinterpret_cast<const float4*>(s + L::kK + off);
#pragma unroll
                    for (int c = 0; c < NL; ++c) {
                        acc[0][c] = h == 0 ? __fmul2_rn(S[c][0], lo2(q4)) : __ffma2_rn(S[c][2 * h], lo2(q4), acc[0][c]);
                        acc[0][c] = __ffma2_rn(S[c][2 * h + 1], hi2(q4), acc[0][c]);
                        if (kCorr) {
                            acc[kSums - 1][c] = h == 0 ? __fmul2_rn(S[c][0], lo2(k4)) : __ffma2_rn(S[c][2 * h], lo2(k4), acc[kSums - 1][c]);
                            acc[kSums - 1][c] = __ffma2_rn(S[c][2 * h + 1], hi2(k4), acc[kSums - 1][c]);
                        }
                    }
                }
#pragma unroll
                for (int w = 0; w < kSums; ++w)
#pragma unroll
                    for (int c = 0; c < NL; ++c) v[w][t * NL + c] = acc[w][c].x + acc[w][c].y;
            }
#pragma unroll
            for (int half = 8; half > 0; half >>= 1) {
                const bool up = r & half;
#pragma unroll
                for (int w = 0; w < kSums; ++w)
#pragma unroll
                    for (int i = 0; i < half; ++i) {
                        const float keep = up ? v[w][i + half] : v[w][i], send = up ? v[w][i] : v[w][i + half];
                        v[w][i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
                    }
            }
            xq[g] = v[0][0];
            if (kCorr) xk[g] = v[kSums - 1][0];
        }
        const int tr = r / NL, myc = cg + r % NL;               // this lane's tokens are kGroup m + tr, its column of the warp's
        const float* T = s + L::kT;
        const float* Qm = s + L::kQm;
        const float* vcol = s + L::kV + warp * kWide + myc;
        // token j's value as the lane's m-th token sees it: a later one not at all, be it infinite or no number (the delta
        // rule's whole mixer at 2048 tokens: 510 us, 482 without; the other recurrences take no longer)
        auto before = [&](float x, int j, int m) -> float { return j >= kGroup * m && j > kGroup * m + tr ? 0.0f : x; };
        float o[NL];
        if (kCorr) {
#pragma unroll
            for (int m = 0; m < NL; ++m) xs[(kGroup * m + tr) * kWide + myc] = vcol[(kGroup * m + tr) * COLS] - xk[m];
            __syncwarp();
            float u[NL];
#pragma unroll
            for (int m = 0; m < NL; ++m) o[m] = xq[m], u[m] = 0.0f;
#pragma unroll
            for (int j = 0; j < kC; j += 4) {
                const float x0 = xs[j * kWide + myc], x1 = xs[(j + 1) * kWide + myc], x2 = xs[(j + 2) * kWide + myc], x3 = xs[(j + 3) * kWide + myc];
#pragma unroll
                for (int m = 0; m < NL; ++m) {
                    if (kGroup * (m + 1) <= j) continue;        // T and Q T are zero above their diagonals
                    const float4 t4 = *reinterpret_cast<const float4*>(T + (kGroup * m + tr) * kPad + j);
                    const float4 q4 = *reinterpret_cast<const float4*>(Qm + (kGroup * m + tr) * kPad + j);
                    const float y0 = before(x0, j, m), y1 = before(x1, j + 1, m), y2 = before(x2, j + 2, m), y3 = before(x3, j + 3, m);
                    u[m] = fmaf(t4.x, y0, fmaf(t4.y, y1, fmaf(t4.z, y2, fmaf(t4.w, y3, u[m]))));
                    o[m] = fmaf(q4.x, y0, fmaf(q4.y, y1, fmaf(q4.z, y2, fmaf(q4.w, y3, o[m]))));
                }
            }
#pragma unroll
            for (int m = 0; m < NL; ++m) us[(kGroup * m + tr) * kWide + myc] = u[m];
            __syncwarp();
        } else {
#pragma unroll
            for (int m = 0; m < NL; ++m) {
                o[m] = xq[m] * T[kGroup * m + tr];
                us[(kGroup * m + tr) * kWide + myc] = T[kPad + kGroup * m + tr] * vcol[(kGroup * m + tr) * COLS];
            }
#pragma unroll
            for (int j = 0; j < kC; j += 4) {
                float y[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) y[e] = vcol[(j + e) * COLS];
#pragma unroll
                for (int m = 0; m < NL; ++m) {
                    if (kGroup * (m + 1) <= j) continue;
                    const float4 q4 = *reinterpret_cast<const float4*>(Qm + (kGroup * m + tr) * kPad + j);
                    o[m] = fmaf(q4.x, before(y[0], j, m), fmaf(q4.y, before(y[1], j + 1, m),
                           fmaf(q4.z, before(y[2], j + 2, m), fmaf(q4.w, before(y[3], j + 3, m), o[m]))));
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int m = 0; m < NL; ++m)
            if (kGroup * m + tr < n) o_raw[((size_t)(start + c0 + kGroup * m + tr) * heads + head) * dv + col0 + warp * kWide + myc] = o[m];
        // the state moves on
        if (kVec) {
#pragma unroll
            for (int h = 0; h < kH; ++h) {
                const float4 g4 = *reinterpret_cast<const float4*>(s + L::kGam + 64 * h + 4 * r);
#pragma unroll
                for (int c = 0; c < NL; ++c) {
                    S[c][2 * h] = __fmul2_rn(S[c][2 * h], lo2(g4));
                    S[c][2 * h + 1] = __fmul2_rn(S[c][2 * h + 1], hi2(g4));
                }
            }
        } else {
            const float2 g2 = dup(T[kC - 1]);
#pragma unroll
            for (int c = 0; c < NL; ++c)
#pragma unroll
                for (int p = 0; p < kPairs; ++p) S[c][p] = __fmul2_rn(S[c][p], g2);
        }
#pragma unroll
        for (int j = 0; j < kC; ++j) {
            float2 u2[NL];
            if (NL == 4) {
                const float4 u4 = *reinterpret_cast<const float4*>(us + j * kWide + cg);
                u2[0] = dup(u4.x), u2[1] = dup(u4.y), u2[NL - 2] = dup(u4.z), u2[NL - 1] = dup(u4.w);
            } else {
                const float2 u4 = *reinterpret_cast<const float2*>(us + j * kWide + cg);
                u2[0] = dup(u4.x), u2[1] = dup(u4.y);
            }
#pragma unroll
            for (int h = 0; h < kH; ++h) {
                const float4 k4 = *reinterpret_cast<const float4*>(s + (kVec ? L::kG : L::kK) + j * DK + 64 * h + 4 * r);
#pragma unroll
                for (int c = 0; c < NL; ++c) {
                    S[c][2 * h] = __ffma2_rn(lo2(k4), u2[c], S[c][2 * h]);
                    S[c][2 * h + 1] = __ffma2_rn(hi2(k4), u2[c], S[c][2 * h + 1]);
                }
            }
        }
        __syncthreads();                                        // the stage may be filled again
    }
#pragma unroll
    for (int c = 0; c < NL; ++c)
#pragma unroll
        for (int h = 0; h < kH; ++h) {
            state_at(h, 0, c) = S[c][2 * h].x;
            state_at(h, 1, c) = S[c][2 * h].y;
            state_at(h, 2, c) = S[c][2 * h + 1].x;
            state_at(h, 3, c) = S[c][2 * h + 1].y;
        }
}

template <int DK, int KIND, int COLS, int NL>
static int launch_chunk_scan(const int* seg_info, int segments, const float* qn, const float* kn, const float* vv, const float* decay,
                             const float* pairs, float* state, long long state_stride, int heads, int kv_heads, int dv, float* o_raw,
                             cudaStream_t stream) {
    constexpr size_t smem = ChunkLayout<DK, KIND, COLS, NL>::kFloats * sizeof(float);
    static OncePerDevice configured;
    if (configured.first()) {
        cudaError_t e = cudaFuncSetAttribute(chunk_scan_kernel<DK, KIND, COLS, NL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { set_error("chunk_scan: %s", cudaGetErrorString(e)); return (int)e; }
        configured.done();
    }
    chunk_scan_kernel<DK, KIND, COLS, NL><<<dim3(heads * (dv / COLS), segments), ChunkLayout<DK, KIND, COLS, NL>::kThreads, smem, stream>>>(
        seg_info, qn, kn, vv, decay, pairs, state, state_stride, segments, heads, kv_heads, dv, o_raw);
    return finish_launch("chunk_scan");
}

template <int DK, int KIND>
static int launch_chunks(const int* seg_info, int segments, int rows, const float* qn, const float* kn, const float* vv,
                         const float* decay, const float* beta, const float* fgate, float* pairs, float* state,
                         long long state_stride, int heads, int kv_heads, int dv, float* o_raw, cudaStream_t stream) {
    const int each = (rows / kC + segments) / segments;        // chunks of a portion on average: a block each
    chunk_pairs_kernel<DK, KIND><<<dim3((heads + 3) / 4, segments, each < 65535 ? each : 65535), 128, 0, stream>>>(
        seg_info, segments, qn, kn, decay, beta, fgate, heads, kv_heads, pairs);
    if (int rc = finish_launch("chunk_pairs")) return rc;
    // Blocks of 32 columns, four per lane, read the tokens' rows from shared memory least often, which is what bounds a full grid
    // (2048 tokens, 128 x 128, delta rule, with the pairs, from a cold L2: 64 heads 601 us, two per lane 755, blocks of 16 columns
    // 951 and 794; 32 heads 384, 388, 497 and 411).  Where they would leave a quarter of the multiprocessors without a block, 16
    // columns, two per lane (16 heads: 235 us against 366; four per lane 359).
    const int sms = sm_count_cached() > 0 ? sm_count_cached() : 148;
#define CHUNK_LAUNCH(COLS, NL) \
    return launch_chunk_scan<DK, KIND, COLS, NL>(seg_info, segments, qn, kn, vv, decay, pairs, state, state_stride, heads, kv_heads, dv, o_raw, stream)
    if (dv % 32 == 0 && (long long)segments * heads * (dv / 32) * 4 >= 3LL * sms) CHUNK_LAUNCH(32, 4);
    CHUNK_LAUNCH(16, 2);
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
