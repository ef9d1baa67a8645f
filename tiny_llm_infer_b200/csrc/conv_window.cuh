// The window of a short causal convolution in a request's state moves on by a portion: `keep` (taps - 1) newest inputs per
// channel, the newest last.  Called by the blocks of a portion's last row for channels [c0, c1); all of a thread's loads are
// issued before its first store, and an old entry is read before its place is written.
// (As a loop of a load and a store per entry, with one block for all channels, this was what the last block of the kernels
// that finish a recurrence spent its time with: 26 us for 6144 channels, three entries each.)
#pragma once

#include "common.cuh"

namespace tllm {

__device__ __forceinline__ float4 window_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 window_load4(const bf16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// `last`: the portion's last row of inputs, rows `ld` elements apart; `len`: the portion's rows, as far as the window reaches.
// vec: four channels per access (channels, ld and the bounds multiples of four, 16-byte boundaries of tail, 8 of bfloat16).
template <typename T>
__device__ __forceinline__ void move_window(const T* last, int ld, int len, int keep, float* tail, int channels, int c0, int c1, bool vec) {
    if (vec && keep <= 3) {
        for (int c = c0 + threadIdx.x * 4; c < c1; c += blockDim.x * 4) {
            float4 x[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                if (i >= keep) continue;
                const int from_end = keep - i;       // this entry is the from_end-th newest input
                x[i] = from_end <= len ? window_load4(last - (size_t)(from_end - 1) * ld + c) : window_load4(tail + (size_t)(i + len) * channels + c);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
                if (i < keep) *reinterpret_cast<float4*>(tail + (size_t)i * channels + c) = x[i];
        }
        return;
    }
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x)
        for (int i = 0; i < keep; ++i) {             // ascending: an old entry is read before its place is written
            const int from_end = keep - i;
            tail[(size_t)i * channels + c] = from_end <= len ? to_f32<T>(last[c - (long long)(from_end - 1) * ld]) : tail[(size_t)(i + len) * channels + c];
        }
}

// Rows of a portion up to `t`, its last, as far as the window reaches.
__device__ __forceinline__ int window_rows(const int* token_slot, int t, int slot, int keep) {
    int len = 1;
    while (len < keep && t - len >= 0 && token_slot[t - len] == slot) ++len;
    return len;
}

}  // namespace tllm
