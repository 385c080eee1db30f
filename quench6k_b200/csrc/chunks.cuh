// What the kernels that walk a portion in chunks of 32 tokens share.
#pragma once
#include "common.cuh"

namespace {

constexpr int WC = 32, WLD = WC + 4;                            // tokens of a chunk; pitch of a row of 32 in shared memory
constexpr int WALK_THREADS = 256, WALK_COLS = 16;               // threads of a walking block and columns of the state it owns

// Requests of more than `beyond` tokens go chunk by chunk, the others token by token in a launch of their own.

// Chunk c (of CT tokens) of all those requests' chunks side by side: its first row and its tokens (0: there is no such chunk).
template <int CT = WC>
__device__ __forceinline__ void chunk_of(const int* q_start, int R, int beyond, int c, int& first, int& tokens) {
    tokens = 0;
    for (int r = 0; r < R; ++r) {
        const int n = q_start[r + 1] - q_start[r], chunks = n > beyond ? (n + CT - 1) / CT : 0;
        if (c < chunks) {
            first = q_start[r] + c * CT;
            tokens = min(CT, n - c * CT);
            return;
        }
        c -= chunks;
    }
}
// The y-th of those requests (-1: there are fewer) and its first chunk among all chunks.
template <int CT = WC>
__device__ __forceinline__ int long_request(const int* q_start, int R, int beyond, int y, int& first_chunk) {
    first_chunk = 0;
    for (int r = 0; r < R; ++r) {
        const int n = q_start[r + 1] - q_start[r];
        if (n <= beyond) continue;
        if (y-- == 0) return r;
        first_chunk += (n + CT - 1) / CT;
    }
    return -1;
}
// How many there can be in a step of T_ rows, and how many chunks.
inline int most_long(int T_, int R, int beyond) { return R < T_ / (beyond + 1) ? R : T_ / (beyond + 1); }
template <int CT = WC>
inline int most_chunks(int T_, int R, int beyond) { return T_ / CT + most_long(T_, R, beyond); }

__device__ __forceinline__ float dot4(const float4& a, const float4& b, float acc) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc)))); }
// v with zeros behind its entry n: no value of a later token, were it infinite, reaches an earlier one.
__device__ __forceinline__ float4 up_to(float4 v, int n) { return make_float4(v.x, n >= 1 ? v.y : 0.0f, n >= 2 ? v.z : 0.0f, n >= 3 ? v.w : 0.0f); }
// Two FP32 multiply-adds in one instruction; a value in both halves; the halves added.
__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long both(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "r"(__float_as_uint(v)));
    return r;
}
__device__ __forceinline__ float low(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
// 16 bytes global -> shared without passing registers; !in: zeros (nothing is read from `from`, which has to be an address all the same).
__device__ __forceinline__ void copy16(uint32_t to, const float* from, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(in ? 16 : 0) : "memory");
}

}  // namespace
