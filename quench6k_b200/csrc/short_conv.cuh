// A short causal convolution over time on rows of FP32 channels, vectorised: a thread takes four channels of eight tokens, so that
// an input is read once for all the taps that see it, 16 bytes at a time, with all of a thread's loads asked for first.  (A thread
// per channel and token read every input once per tap, four bytes at a time: 60 us for 2,048 tokens of 4,096 channels with
// four taps, 50 MB; so 24 us, bound by the loads in flight.)  The sums are those of the kernels it stands in for, tap by tap in order.
#pragma once
#include "common.cuh"

namespace {

constexpr int CONV_TOKENS = 8;

__device__ __forceinline__ void conv_store(float* out, float4 v) { *reinterpret_cast<float4*>(out) = v; }
__device__ __forceinline__ void conv_store(__nv_bfloat16* out, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(out) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// grid (ceil(T / 8), ceil(C / 512)), 128 threads.  STARTS_WITH_BIAS: the sum starts at the bias (else the bias, if there is one, is
// part of every input).  x: FP32 [T, ldx]; w: FP32 [C, TAPS]; tail: FP32 [slots, TAPS - 1, C]; out: T [T, ldo].
template <typename T, int TAPS, bool STARTS_WITH_BIAS>
__global__ void __launch_bounds__(128) conv_rows_kernel(const float* x, int ldx, const float* w, const float* bias, const float* tail, const int* req_of_token,
                                                        const int* q_start, const int* slot_ids, T* out, int ldo, int T_, int C, int act) {
    pdl_enter();
    const int t0 = blockIdx.x * CONV_TOKENS, t1 = min(T_, t0 + CONV_TOKENS), c = (blockIdx.y * 128 + threadIdx.x) * 4;
    if (c >= C) return;
    float ww[4][TAPS];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int k = 0; k < TAPS; ++k) ww[e][k] = w[(size_t)(c + e) * TAPS + k];
    const float4 b = bias ? *reinterpret_cast<const float4*>(bias + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const bool add = !STARTS_WITH_BIAS && bias != nullptr;
    auto plus = [&](float4 v) { return add ? make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w) : v; };
    for (int ta = t0; ta < t1;) {                       // the tokens of one request at a time (nearly always all of them)
        const int r = req_of_token[ta], first = q_start[r], tb = max(ta + 1, min(t1, q_start[r + 1]));
        const float* old = tail + (size_t)slot_ids[r] * (TAPS - 1) * C + c;
        float4 v[TAPS - 1 + CONV_TOKENS];
#pragma unroll
        for (int j = 0; j < TAPS - 1 + CONV_TOKENS; ++j) {
            const int t = ta - (TAPS - 1) + j;          // a row of the step, or, before the portion, of the tail
            v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (t < tb) v[j] = t >= first ? plus(*reinterpret_cast<const float4*>(x + (size_t)t * ldx + c)) : *reinterpret_cast<const float4*>(old + (size_t)(TAPS - 1 + t - first) * C);
        }
#pragma unroll
        for (int i = 0; i < CONV_TOKENS; ++i) {
            if (ta + i >= tb) break;
            float4 s = STARTS_WITH_BIAS ? b : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < TAPS; ++k) {
                s.x = fmaf(ww[0][k], v[i + k].x, s.x), s.y = fmaf(ww[1][k], v[i + k].y, s.y);
                s.z = fmaf(ww[2][k], v[i + k].z, s.z), s.w = fmaf(ww[3][k], v[i + k].w, s.w);
            }
            if (act) s = make_float4(s.x / (1.0f + expf(-s.x)), s.y / (1.0f + expf(-s.y)), s.z / (1.0f + expf(-s.z)), s.w / (1.0f + expf(-s.w)));
            conv_store(out + (size_t)(ta + i) * ldo + c, s);
        }
        ta = tb;
    }
}

// Whether these rows go four channels at a time; else the kernels that take any.  A thread's walk over eight tokens takes some 5 us however
// few there are, a thread per channel and token 2.5 and more with every token: the lines meet at about 750,000 values (4,096 channels:
// 130 tokens 5.6 and 5.4 us, 64 tokens 3.8 and 5.3; 3,072 channels with a tail to move on: 130 tokens 7.4 and 9.3, 256 tokens 9.9 and 9.7, 512 tokens 15.0 and
// 10.5; 2,048 tokens 60 and 24).  Beside many requests of a token each, eight requests' tokens in a row are eight trips to memory one
// after the other (256 tokens beside 32 requests 11.0 and 13.8 us, 512 beside 32 16.0 and 14.8).
inline bool conv_rows_taken(int T_, int requests, const float* x, int ldx, const float* bias, const float* tail, const void* out, int ldo, int C, int taps) {
    return requests > 0 && (long long)T_ * C >= 750000 && T_ >= 16 * requests && taps >= 1 && taps <= 4 && C % 4 == 0 && ldx % 4 == 0 && ldo % 4 == 0 &&
           (((uintptr_t)x | (uintptr_t)bias | (uintptr_t)tail | (uintptr_t)out) & 15) == 0;
}

template <typename T, bool STARTS_WITH_BIAS>
void conv_rows(const float* x, int ldx, const float* w, const float* bias, const float* tail, const int* req_of_token, const int* q_start, const int* slot_ids,
               T* out, int ldo, int T_, int C, int taps, int act, cudaStream_t st) {
    const dim3 grid((T_ + CONV_TOKENS - 1) / CONV_TOKENS, (C + 511) / 512);
    auto* kernel = taps == 1 ? conv_rows_kernel<T, 1, STARTS_WITH_BIAS> : taps == 2 ? conv_rows_kernel<T, 2, STARTS_WITH_BIAS> : taps == 3 ? conv_rows_kernel<T, 3, STARTS_WITH_BIAS> : conv_rows_kernel<T, 4, STARTS_WITH_BIAS>;
    q6k_launch(kernel, grid, 128, 0, st, x, ldx, w, bias, tail, req_of_token, q_start, slot_ids, out, ldo, T_, C, act);
}

}  // namespace
