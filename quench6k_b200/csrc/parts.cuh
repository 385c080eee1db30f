// FP32 operands of the tensor cores: a number as the sum of three bfloat16 numbers of 8 significant bits each, exactly (x0 = x rounded, x1 = the
// rest rounded, x2 = what is left), and a product of two bfloat16 numbers is exact in FP32.  So a b is taken as the six products a0 b0 + (a0 b1 + a1 b0) +
// (a1 b1 + a0 b2 + a2 b0) on tcgen05.mma, the smallest first; the three left out are below 2^-25 of it.  Tensor memory truncates where it adds, which
// over a few hundred terms stays below the rounding of a sum in FP32 (1.1e-7 of the norm over 1,024 terms added 64 at a time; multiply-adds in four chains
// 2.9e-7).  An operand that is infinite, not a number or beyond bfloat16's largest makes its results NaN: who stores them sums those that are not finite
// again with multiply-adds.  Parts of numbers below 2^-110 may be lost.
#pragma once
#include "umma.cuh"

namespace {

// Two values as three pairs of bfloat16 (x in the low half) that add up to them.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& h0, uint32_t& h1, uint32_t& h2) {
    auto pack = [](float lo, float hi) {
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    };
    h0 = pack(x, y);
    x -= __uint_as_float(h0 << 16), y -= __uint_as_float(h0 & 0xffff0000u);
    h1 = pack(x, y);
    x -= __uint_as_float(h1 << 16), y -= __uint_as_float(h1 & 0xffff0000u);
    h2 = pack(x, y);
}

// Four floats from `from`, or zeros; the registers are written by the load alone, so that nothing waits for it before their first use.
__device__ __forceinline__ void load4(float* v, const float* from, bool in) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
        "@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}" : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]) : "l"(from), "r"((int)in) : "memory");
}

// The order of the products: part PARTS_A[e] of A times part PARTS_B[e] of B, the smallest first.
#define Q6K_PARTS_ORDER constexpr int PARTS_A[6] = {0, 2, 1, 0, 1, 0}, PARTS_B[6] = {2, 0, 1, 1, 0, 0}

// A tile [ROWS x 64 * blocks] of parts in shared memory: per part, blocks of 64 columns, a row of a block 128 bytes with the 128-byte swizzle.  Its
// rows may be the operand's M or N (K-major: umma_desc_k, a step of 16 k is 32 bytes, 64 k a block) or its K (MN-major: umma_desc_mn with blocks
// ROWS * 128 bytes apart, a step of 16 k is 2,048 bytes).  Columns 8 c8 .. 8 c8 + 7 of row r:
template <int ROWS>
__device__ __forceinline__ void store_parts(uint32_t tile, uint32_t part_bytes, int r, int c8, const float* v) {
    uint32_t h[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split_pair(v[2 * e], v[2 * e + 1], h[0][e], h[1][e], h[2][e]);
    const uint32_t at = tile + (c8 >> 3) * ROWS * 128 + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + i * part_bytes), "r"(h[i][0]), "r"(h[i][1]), "r"(h[i][2]), "r"(h[i][3]) : "memory");
}

// acc (+)= A B over STEPS steps of 16 k.  a[i], b[i]: descriptors of the parts at their first k; a_step(k), b_step(k): what step k adds to one (16 bytes each).
template <int STEPS, typename FA, typename FB>
__device__ __forceinline__ void umma_parts(uint32_t acc, const uint64_t* a, const uint64_t* b, uint32_t idesc, bool accumulate, FA a_step, FB b_step) {
    Q6K_PARTS_ORDER;
#pragma unroll
    for (int e = 0; e < 6; ++e)
#pragma unroll
        for (int k = 0; k < STEPS; ++k) umma_ss(acc, a[PARTS_A[e]] + a_step(k), b[PARTS_B[e]] + b_step(k), idesc, accumulate || (e | k) != 0);
}
// A in tensor memory, `a_cols` columns a part (two entries of K a column).
template <int STEPS, typename FB>
__device__ __forceinline__ void umma_parts_ts(uint32_t acc, uint32_t a, uint32_t a_cols, const uint64_t* b, uint32_t idesc, bool accumulate, FB b_step) {
    Q6K_PARTS_ORDER;
#pragma unroll
    for (int e = 0; e < 6; ++e)
#pragma unroll
        for (int k = 0; k < STEPS; ++k) umma_ts(acc, a + PARTS_A[e] * a_cols + 8 * k, b[PARTS_B[e]] + b_step(k), idesc, accumulate || (e | k) != 0);
}

}  // namespace
