// FP32 matrix products on the tensor cores, at FP32's own precision: the arithmetic of the true 32-bit path.
//
//   out[r, n] (+)= sum_k A[row(r), k] * W_g[n, k]        the contract of q6k_gemm_simt, FP32 operands
//
// An FP32 number is the sum of three bfloat16 numbers (8 significant bits each: x0 = x rounded, x1 = the rest rounded, x2 = what is left,
// exactly), and a product of two bfloat16 numbers is exact in FP32.  So a . w is taken as the six products a0 w0 + (a0 w1 + a1 w0) +
// (a1 w1 + a0 w2 + a2 w0) on tcgen05.mma; the three left out are below 2^-25 of a . w.  K goes in chunks of 64: within a chunk the
// small products are accumulated first, then a0 w0, in tensor memory; the chunks' sums are added in registers, in ascending order,
// with FP32 additions that round to nearest.  (Tensor memory truncates where it adds; four additions of full size a chunk instead of one
// for every 16 products of K keep that below the rounding of a sum in FP32.)  Every output is the same sequence of operations
// whatever its tile, its group and the rows beside it.  Against float64, K = 1,024 / 4,096: 1.1e-7 / 1.7e-7 of the results' norm (multiply-adds in
// four chains on CUDA cores: 2.9e-7 / 5.8e-7), largest 1.0e-6 / 1.8e-6 of their root mean square (2.4e-6 / 5.7e-6).
// An operand that is infinite, not a number or beyond bfloat16's largest (3.39e38) makes its outputs NaN above; an output that is not finite is
// therefore summed again with FP32 multiply-adds by the thread that stores it.  Parts of numbers below 2^-110 may be lost.
//
// A CTA makes [128 weight rows x BT tokens]; SwiGLU takes 64 rows of each matrix.
//   warps 0-7    split the weights: a thread a row and half of a chunk's k, from where the copies put them (rows of 128 bytes, swizzled) into
//                tensor memory, where the MMAs read them as their first operand
//   warps 8-15   fetch the tokens' rows two chunks ahead (32 bytes a thread, straight into registers: any row can be gathered), split them and
//                lay the three parts out in shared memory as the MMAs read them (K-major, 128-byte swizzle)
//   warp 16      tensor memory; one lane issues a chunk's 24 MMAs into one of two accumulators
//   warps 17-24  a chunk's sums from tensor memory into their own (a lane a weight row, a register a token, half of the tokens each); in the end the result
//   warp 25      one lane sends for the weights, 16 KB a copy
// What bounds it: shared memory's 128 bytes a clock.  A chunk of 64 tokens moves 168 KB there (32 in and 32 out of the weights, 56 of the tokens,
// 48 that the MMAs read): 1,310 clocks, and 1,340 were measured; with the weights' parts in shared memory too it was 312 KB and 2,700.
// (M x N x K, us, the multiply-adds of before in brackets) 509 x 1,536 x 1,024 18.2 (56.7), 509 x 1,024 x 4,096 51.5 (144), gate and up of
// 509 x 4,096 x 1,024 87 (229), 16 x 32,768 x 1,024 31.9 (73), 1 x 1,536 x 1,024 13.5 (21.3), 100 x 1,024 x 512 11.9 (12.6).
#include "umma.cuh"

namespace {

constexpr int FK = 64, FM = 128, F32_THREADS = 26 * 32, RAW_STAGES = 4, X_STAGES = 3, A_STAGES = 3;

enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_ACT = 4 };

__device__ int g_f32_status = 0;

constexpr uint32_t RAW_BYTES = FM * FK * 4, A_COLS = 3 * FK / 2;
__host__ __device__ constexpr int f32_smem_bytes(int bt) { return RAW_STAGES * (int)RAW_BYTES + X_STAGES * 3 * bt * 128; }

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

__device__ __noinline__ float plain_sum(const float* a, const float* w, int K) {
    float acc = 0.0f;
    for (int k = 0; k < K; ++k) acc = fmaf(a[k], w[k], acc);
    return acc;
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
                 : "memory");
}
// Four floats from `from`, or zeros; the registers are written by the load alone, so that nothing waits for it before their first use.
__device__ __forceinline__ void load4(float* v, const float* from, bool in) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
        "@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}" : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]) : "l"(from), "r"((int)in) : "memory");
}

// grid (ceil(N / 128), row tiles of BT (dense) or of the tile list), 832 threads; DUAL: ceil(N / 64).  WIDE: rows start on 16 bytes and K is a multiple of 4;
// else the weights' rows are read by the threads that split them.
template <int BT, int EPI, bool WIDE>
__global__ void __launch_bounds__(F32_THREADS, 1) gemm_f32_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_w2, const float* A, int lda,
                                                                const int* a_rows, const float* W, const float* W2, size_t w_group_stride, float* out, int ldo, int M, int N,
                                                                int K, const int* tile_group, const int* tile_row0, const int* group_offsets, const int* num_tiles, int act,
                                                                float act_limit) {
    pdl_enter();
    constexpr bool DUAL = EPI == EPI_SWIGLU;
    constexpr int ROWS_N = DUAL ? FM / 2 : FM, TMEM_COLS = 512;
    constexpr uint32_t X_BYTES = BT * 128;
    int g = 0, row0 = blockIdx.y * BT, row_end = M;
    if (tile_group) {
        if ((int)blockIdx.y >= *num_tiles) return;
        g = tile_group[blockIdx.y];
        row0 = tile_row0[blockIdx.y];
        row_end = group_offsets[g + 1];
    }
    if (row0 >= row_end) return;
    W += (size_t)g * w_group_stride;
    if (DUAL) W2 += (size_t)g * w_group_stride;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * (RAW_STAGES + X_STAGES + A_STAGES + 2)];
    __shared__ uint32_t tmem_slot;
    const uint32_t raw0 = smem_u32(smem), x0 = raw0 + RAW_STAGES * RAW_BYTES;
    const uint32_t raw_full = smem_u32(&bars[0]), raw_empty = raw_full + 8 * RAW_STAGES, x_full = raw_empty + 8 * RAW_STAGES, x_empty = x_full + 8 * X_STAGES;
    const uint32_t a_full = x_empty + 8 * X_STAGES, a_empty = a_full + 8 * A_STAGES, acc_full = a_empty + 8 * A_STAGES, acc_empty = acc_full + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = blockIdx.x * ROWS_N, chunks = (K + FK - 1) / FK, valid = min(BT, row_end - row0);
    if (threadIdx.x == 0) {
        for (int s = 0; s < RAW_STAGES; ++s) mbar_init(raw_full + 8 * s, 1), mbar_init(raw_empty + 8 * s, 8);
        for (int s = 0; s < X_STAGES; ++s) mbar_init(x_full + 8 * s, 8), mbar_init(x_empty + 8 * s, 1);
        for (int s = 0; s < A_STAGES; ++s) mbar_init(a_full + 8 * s, 8), mbar_init(a_empty + 8 * s, 1);
        for (int b = 0; b < 2; ++b) mbar_init(acc_full + 8 * b, 1), mbar_init(acc_empty + 8 * b, 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, tmem_a = tmem + 2 * BT;

    if (warp < 8) {
        const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane;
        const int n = n0 + (DUAL ? row & (ROWS_N - 1) : row);
        const float* src = n < N ? (DUAL && row >= ROWS_N ? W2 : W) + (size_t)n * K : nullptr;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        int rs = 0, as = 0;
        uint32_t r_phase = 0, a_phase = 1;
        for (int c = 0; c < chunks; ++c) {
            if ((WIDE && !mbar_wait(raw_full + 8 * rs, r_phase)) || !mbar_wait(a_empty + 8 * as, a_phase)) {
                if (lane == 0) atomicExch(&g_f32_status, 1);
                break;
            }
            tc_fence_after();
            const uint32_t from = raw0 + rs * RAW_BYTES + half * (RAW_BYTES / 2) + row * 128, to = tmem_a + as * A_COLS + half * 16 + lanes;
#pragma unroll
            for (int q = 0; q < 2; ++q) {                    // 16 of the 32 k at a time
                float x[16];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (WIDE) {
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[4 * u]), "=f"(x[4 * u + 1]), "=f"(x[4 * u + 2]), "=f"(x[4 * u + 3])
                                     : "r"(from + (((q * 4 + u) ^ (row & 7)) << 4)));
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int k = c * FK + half * 32 + q * 16 + u * 4 + e;
                            x[4 * u + e] = src && k < K ? src[k] : 0.0f;
                        }
                    }
                }
                uint32_t h[3][8];
#pragma unroll
                for (int e = 0; e < 8; ++e) split_pair(x[2 * e], x[2 * e + 1], h[0][e], h[1][e], h[2][e]);
#pragma unroll
                for (int i = 0; i < 3; ++i) tmem_st8(to + i * (FK / 2) + q * 8, h[i]);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (WIDE) mbar_arrive(raw_empty + 8 * rs);
                mbar_arrive(a_full + 8 * as);
            }
            if (++rs == RAW_STAGES) rs = 0, r_phase ^= 1;
            if (++as == A_STAGES) as = 0, a_phase ^= 1;
        }
    } else if (warp < 16) {
        // eight threads a row, each 8 of the chunk's 64 k; rows tid / 8 + 32 j
        constexpr int UNITS = BT / 32;
        const int part = threadIdx.x & 7, r0 = (threadIdx.x - 256) >> 3;
        const float* src[UNITS];
#pragma unroll
        for (int j = 0; j < UNITS; ++j) {
            const int t = r0 + 32 * j;
            src[j] = t < valid ? A + (size_t)(a_rows ? a_rows[row0 + t] : row0 + t) * lda : nullptr;
        }
        const uint32_t dst = x0 + r0 * 128 + ((part ^ (r0 & 7)) << 4);
        float x[2][UNITS][8];
        auto fetch = [&](float (&v)[UNITS][8], int c) {
            const int k = c * FK + part * 8;
#pragma unroll
            for (int j = 0; j < UNITS; ++j) {
                if (WIDE) {
                    load4(v[j], src[j] + k, src[j] && k < K);
                    load4(v[j] + 4, src[j] + k + 4, src[j] && k + 4 < K);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[j][e] = src[j] && k + e < K ? src[j][k + e] : 0.0f;
                }
            }
        };
        int s = 0;
        uint32_t phase = 1;
        bool ok = true;
        auto hand_over = [&](float (&v)[UNITS][8]) {
            if (!mbar_wait(x_empty + 8 * s, phase)) {
                if (lane == 0) atomicExch(&g_f32_status, 2);
                ok = false;
                return;
            }
#pragma unroll
            for (int j = 0; j < UNITS; ++j) {
                uint32_t h[3][4];
#pragma unroll
                for (int e = 0; e < 4; ++e) split_pair(v[j][2 * e], v[j][2 * e + 1], h[0][e], h[1][e], h[2][e]);
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + s * 3 * X_BYTES + i * X_BYTES + j * 32 * 128), "r"(h[i][0]), "r"(h[i][1]), "r"(h[i][2]), "r"(h[i][3])
                                 : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(x_full + 8 * s);
            if (++s == X_STAGES) s = 0, phase ^= 1;
        };
        fetch(x[0], 0);
        fetch(x[1], 1);
        for (int c = 0; c < chunks && ok; c += 2) {
            hand_over(x[0]);
            fetch(x[0], c + 2);
            if (c + 1 < chunks && ok) {
                hand_over(x[1]);
                fetch(x[1], c + 3);
            }
        }
    } else if (warp == 16) {
        if (elect_one()) {
            constexpr uint32_t idesc = umma_idesc_m128(BT, false);
            int xs = 0, as = 0;
            uint32_t x_phase = 0, a_phase = 0;
            for (int c = 0; c < chunks; ++c) {
                const int buf = c & 1;
                if (!mbar_wait(acc_empty + 8 * buf, ((c >> 1) & 1) ^ 1) || !mbar_wait(x_full + 8 * xs, x_phase) || !mbar_wait(a_full + 8 * as, a_phase)) {
                    atomicExch(&g_f32_status, 3);
                    break;
                }
                tc_fence_after();
                const uint32_t acc = tmem + buf * BT, w = tmem_a + as * A_COLS;
                uint64_t x[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) x[i] = umma_desc_k(x0 + (xs * 3 + i) * X_BYTES);
                constexpr int WI[6] = {0, 2, 1, 0, 1, 0}, XI[6] = {2, 0, 1, 1, 0, 0};      // the smallest first
#pragma unroll
                for (int e = 0; e < 6; ++e)
#pragma unroll
                    for (int k = 0; k < FK / 16; ++k) umma_ts(acc, w + WI[e] * (FK / 2) + 8 * k, x[XI[e]] + 2 * k, idesc, (e | k) != 0);
                umma_commit(x_empty + 8 * xs);
                umma_commit(a_empty + 8 * as);
                umma_commit(acc_full + 8 * buf);
                if (++xs == X_STAGES) xs = 0, x_phase ^= 1;
                if (++as == A_STAGES) as = 0, a_phase ^= 1;
            }
        }
    } else if (warp == 25) {
        if (WIDE && elect_one()) {
            int s = 0;
            uint32_t phase = 1;
            for (int c = 0; c < chunks; ++c) {
                if (!mbar_wait(raw_empty + 8 * s, phase)) {
                    atomicExch(&g_f32_status, 4);
                    break;
                }
                const uint32_t bar = raw_full + 8 * s, to = raw0 + s * RAW_BYTES;
                mbar_expect_tx(bar, RAW_BYTES);
#pragma unroll
                for (int h = 0; h < 2; ++h) {                // 32 k of every row: a row of 128 bytes
                    tma_load_3d(to + h * (RAW_BYTES / 2), &tm_w, c * FK + h * 32, n0, g, bar);
                    if (DUAL) tma_load_3d(to + h * (RAW_BYTES / 2) + ROWS_N * 128, &tm_w2, c * FK + h * 32, n0, g, bar);
                }
                if (++s == RAW_STAGES) s = 0, phase ^= 1;
            }
        }
    } else {
        // tensor memory's lane: the tile's weight row; and which half of the tokens
        constexpr int MINE = BT / 2;
        const int quarter = warp & 3, row = quarter * 32 + lane, t0 = (warp - 17) / 4 * MINE;
        float sum[MINE];
#pragma unroll
        for (int t = 0; t < MINE; ++t) sum[t] = 0.0f;
        bool ok = true;
        for (int c = 0; c < chunks; ++c) {
            const int buf = c & 1;
            if (!mbar_wait(acc_full + 8 * buf, (c >> 1) & 1)) {
                if (lane == 0) atomicExch(&g_f32_status, 5);
                ok = false;
                break;
            }
            tc_fence_after();
            float v[MINE];
            const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + buf * BT + t0;
            if constexpr (MINE == 32) tmem_ld32_issue(at, v);
            else tmem_ld16_issue(at, v);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty + 8 * buf);
#pragma unroll
            for (int j = 0; j < MINE; ++j) sum[j] += v[j];
        }
        const int n = n0 + (DUAL ? row & (ROWS_N - 1) : row), left = valid - t0;
        const bool mine = n < N && ok;
        const float* w_row = (DUAL && row >= ROWS_N ? W2 : W) + (size_t)(n < N ? n : 0) * K;
#pragma unroll
        for (int t = 0; t < MINE; ++t)                                                      // outputs that are not finite: once more, without parts
            if (mine && t < left && !(fabsf(sum[t]) <= 3.402823466e38f)) sum[t] = plain_sum(A + (size_t)(a_rows ? a_rows[row0 + t0 + t] : row0 + t0 + t) * lda, w_row, K);
        float* o = out + (size_t)(row0 + t0) * ldo + n;
        if (DUAL) {                                                                          // the up product's sums to the gate's threads, through the ring, which is done with
            float* ex = reinterpret_cast<float*>(smem) + t0 * ROWS_N + (row & (ROWS_N - 1));
            if (row >= ROWS_N && ok) {
#pragma unroll
                for (int t = 0; t < MINE; ++t) ex[t * ROWS_N] = sum[t];
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (row < ROWS_N && mine) {
#pragma unroll
                for (int t = 0; t < MINE; ++t)
                    if (t < left) {
                        const float up = ex[t * ROWS_N], v = sum[t];
                        o[(size_t)t * ldo] = act == 0 ? v / (1.0f + expf(-v)) * up : q6k_gated(v, up, act, act_limit);
                    }
            }
        } else if (mine) {
#pragma unroll
            for (int t1 = 0; t1 < MINE; t1 += 8) {
                float old[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) old[t] = EPI == EPI_ADD && t1 + t < left ? o[(size_t)(t1 + t) * ldo] : 0.0f;
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    if (t1 + t < left) o[(size_t)(t1 + t) * ldo] = EPI == EPI_ADD ? old[t] + sum[t1 + t] : EPI == EPI_ACT ? q6k_activation(sum[t1 + t], act) : sum[t1 + t];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// FP32 matrices [N, K], `stride` floats from one to the next, in boxes of [box_rows x 32 columns] of one of them, 128-byte swizzle; zeros beyond a
// matrix.  (How many there are is not known here: a tile list names only those that are.)
int make_f32_map(CUtensorMap* map, const void* base, size_t stride, int N, int K, int box_rows) {
    EncodeTiled fn = encode_fn();
    if (!fn) return q6k_fail("gemm_f32: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)N, stride ? 1u << 24 : 1u}, strides[2] = {(cuuint64_t)K * 4, (stride ? stride : (size_t)N * K) * 4};
    const cuuint32_t box[3] = {32u, (cuuint32_t)box_rows, 1u}, estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return q6k_fail("gemm_f32: cuTensorMapEncodeTiled failed with code %d (matrices of [%d, %d])", (int)r, N, K);
    return 0;
}

template <int BT, int EPI>
int launch_f32(bool wide, int tiles, cudaStream_t st, const float* A, int lda, const int* a_rows, const float* W, const float* W2, size_t w_group_stride, float* out,
               int ldo, int M, int N, int K, const int* tile_group, const int* tile_row0, const int* group_offsets, const int* num_tiles, int act, float act_limit) {
    constexpr int rows_n = EPI == EPI_SWIGLU ? FM / 2 : FM;
    constexpr size_t smem = (size_t)f32_smem_bytes(BT) + 1024;
    CUtensorMap tw{}, tw2{};
    if (wide) {
        if (int rc = make_f32_map(&tw, W, w_group_stride, N, K, rows_n)) return rc;
        if (EPI == EPI_SWIGLU)
            if (int rc = make_f32_map(&tw2, W2, w_group_stride, N, K, rows_n)) return rc;
    }
    auto* kernel = wide ? gemm_f32_kernel<BT, EPI, true> : gemm_f32_kernel<BT, EPI, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return q6k_check_launch("gemm_f32: shared memory attribute");
    q6k_launch(kernel, dim3((N + rows_n - 1) / rows_n, tiles), F32_THREADS, smem, st, tw, tw2, A, lda, a_rows, W, W2, w_group_stride, out, ldo, M, N, K, tile_group, tile_row0,
               group_offsets, num_tiles, act, act_limit);
    return q6k_check_launch("gemm_f32");
}

}  // namespace

Q6K_API int q6k_gemm_f32_status() {
    int v = -1;
    if (cudaMemcpyFromSymbol(&v, g_f32_status, sizeof v) != cudaSuccess) return -1;
    return v;
}

// q6k_gemm_simt's arguments, already checked there; grouped row tiles of 64.
int q6k_gemm_f32(const float* A, int lda, const int* a_rows, const float* W, const float* W2, size_t w_group_stride, float* out, int ldo, int M, int N, int K, const int* tile_group,
                 const int* tile_row0, const int* group_offsets, const int* num_tiles, int max_tiles, int epilogue, int act, float act_limit, cudaStream_t st) {
    const bool wide = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W | (uintptr_t)W2) & 15) == 0 && w_group_stride % 4 == 0;
    // up to 32 rows (in all groups together): tiles of 32 tokens (1 x 1,024 x 4,096: 41.5 us, 51.5 with tiles of 64)
    const int bt = M <= 32 ? 32 : 64, tiles = tile_group ? max_tiles : (M + bt - 1) / bt;
#define GO(BT_, EPI_) launch_f32<BT_, EPI_>(wide, tiles, st, A, lda, a_rows, W, W2, w_group_stride, out, ldo, M, N, K, tile_group, tile_row0, group_offsets, num_tiles, act, act_limit)
#define GO_EPI(BT_) epilogue == EPI_STORE ? GO(BT_, EPI_STORE) : epilogue == EPI_ADD ? GO(BT_, EPI_ADD) : epilogue == EPI_ACT ? GO(BT_, EPI_ACT) : GO(BT_, EPI_SWIGLU)
    return bt == 32 ? GO_EPI(32) : GO_EPI(64);
#undef GO_EPI
#undef GO
}
