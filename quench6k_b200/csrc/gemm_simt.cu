// Matrix products on CUDA cores with FP32 fused multiply-adds: the arithmetic of the true 32-bit
// path, and the fallback of the bfloat16 path for shapes the tensor-core kernels refuse.
//
//   out[r, n] (+)= sum_k A[row(r), k] * W_g[n, k]        (W is [N, K], K contiguous, as the
//   reference stores its projection weights: crates/engine/src/flint.rs:293-300)
//
// Rows may be grouped (one weight matrix per group: the experts of a MoE layer, as the reference
// runs them through one grouped kernel, crates/cuda/kernels/moe.cu:142-255) and may be gathered
// through an index.  With two weight matrices the epilogue is SwiGLU: out = silu(A.Wg) * (A.Wu).
//
// Each output element is summed over k in an order that follows from K alone, so its value does not
// depend on which tile or batch the row was in.
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16;

enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_ACT = 4 };      // EPI_ACT: one matrix, out = T(act(A.W))

template <typename T, int EPI>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const T* A, int lda, const int* a_rows, const T* W, const T* W2,
                                                        size_t w_group_stride, void* out_, int ldo, int M, int N, int K,
                                                        const int* tile_group, const int* tile_row0,
                                                        const int* group_offsets, const int* num_tiles, int act, float act_limit) {
    pdl_enter();
    constexpr bool DUAL = EPI == EPI_SWIGLU;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ float Ws2[DUAL ? BK : 1][BN + 4];
    int g = 0, row0 = blockIdx.y * BM, row_end = M;
    if (tile_group) {
        if ((int)blockIdx.y >= *num_tiles) return;
        g = tile_group[blockIdx.y];
        row0 = tile_row0[blockIdx.y];
        row_end = group_offsets[g + 1];
    }
    if (row0 >= row_end) return;
    const int n0 = blockIdx.x * BN;
    const T* Wg = W + (size_t)g * w_group_stride;
    const T* Wg2 = DUAL ? W2 + (size_t)g * w_group_stride : nullptr;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    // loader: this thread brings 4 consecutive k of one tile row of A and of W
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    const int arow_g = row0 + lr;
    const T* a_src = nullptr;
    if (arow_g < row_end) a_src = A + (size_t)(a_rows ? a_rows[arow_g] : arow_g) * lda;
    const T* w_src = (n0 + lr < N) ? Wg + (size_t)(n0 + lr) * K : nullptr;
    const T* w2_src = (DUAL && n0 + lr < N) ? Wg2 + (size_t)(n0 + lr) * K : nullptr;

    float acc[4][4] = {}, acc2[DUAL ? 4 : 1][4] = {};
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            As[lk + i][lr] = (a_src && k < K) ? to_f32(a_src[k]) : 0.0f;
            Ws[lk + i][lr] = (w_src && k < K) ? to_f32(w_src[k]) : 0.0f;
            if (DUAL) Ws2[lk + i][lr] = (w2_src && k < K) ? to_f32(w2_src[k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4], b[4], b2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[k][tx * 4 + j];
            if (DUAL) {
#pragma unroll
                for (int j = 0; j < 4; ++j) b2[j] = Ws2[k][tx * 4 + j];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
                    if (DUAL) acc2[i][j] = fmaf(a[i], b2[j], acc2[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= row_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            const size_t o = (size_t)r * ldo + n;
            if (EPI == EPI_STORE) {
                ((float*)out_)[o] = acc[i][j];
            } else if (EPI == EPI_ADD) {
                ((float*)out_)[o] += acc[i][j];
            } else if (EPI == EPI_ACT) {
                ((T*)out_)[o] = from_f32<T>(q6k_activation(acc[i][j], act));
            } else {
                const float gte = acc[i][j];
                ((T*)out_)[o] = from_f32<T>(act == 0 ? gte / (1.0f + expf(-gte)) * acc2[DUAL ? i : 0][j] : q6k_gated(gte, acc2[DUAL ? i : 0][j], act, act_limit));
            }
        }
    }
}

// FP32 operands.  The kernel above loads one value at a time into a transposed tile that everyone then waits for, and leaves the
// multipliers idle two thirds of the time.  Here rows go to shared memory as they lie, 16 bytes a copy, two blocks of 32 k ahead of the one in
// use, and the products go through the packed multiply-add, which takes two FP32 products an instruction: with operands read four k at a time,
// the even and the odd k of an output are its two halves, so nothing has to be rearranged.  An output is then four sums over ascending k (even and
// odd, of either half of each block of 32), added in the end: no larger an error than one sum, and the same for a row whatever its tile.
// A block makes 32 x 64 outputs, half of its threads the first 16 k of every block and half the others: small enough that 512
// rows fill the chip and that experts of some 60 rows waste little, with 4 x 4 outputs a thread all the same (8 loads of 16 bytes
// for 64 products; rows 144 bytes apart, so that eight threads' reads fall into different banks).
// The 20 products of a step of 509 tokens through four layers (1,024 wide, experts of 512): 1,835 -> 1,670 us against tiles of 64 x 64 with
// an instruction per product (2,930 us with the kernel above).  What bounds it now: the FP32 pipe, half of its cycles, and reads of
// shared memory, two thirds (3.3 wavefronts a read).  Warps of 8 x 128 outputs, whose reads of one address were to cost less, took 2,100 us.
// WIDE: rows start on 16 bytes and K is a multiple of 4; else copies of 4 bytes.
constexpr int FM = 32, FN = 64, FK = 32, FLD = FK + 4, FSTAGES = 3;
static_assert(BM == 2 * FM, "a tile of the tile lists is two of these");

__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum_pair(unsigned long long v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }

// grid (ceil(N / 64), tiles of 64 rows, 2), 256 threads.
template <int EPI, bool WIDE>
__global__ void __launch_bounds__(256, 2) gemm_f32_kernel(const float* A, int lda, const int* a_rows, const float* W, const float* W2,
                                                                                  size_t w_group_stride, float* out, int ldo, int M, int N, int K,
                                                                                  const int* tile_group, const int* tile_row0, const int* group_offsets,
                                                                                  const int* num_tiles, int act, float act_limit) {
    pdl_enter();
    constexpr bool DUAL = EPI == EPI_SWIGLU;
    constexpr int MATS = DUAL ? 2 : 1, STAGE = (FM + MATS * FN) * FLD;
    extern __shared__ __align__(16) float f_smem[];          // [FSTAGES][A 32 rows | W 64 | W2 64][FLD]
    int g = 0, row0 = blockIdx.y * BM, row_end = M;
    if (tile_group) {
        if ((int)blockIdx.y >= *num_tiles) return;
        g = tile_group[blockIdx.y];
        row0 = tile_row0[blockIdx.y];
        row_end = group_offsets[g + 1];
    }
    row0 += blockIdx.z * FM;
    if (row0 >= row_end) return;
    const int n0 = blockIdx.x * FN, tid = threadIdx.x;
    // loader: WIDE pieces of 4 k of rows tid / 8 (+ 32), else single k of rows tid / 32 + 8 e
    constexpr int STEP = WIDE ? 32 : 8, A_ROWS = FM / STEP, W_ROWS = FN / STEP;
    const int lr = WIDE ? tid >> 3 : tid >> 5, lk = WIDE ? (tid & 7) * 4 : tid & 31;
    const float *a_src[A_ROWS], *w_src[MATS][W_ROWS];
#pragma unroll
    for (int e = 0; e < A_ROWS; ++e) {
        const int r = row0 + lr + e * STEP;
        a_src[e] = r < row_end ? A + (size_t)(a_rows ? a_rows[r] : r) * lda : nullptr;
    }
#pragma unroll
    for (int e = 0; e < W_ROWS; ++e) {
        const int n = n0 + lr + e * STEP;
        w_src[0][e] = n < N ? W + (size_t)g * w_group_stride + (size_t)n * K : nullptr;
        if (DUAL) w_src[MATS - 1][e] = n < N ? W2 + (size_t)g * w_group_stride + (size_t)n * K : nullptr;
    }
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(f_smem);
    const int blocks = (K + FK - 1) / FK;
    auto fetch = [&](int b) {
        if (b < blocks) {
            const int k = b * FK + lk;
            const uint32_t at = base + 4 * ((b % FSTAGES) * STAGE + lr * FLD + lk);
            auto copy = [&](const float* row, int to_row) {
                const bool in = row != nullptr && k < K;
                const float* from = in ? row + k : A;
                if (WIDE) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + 4 * to_row * FLD), "l"(from), "r"(in ? 16 : 0) : "memory");
                else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at + 4 * to_row * FLD), "l"(from), "r"(in ? 4 : 0) : "memory");
            };
#pragma unroll
            for (int e = 0; e < A_ROWS; ++e) copy(a_src[e], e * STEP);
#pragma unroll
            for (int m = 0; m < MATS; ++m)
#pragma unroll
                for (int e = 0; e < W_ROWS; ++e) copy(w_src[m][e], FM + m * FN + e * STEP);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // this thread's outputs: rows ty + 4 i, columns tx + 8 j; its k: 16 of each block's 32
    const int half = tid >> 7, warp = (tid >> 5) & 3, lane = tid & 31, tx = (warp & 1) * 32 + (lane & 7), ty = (warp >> 1) * 16 + (lane >> 3);
    unsigned long long acc[MATS][4][4] = {};
    fetch(0);
    fetch(1);
    for (int b = 0; b < blocks; ++b) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                     // this block has landed for everyone; the one before it is done with
        fetch(b + 2);
        const float* As = f_smem + (b % FSTAGES) * STAGE + ty * FLD + half * (FK / 2);
        const float* Ws = f_smem + (b % FSTAGES) * STAGE + (FM + tx) * FLD + half * (FK / 2);
#pragma unroll
        for (int k = 0; k < FK / 2; k += 4) {
            ulonglong2 a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(As + i * 4 * FLD + k);
#pragma unroll
            for (int m = 0; m < MATS; ++m) {
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(Ws + (m * FN + j * 8) * FLD + k);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma_pair(acc[m][i][j], a[i].x, w[j].x);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma_pair(acc[m][i][j], a[i].y, w[j].y);
            }
        }
    }
    // the second half of the threads hands its sums over
    __syncthreads();
    float* sums = f_smem + (tid & 127);                      // [matrix, i, j][128 threads]
    if (half == 1) {
#pragma unroll
        for (int e = 0; e < MATS * 16; ++e) sums[e * 128] = sum_pair(acc[e / 16][e / 4 % 4][e % 4]);
    }
    __syncthreads();
    if (half == 1) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty + 4 * i;
        if (r >= row_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + 8 * j;
            if (n >= N) continue;
            float* o = out + (size_t)r * ldo + n;
            const float v = sum_pair(acc[0][i][j]) + sums[(i * 4 + j) * 128];
            if (EPI == EPI_STORE) *o = v;
            else if (EPI == EPI_ADD) *o += v;
            else if (EPI == EPI_ACT) *o = q6k_activation(v, act);
            else {
                const float up = sum_pair(acc[MATS - 1][i][j]) + sums[(MATS * 16 - 16 + i * 4 + j) * 128];
                *o = act == 0 ? v / (1.0f + expf(-v)) * up : q6k_gated(v, up, act, act_limit);
            }
        }
    }
}

template <int EPI>
int launch_f32(dim3 grid, bool wide, cudaStream_t st, const float* A, int lda, const int* a_rows, const float* W, const float* W2, size_t w_group_stride,
               float* out, int ldo, int M, int N, int K, const int* tile_group, const int* tile_row0, const int* group_offsets, const int* num_tiles, int act,
               float act_limit) {
    const size_t smem = (size_t)FSTAGES * (FM + (EPI == EPI_SWIGLU ? 2 : 1) * FN) * FLD * sizeof(float);
    grid.z = BM / FM;
    auto* kernel = wide ? gemm_f32_kernel<EPI, true> : gemm_f32_kernel<EPI, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return q6k_check_launch("gemm_f32: shared memory attribute");
    q6k_launch(kernel, grid, 256, smem, st, A, lda, a_rows, W, W2, w_group_stride, out, ldo, M, N, K, tile_group, tile_row0, group_offsets, num_tiles, act, act_limit);
    return q6k_check_launch("gemm_f32");
}

// Row tiles of the groups: for offsets[0..G] the list of (group, first row) of every BM-row tile.
// One block; groups are walked in order so the list is a function of the offsets only.
__global__ void tile_list_kernel(const int* offsets, int G, int bm, int* tile_group, int* tile_row0, int* num_tiles,
                                 int max_tiles) {
    pdl_enter();
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int g0 = 0; g0 < G; g0 += blockDim.x) {
        const int g = g0 + threadIdx.x;
        int mine = 0;
        if (g < G) mine = (offsets[g + 1] - offsets[g] + bm - 1) / bm;
        // exclusive scan over the block in group order (serial over warps is fine: G is small)
        __shared__ int scan[1024];
        scan[threadIdx.x] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = base;
            for (int i = 0; i < (int)blockDim.x; ++i) {
                const int c = scan[i];
                scan[i] = run;
                run += c;
            }
            base = run;
        }
        __syncthreads();
        if (g < G) {
            const int first = scan[threadIdx.x];
            for (int i = 0; i < mine; ++i)
                if (first + i < max_tiles) {
                    tile_group[first + i] = g;
                    tile_row0[first + i] = offsets[g] + i * bm;
                }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *num_tiles = base < max_tiles ? base : max_tiles;
}

}  // namespace

Q6K_API int q6k_gemm_tile_rows() { return BM; }

Q6K_API int q6k_tile_list(const int* offsets, int G, int bm, int* tile_group, int* tile_row0, int* num_tiles,
                          int max_tiles, cudaStream_t st) {
    Q6K_REQUIRE(G > 0 && bm > 0 && max_tiles > 0, "tile_list: bad sizes G=%d bm=%d max_tiles=%d", G, bm, max_tiles);
    q6k_launch(tile_list_kernel, 1, 256, 0, st, offsets, G, bm, tile_group, tile_row0, num_tiles, max_tiles);
    return q6k_check_launch("tile_list");
}

// epilogue: 0 store FP32, 1 add into FP32, 2 act(A.W) * (A.W2) stored in the operand dtype (SwiGLU with activation 0), 4 act(A.W)
// stored in the operand dtype; the activation's code above bit 8.
// Grouped when tile_group != null (max_tiles bounds the tile list; group_offsets has one more entry
// than there are groups); otherwise one group of M rows.
Q6K_API int q6k_gemm_simt(const void* A, int lda, const int* a_rows, const void* W, const void* W2, long long w_group_stride,
                          void* out, int ldo, int M, int N, int K, const int* tile_group, const int* tile_row0,
                          const int* group_offsets, const int* num_tiles, int max_tiles, int epilogue, float act_param, int dtype,
                          cudaStream_t st) {
    if (M == 0 || N == 0) return 0;
    Q6K_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    const int act = epilogue >> 8;
    epilogue &= 255;
    Q6K_REQUIRE(((epilogue >= 0 && epilogue <= 2) || epilogue == EPI_ACT) && act >= 0 && act <= (epilogue == EPI_SWIGLU ? 3 : 2),
                "gemm: unknown epilogue %d (activation %d)", epilogue, act);
    Q6K_REQUIRE(epilogue != EPI_SWIGLU || W2, "gemm: the SwiGLU epilogue needs two weight matrices");
    const int ytiles = tile_group ? max_tiles : (M + BM - 1) / BM;
    Q6K_REQUIRE(ytiles <= 65535, "gemm: %d row tiles exceed the grid limit", ytiles);
    dim3 grid((N + BN - 1) / BN, ytiles);
    if (dtype == Q6K_F32) {
        const bool wide = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W | (uintptr_t)W2) & 15) == 0 && w_group_stride % 4 == 0;
#define LAUNCH_F32(EPI) launch_f32<EPI>(grid, wide, st, (const float*)A, lda, a_rows, (const float*)W, (const float*)W2, (size_t)w_group_stride, (float*)out, ldo, M, N, K, \
                                        tile_group, tile_row0, group_offsets, num_tiles, act, act_param)
        if (epilogue == EPI_STORE) return LAUNCH_F32(EPI_STORE);
        if (epilogue == EPI_ADD) return LAUNCH_F32(EPI_ADD);
        if (epilogue == EPI_ACT) return LAUNCH_F32(EPI_ACT);
        return LAUNCH_F32(EPI_SWIGLU);
#undef LAUNCH_F32
    }
    using T = __nv_bfloat16;
#define LAUNCH(EPI)                                                                                                     \
    q6k_launch(gemm_simt_kernel<T, EPI>, grid, 256, 0, st, (const T*)A, lda, a_rows, (const T*)W, (const T*)W2,                 \
                                                   (size_t)w_group_stride, out, ldo, M, N, K, tile_group, tile_row0, \
                                                   group_offsets, num_tiles, act, act_param)
    Q6K_REQUIRE(dtype == Q6K_BF16, "unknown dtype code %d", dtype);
    if (epilogue == EPI_STORE) LAUNCH(EPI_STORE);
    else if (epilogue == EPI_ADD) LAUNCH(EPI_ADD);
    else if (epilogue == EPI_ACT) LAUNCH(EPI_ACT);
    else LAUNCH(EPI_SWIGLU);
#undef LAUNCH
    return q6k_check_launch("gemm_simt");
}
