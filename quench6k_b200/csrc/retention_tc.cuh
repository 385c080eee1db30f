// Retention's chunks on the tensor cores: chunks of 128 tokens, heads of more than 64 and up to 128 keys, FP32 operands as three bfloat16 parts (parts.cuh).
// The same sums as the FP32 kernels' beside it (retention.cu), of the same precision:
//
//   ret_outer_tc_kernel   KV = K'^T V, K' the keys times their tokens' powers of d: [dk x dv] with the tokens as K, both operands as their rows lie
//   ret_out_tc_kernel     O_i = d^(i+1) (Q S)_i + (M V)_i,  M = (Q K^T) times d^(i-m) below the diagonal
//
// Shared memory holds the parts of two tiles of 128 x 128 (96 KB each); in ret_out_tc_kernel S takes the place of K when Q K^T is done, V that of S
// when Q S is, each fetched into registers before, and M goes from its accumulator through registers into tensor memory, the A operand of M V.
// A result that is not finite is summed again as the FP32 kernels do it: a value of a later token, were it infinite, must not reach an earlier one, and the
// zeros of M do not keep it away.
// Blocks walk the (head, chunk)s, the next one's rows on their way in registers under the last product of this one.  2,550 tokens in three portions, 16 heads
// of 128 x 128: 97 + 42 us with FP32 multiply-adds in chunks of 64, 52 + 34 us so, and the fold between them 15 -> 9.5 us (half as many states); the three
// launches together 100 us, 88 since sums of results that are not finite leave the products' registers alone.
// What bounds it: the phases of a block follow one another (rows from L2, the split, 1.6 us a product), and shared memory lets one block to an SM; the
// last round of blocks (336 on 148 SMs).  Distance to float64 of the state left behind and of the results: as before (the products' own is smaller).
#pragma once
#include "parts.cuh"

namespace {

constexpr int RT = 128, RT_THREADS = 512;                                    
constexpr uint32_t RT_PART = RT * RT * 2, RT_TILE = 3 * RT_PART;               // bytes of a part of a tile and of its three

__device__ int g_retention_tc_status = 0;

// This thread's share of a [128 x 128] tile of FP32 rows `ld` apart: units of 8 columns, unit (tid + 512 j) of 16 a row; zeros from row `rows` and column `cols` on.
__device__ __forceinline__ void rt_fetch(float (&v)[4][8], const float* src, size_t ld, int rows, int cols) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int u = threadIdx.x + RT_THREADS * j, r = u >> 4, c = (u & 15) * 8;
#pragma unroll
        for (int e = 0; e < 8; e += 4) load4(v[j] + e, src + (size_t)r * ld + c + e, r < rows && c + e < cols);
    }
}
__device__ __forceinline__ void rt_store(uint32_t tile, const float (&v)[4][8]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int u = threadIdx.x + RT_THREADS * j;
        store_parts<RT>(tile, RT_PART, u >> 4, u & 15, v[j]);
    }
}
// Tensor memory for the block and a barrier for its products; the address of the former.
__device__ __forceinline__ uint32_t rt_begin(uint32_t* slot, uint32_t bar, int cols) {
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();                                                                 // this block holds its tensor memory: a successor may come
    return *slot;
}
__device__ __forceinline__ void rt_end(uint32_t tmem, int cols) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    }
}
// What the block's threads stored is there for the tensor cores; one thread goes on to issue products.
__device__ __forceinline__ bool rt_issuer() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x >= 32) return false;
    tc_fence_after();
    return elect_one();
}
__device__ __forceinline__ bool rt_done(uint32_t bar, uint32_t parity) {
    const bool ok = mbar_wait(bar, parity);
    if (!ok) atomicExch(&g_retention_tc_status, 1);
    tc_fence_after();
    return ok;
}

// Where results are not finite, the whole block sums its tile again with multiply-adds, from rows in shared memory; only those that are not finite are taken.
// (A result at a time from global memory held a block up for 11 ms: 2,550 tokens with one key that is not a number 77 ms, so 0.24.)
constexpr int RP_LD = RT + 1, RP_STAGE = 132;                                 // floats a row: of an operand, of the results
// This thread's 4 x 8 sums: rows 4 (tid / 16) + r, columns tid % 16 + 16 c.  TRANS: A lies with the terms as rows; LOWER: terms up to a row's own only.
template <bool A_TRANS, bool B_TRANS, bool LOWER>
__device__ __forceinline__ void rp_product(float (&acc)[4][8], const float* A, const float* B, int terms) {
    const int tx = threadIdx.x & 15, r0 = (threadIdx.x >> 4) * 4;
    for (int i = 0; i < terms; ++i) {
        float b[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) b[c] = B_TRANS ? B[(tx + 16 * c) * RP_LD + i] : B[i * RP_LD + tx + 16 * c];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (LOWER && i > r0 + r) continue;
            const float a = A_TRANS ? A[i * RP_LD + r0 + r] : A[(r0 + r) * RP_LD + i];
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[r][c] = fmaf(a, b[c], acc[r][c]);
        }
    }
}
__device__ __forceinline__ void rp_fetch(float* to, const float* src, size_t ld, int rows, int cols) {
    for (int i = threadIdx.x; i < RT * RT; i += RT_THREADS) to[(i >> 7) * RP_LD + (i & 127)] = (i >> 7) < rows && (i & 127) < cols ? src[(size_t)(i >> 7) * ld + (i & 127)] : 0.0f;
}
__device__ __forceinline__ void rp_store(float* to, const float (&acc)[4][8], int ld) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) to[((threadIdx.x >> 4) * 4 + r) * ld + (threadIdx.x & 15) + 16 * c] = acc[r][c];
}
// K'^T V to smem [128][RP_STAGE].
__device__ __noinline__ void ret_outer_plain(float* smem, const float* k, const float* v, int ld, int n, int dk, int cols, const float* pw) {
    float *A = smem, *B = smem + RT * RP_LD, acc[4][8] = {};
    rp_fetch(A, k, ld, n, dk);
    rp_fetch(B, v, ld, n, cols);
    __syncthreads();
    for (int i = threadIdx.x; i < n * RT; i += RT_THREADS) A[(i >> 7) * RP_LD + (i & 127)] *= pw[i >> 7];
    __syncthreads();
    rp_product<true, false, false>(acc, A, B, n);
    __syncthreads();
    rp_store(smem, acc, RP_STAGE);
    __syncthreads();
}
// d^(i+1) (Q S)_i + (M V)_i to smem [128][RP_STAGE].
__device__ __noinline__ void ret_out_plain(float* smem, const float* q, const float* k, const float* v, const float* S, int ld, int dk, int dv, int n, int cols, const float* pw) {
    float *A = smem, *B = smem + RT * RP_LD, m[4][8] = {}, acc[4][8] = {};
    rp_fetch(A, q, ld, n, dk);
    rp_fetch(B, k, ld, n, dk);
    __syncthreads();
    rp_product<false, true, false>(m, A, B, dk);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) m[r][c] *= pw[max(0, (int)(threadIdx.x >> 4) * 4 + r - (int)(threadIdx.x & 15) - 16 * c)];       // above the diagonal nothing is read
    __syncthreads();
    for (int i = threadIdx.x; i < RT * RT; i += RT_THREADS) A[(i >> 7) * RP_LD + (i & 127)] *= pw[(i >> 7) + 1];
    rp_fetch(B, S, dv, dk, cols);
    __syncthreads();
    rp_product<false, false, false>(acc, A, B, dk);
    __syncthreads();
    rp_store(A, m, RP_LD);
    rp_fetch(B, v, ld, n, cols);
    __syncthreads();
    rp_product<false, false, true>(acc, A, B, n);
    __syncthreads();
    rp_store(smem, acc, RP_STAGE);
    __syncthreads();
}

// Task t of a launch: one (head, 128 value columns) of one chunk, the heads fastest.
struct RtTask {
    int head, col0, cols, chunk, first, n;
};
__device__ __forceinline__ RtTask rt_task(int t, const int* q_start, int R, int beyond, int H, int dv) {
    RtTask o;
    const int zb = (dv + 127) / 128;
    o.head = t % H, o.col0 = t / H % zb * 128, o.cols = min(128, dv - o.col0), o.chunk = t / (H * zb);
    o.first = o.n = 0;
    chunk_of<RT>(q_start, R, beyond, o.chunk, o.first, o.n);
    return o;
}

// Blocks walk the tasks (the last chunks may not exist: they end the walk).  grid min(tasks, SMs), 512 threads; KV: FP32 [chunks, H, dk, dv].
__global__ void __launch_bounds__(RT_THREADS, 1) ret_outer_tc_kernel(const float* kp, const float* vp, int ld, const float* decay, const int* q_start, int R, int beyond, float* KV, int H,
                                                                     int dk, int dv, int tasks) {
    pdl_wait();
    extern __shared__ uint8_t rt_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)rt_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bar_slot;
    __shared__ uint32_t tmem_slot;
    const uint32_t bar = smem_u32(&bar_slot), ks = smem_u32(smem), vs = ks + RT_TILE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
    __shared__ float pw[RT];
    const uint32_t tmem = rt_begin(&tmem_slot, bar, 128);
    RtTask task = rt_task(blockIdx.x, q_start, R, beyond, H, dv);
    float a[4][8], b[4][8];
    auto fetch = [&](const RtTask& x) {
        rt_fetch(a, kp + (size_t)x.first * ld + (size_t)x.head * dk, ld, x.n, dk);
        rt_fetch(b, vp + (size_t)x.first * ld + (size_t)x.head * dv + x.col0, ld, x.n, x.cols);
    };
    fetch(task);
    uint32_t parity = 0;
    for (int t = blockIdx.x; t < tasks && task.n > 0; t += gridDim.x) {
        const RtTask now = task;
        const float d = decay[now.head];
        const int n = now.n;
        if (threadIdx.x < RT) pw[threadIdx.x] = ret_power(d, threadIdx.x < n ? n - 1 - threadIdx.x : 0);
        rt_store(vs, b);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float p = pw[(threadIdx.x + RT_THREADS * j) >> 4];
#pragma unroll
            for (int e = 0; e < 8; ++e) a[j][e] *= p;
        }
        rt_store(ks, a);
        if (rt_issuer()) {
            uint64_t da[3], db[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) da[i] = umma_desc_mn(ks + i * RT_PART, RT * 128), db[i] = umma_desc_mn(vs + i * RT_PART, RT * 128);
            const auto step = [](int s) { return s * (2048 >> 4); };
            umma_parts<RT / 16>(tmem, da, db, umma_idesc_m128(128, true, true), false, step, step);
            umma_commit(bar);
        }
        task.n = 0;
        if (t + (int)gridDim.x < tasks) task = rt_task(t + gridDim.x, q_start, R, beyond, H, dv);
        fetch(task);                                                                // on its way under this task's products and stores
        const bool ok = rt_done(bar, parity);
        parity ^= 1;
        float acc[32];
        tmem_ld32_issue(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0, acc);
        tmem_ld_wait();
        float* stage = reinterpret_cast<float*>(smem) + row * RP_STAGE + c0;         // through shared memory, which no product reads any more: whole rows leave
        bool finite = true;
#pragma unroll
        for (int c = 0; c < 32; ++c) finite = finite && !(row < dk && c0 + c < now.cols && !(fabsf(acc[c]) <= 3.402823466e38f));
#pragma unroll
        for (int c = 0; c < 32; c += 4) *reinterpret_cast<float4*>(stage + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
        tc_fence_before();
        if (!__syncthreads_and(finite)) {
            ret_outer_plain(reinterpret_cast<float*>(smem), kp + (size_t)now.first * ld + (size_t)now.head * dk, vp + (size_t)now.first * ld + (size_t)now.head * dv + now.col0, ld, n, dk,
                            now.cols, pw);
#pragma unroll
            for (int c = 0; c < 32; ++c)
                if (fabsf(acc[c]) <= 3.402823466e38f) stage[c] = acc[c];
            fetch(task);                                                             // its registers need not outlast the sums above
            __syncthreads();
        }
        float* out = KV + ((size_t)now.chunk * H + now.head) * dk * dv + now.col0;
        if (ok)
            for (int i = threadIdx.x; i < dk * 32; i += RT_THREADS) {
                const int r = i >> 5, c = (i & 31) * 4;
                if (c < now.cols) *reinterpret_cast<float4*>(out + (size_t)r * dv + c) = *reinterpret_cast<const float4*>(reinterpret_cast<float*>(smem) + r * RP_STAGE + c);
            }
        if (!__syncthreads_and(ok)) break;                                          // all threads or none: a wait may run out in one and not in the next
    }
    rt_end(tmem, 128);
}

// The same walk; grid and threads as above.
__global__ void __launch_bounds__(RT_THREADS, 1) ret_out_tc_kernel(const float* qp, const float* kp, const float* vp, int ld, const float* decay, const float* KV, const int* q_start, int R,
                                                                   int beyond, float* o, int H, int dk, int dv, int tasks) {
    pdl_wait();
    extern __shared__ uint8_t rt_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)rt_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bar_slot;
    __shared__ uint32_t tmem_slot;
    __shared__ float pw[RT + 1];
    const uint32_t bar = smem_u32(&bar_slot), qs = smem_u32(smem), xs = qs + RT_TILE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const auto k_step = [](int s) { return (s >> 2) * (RT * 128 >> 4) + (s & 3) * 2; };
    const auto mn_step = [](int s) { return s * (2048 >> 4); };
    uint64_t dq[3], dx[3], dxm[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) dq[i] = umma_desc_k(qs + i * RT_PART), dx[i] = umma_desc_k(xs + i * RT_PART), dxm[i] = umma_desc_mn(xs + i * RT_PART, RT * 128);
    const uint32_t tmem = rt_begin(&tmem_slot, bar, 512), acc_m = tmem, acc_s = tmem + 128, parts_m = tmem + 256;       // M V goes where Q K^T was
    RtTask task = rt_task(blockIdx.x, q_start, R, beyond, H, dv);
    float a[4][8], b[4][8];
    auto fetch = [&](const RtTask& x) {
        const size_t at = (size_t)x.first * ld + (size_t)x.head * dk;
        rt_fetch(a, qp + at, ld, x.n, dk);
        rt_fetch(b, kp + at, ld, x.n, dk);
    };
    fetch(task);
    uint32_t parity = 0;
    for (int t = blockIdx.x; t < tasks && task.n > 0; t += gridDim.x) {
        const RtTask now = task;
        const int n = now.n;
        const float *v = vp + (size_t)now.first * ld + (size_t)now.head * dv + now.col0, *S = KV + ((size_t)now.chunk * H + now.head) * dk * dv + now.col0;
        if (threadIdx.x <= RT) pw[threadIdx.x] = ret_power(decay[now.head], threadIdx.x);
        rt_store(qs, a);
        rt_store(xs, b);
        if (rt_issuer()) {
            umma_parts<RT / 16>(acc_m, dq, dx, umma_idesc_m128(128, false), false, k_step, k_step);
            umma_commit(bar);
        }
        rt_fetch(a, S, dv, dk, now.cols);
        rt_fetch(b, v, ld, n, now.cols);
        bool ok = rt_done(bar, parity);
        rt_store(xs, a);
        if (rt_issuer()) {
            umma_parts<RT / 16>(acc_s, dq, dxm, umma_idesc_m128(128, true), false, k_step, mn_step);
            umma_commit(bar);
        }
        {   // M's parts: row i = this lane's token, columns m = c0 .. c0 + 31
            float m[32];
            tmem_ld32_issue(acc_m + lanes + c0, m);
            tmem_ld_wait();
            uint32_t h[3][16];
#pragma unroll
            for (int e = 0; e < 32; ++e) m[e] = c0 + e <= row ? m[e] * pw[row - c0 - e] : 0.0f;
#pragma unroll
            for (int e = 0; e < 16; ++e) split_pair(m[2 * e], m[2 * e + 1], h[0][e], h[1][e], h[2][e]);
#pragma unroll
            for (int i = 0; i < 3; ++i) tmem_st16(parts_m + lanes + i * (RT / 2) + c0 / 2, h[i]);
            tmem_st_wait();
        }
        ok = rt_done(bar, parity ^ 1) && ok;
        rt_store(xs, b);
        if (rt_issuer()) {
            umma_parts_ts<RT / 16>(acc_m, parts_m, RT / 2, dxm, umma_idesc_m128(128, true), false, mn_step);
            umma_commit(bar);
        }
        task.n = 0;
        if (t + (int)gridDim.x < tasks) task = rt_task(t + gridDim.x, q_start, R, beyond, H, dv);
        fetch(task);                                                                // on its way under the last product and the stores
        float x[32];
        ok = rt_done(bar, parity) && ok;
        parity ^= 1;
        const float p = pw[row + 1];
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
            float y[16];
            tmem_ld16_issue(acc_s + lanes + c0 + h, x + h);
            tmem_ld16_issue(acc_m + lanes + c0 + h, y);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 16; ++c) x[h + c] = fmaf(p, x[h + c], y[c]);
        }
        float* stage = reinterpret_cast<float*>(smem) + row * RP_STAGE + c0;
        bool finite = true;
#pragma unroll
        for (int c = 0; c < 32; ++c) finite = finite && !(row < n && c0 + c < now.cols && !(fabsf(x[c]) <= 3.402823466e38f));
#pragma unroll
        for (int c = 0; c < 32; c += 4) *reinterpret_cast<float4*>(stage + c) = make_float4(x[c], x[c + 1], x[c + 2], x[c + 3]);
        tc_fence_before();
        if (!__syncthreads_and(finite)) {
            const size_t at = (size_t)now.first * ld + (size_t)now.head * dk;
            ret_out_plain(reinterpret_cast<float*>(smem), qp + at, kp + at, v, S, ld, dk, dv, n, now.cols, pw);
#pragma unroll
            for (int c = 0; c < 32; ++c)
                if (fabsf(x[c]) <= 3.402823466e38f) stage[c] = x[c];
            fetch(task);
            __syncthreads();
        }
        if (ok)
            for (int i = threadIdx.x; i < n * 32; i += RT_THREADS) {
                const int r = i >> 5, c = (i & 31) * 4;
                if (c < now.cols)
                    *reinterpret_cast<float4*>(o + ((size_t)(now.first + r) * H + now.head) * dv + now.col0 + c) = *reinterpret_cast<const float4*>(reinterpret_cast<float*>(smem) + r * RP_STAGE + c);
            }
        if (!__syncthreads_and(ok)) break;                                          // all threads or none: a wait may run out in one and not in the next
    }
    rt_end(tmem, 512);
}

constexpr size_t RT_SMEM = 2 * RT_TILE + 1024;

}  // namespace
