// Retention: linear attention with one fixed decay per head and neither softmax nor denominator.  Per head, with a
// state S [dk, dv] that starts at zero and is carried from token to token in the request's state slot:
//
//     S <- decay S + k v^T;      o = S^T q
//
//  * retention_prep_kernel turns the first `rd` dimensions of every head of q and k by position * inv_freq[pair] (pairs by
//    halves, or of neighbours) and multiplies k by a scale, in place on the FP32 result of the projection; a block per token.
//    Before that it may pass the row's first `act_cols` columns (q, k and v of a mixer that activates them) through silu.
//  * retention_kernel walks a request's tokens in order.  A block owns 16 columns of one head of one request; a thread holds
//    a stretch of consecutive rows of ONE column in registers (lane = column and one of two stretches, eight warps = sixteen
//    stretches), so k and q of its rows come as 16-byte reads every lane of a half-warp shares and a token costs three
//    floating-point instructions per element of the state and little else.  A token's sum over the rows is the thread's own
//    (in row order), then the two stretches of a warp (one shuffle), then the eight warps' through shared memory, in the
//    warps' order: the same tree for every token wherever a prompt was cut.  q, k and v of eight tokens at a time are
//    copied to shared memory asynchronously, three tiles ahead of the one that is walked (a tile's first read is a miss in
//    L2 for one block of a head, and its latency is several times a tile's work).
//
// The same walk serves a second recurrence (TM below): a decay per token and key channel, the read-out before the write, and
// the current token entering the read-out through a bonus vector u per head,
//
//     o = S^T r + (sum_x u[x] k[x] r[x]) v;      S <- diag(w) S + k v^T
//
//  * token_shift_kernel makes what its projections read: per token n mixes x + (x' - x) mu_j of the token's row with the row
//    before it (x' = 0 for a sequence's first token; the row before a portion is kept in the request's state slot).
//  * time_mix_prep_kernel makes the decays w = exp(-exp(z + w0)) in place and the token's bonus number per head.
//
// Everything is FP32: angles, the rotation, decays and their powers, the state and every sum.
#include "chunks.cuh"

namespace {

constexpr int RET_WARPS = 8, RET_THREADS = RET_WARPS * 32, RET_COLS = 16, RET_CHUNKS = 2 * RET_WARPS, RET_TILE = 8, RET_STAGES = 4, RET_MAX_DK = 256;

// One block per token: the sines and cosines of its rd / 2 angles are made once (they are the same for every head, for q
// and for k), then every pair of q and of k is turned in place and the rest of k scaled; what neither turns nor scales
// is not touched.
__global__ void __launch_bounds__(256) retention_prep_kernel(float* p, int ld, int H, int dk, int q_col, int k_col,
                                                             const float* inv_freq, int rd, int neighbours, float k_scale,
                                                             const int* positions, int act_cols) {
    pdl_enter();
    extern __shared__ float xs[];            // cos [rd / 2] | sin [rd / 2]
    const int t = blockIdx.x, half = rd / 2;
    const float pos = (float)positions[t];
    for (int i = threadIdx.x; i < half; i += blockDim.x) sincosf(pos * inv_freq[i], &xs[half + i], &xs[i]);
    float* row = p + (size_t)t * ld;
    for (int c = threadIdx.x; c < act_cols; c += blockDim.x) {             // silu on the projections, before anything else
        const float z = row[c];
        row[c] = z / (1.0f + expf(-z));
    }
    __syncthreads();
    for (int w = threadIdx.x; w < 2 * H * half; w += blockDim.x) {          // (q or k, head, pair)
        const int i = w % half, h = (w / half) % H, is_k = w / (half * H);
        float* x = row + (is_k ? k_col : q_col) + (size_t)h * dk;
        const int a = neighbours ? 2 * i : i, b = neighbours ? 2 * i + 1 : i + half;
        const float u = x[a], v = x[b], cs = xs[i], sn = xs[half + i], mul = is_k ? k_scale : 1.0f;
        x[a] = (u * cs - v * sn) * mul;
        x[b] = (v * cs + u * sn) * mul;
    }
    if (k_scale != 1.0f) {
        const int rest = dk - rd;
        for (int w = threadIdx.x; w < H * rest; w += blockDim.x) {
            float* x = row + k_col + (size_t)(w / rest) * dk + rd + w % rest;
            *x *= k_scale;
        }
    }
}

// The same for halves that pair up 16 bytes at a time (rd / 2 a multiple of 4, rows and heads on 16 bytes, no activation before it): a
// thread asks for two pairs before the angles are made.  26 us for 2,550 tokens of 16 heads of 128, 84 MB, four bytes at a time;
// this one takes 14.
__global__ void __launch_bounds__(256) retention_turn4_kernel(float* p, int ld, int H, int dk, int q_col, int k_col, const float* inv_freq, int rd, float k_scale,
                                                              const int* positions) {
    pdl_enter();
    extern __shared__ __align__(16) float xs[];            // cos [rd / 2] | sin [rd / 2]
    const int t = blockIdx.x, half = rd / 2, half4 = half / 4, all = 2 * H * half4;
    float* row = p + (size_t)t * ld;
    auto at = [&](int w) { return row + (w >= all / 2 ? k_col : q_col) + (size_t)(w / half4 % H) * dk + w % half4 * 4; };      // (q or k, head, four pairs)
    bool made = false;
    for (int w0 = threadIdx.x; w0 < all || !made; w0 += 512) {
        float4 u[2], v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (w0 + 256 * e < all) {
                const float* x = at(w0 + 256 * e);
                u[e] = *reinterpret_cast<const float4*>(x), v[e] = *reinterpret_cast<const float4*>(x + half);
            }
        if (!made) {
            const float pos = (float)positions[t];
            for (int i = threadIdx.x; i < half; i += 256) sincosf(pos * inv_freq[i], &xs[half + i], &xs[i]);
            __syncthreads();
            made = true;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (w0 + 256 * e < all) {
                float* x = at(w0 + 256 * e);
                const int i = (w0 + 256 * e) % half4 * 4;
                const float mul = w0 + 256 * e >= all / 2 ? k_scale : 1.0f;
                const float4 c = *reinterpret_cast<const float4*>(xs + i), s = *reinterpret_cast<const float4*>(xs + half + i);
                *reinterpret_cast<float4*>(x) = make_float4((u[e].x * c.x - v[e].x * s.x) * mul, (u[e].y * c.y - v[e].y * s.y) * mul,
                                                            (u[e].z * c.z - v[e].z * s.z) * mul, (u[e].w * c.w - v[e].w * s.w) * mul);
                *reinterpret_cast<float4*>(x + half) = make_float4((v[e].x * c.x + u[e].x * s.x) * mul, (v[e].y * c.y + u[e].y * s.y) * mul,
                                                                   (v[e].z * c.z + u[e].z * s.z) * mul, (v[e].w * c.w + u[e].w * s.w) * mul);
            }
    }
    if (k_scale != 1.0f) {
        const int rest = dk - rd;
        for (int w = threadIdx.x; w < H * rest; w += 256) row[k_col + (size_t)(w / rest) * dk + rd + w % rest] *= k_scale;
    }
}

// Four bytes from global to shared memory without passing registers; `in` false writes a zero and reads nothing.
__device__ __forceinline__ void ret_copy(float* dst, const float* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = in ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void ret_copy16(float* dst, const float* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = in ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// grid (R, H, ceil(dv / 16)), 256 threads.  qp, kp (prepared), vp: FP32, a token's heads side by side, rows ld apart; state: FP32
// [slots, H, dk, dv]; o: FP32 [T, H dv].  RPT: rows per thread (dk <= 16 RPT).  STAGES tiles are in flight or in use.
// WIDE: every head's q and k (and decays) start on 16 bytes in every row and dk is a multiple of 4 (copies of 16 bytes).
// TM: the second recurrence; q is r, wt: FP32 [T, ld_w] with the decays of head h from column h dk on, bonus: FP32 [T, H].
// Requests of more than `most` tokens are not this launch's.
template <int RPT, int STAGES, bool WIDE, bool TM>
__global__ void __launch_bounds__(RET_THREADS) retention_kernel(const float* qp, const float* kp, const float* vp, int ld, const float* decay,
                                                                const float* wt, int ld_w, const float* bonus, float* state, const int* q_start,
                                                                const int* slot_ids, float* o, int H, int dk, int dv, int most) {
    pdl_enter();
    constexpr int DKP = RET_CHUNKS * RPT;                                // rows, padded
    constexpr int PER_THREAD = RET_TILE * DKP / RET_THREADS;             // elements of q (and of k) a thread stages per tile
    static_assert(RPT % 4 == 0 && RET_TILE * DKP % RET_THREADS == 0 && RET_TILE * RET_COLS <= RET_THREADS, "16-byte reads; a tile divides among the threads");
    // q [STAGES][TILE][DKP] | k likewise | (TM: decays likewise) | v [STAGES][TILE][COLS] | sums [2][TILE][WARPS][COLS] | (TM: bonus [STAGES][TILE])
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;
    float* ks = qs + STAGES * RET_TILE * DKP;
    float* ws = ks + STAGES * RET_TILE * DKP;
    float* vs = ws + (TM ? STAGES * RET_TILE * DKP : 0);
    float* red = vs + STAGES * RET_TILE * RET_COLS;
    float* bs = red + 2 * RET_TILE * RET_WARPS * RET_COLS;
    const int r = blockIdx.x, head = blockIdx.y, c0 = blockIdx.z * RET_COLS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cl = lane % RET_COLS, col = c0 + cl;
    const int row0 = (warp * 2 + lane / RET_COLS) * RPT;                 // this thread's first row
    const int t0 = q_start[r], t1 = q_start[r + 1];
    if (t0 >= t1 || t1 - t0 > most) return;
    const float d = TM ? 0.0f : decay[head];
    float* mine = state + ((size_t)slot_ids[r] * H + head) * dk * dv + (col < dv ? col : 0);
    float s[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) s[i] = (col < dv && row0 + i < dk) ? mine[(size_t)(row0 + i) * dv] : 0.0f;
    auto fetch = [&](int ta, int b) {         // this thread's share of the tile that starts at token ta, on its way to buffer b
        const int n = min(RET_TILE, t1 - ta);
        if (n > 0) {
            if (WIDE) {
#pragma unroll
                for (int e = 0; e < (PER_THREAD + 3) / 4; ++e) {
                    const int i = (threadIdx.x + e * RET_THREADS) * 4, tt = i / DKP, row = i % DKP;
                    if (PER_THREAD >= 4 || i < RET_TILE * DKP) {
                        const bool in = tt < n && row < dk;
                        const size_t at = in ? (size_t)(ta + tt) * ld + (size_t)head * dk + row : 0;
                        ret_copy16(qs + b * RET_TILE * DKP + i, qp + at, in);
                        ret_copy16(ks + b * RET_TILE * DKP + i, kp + at, in);
                        if (TM) ret_copy16(ws + b * RET_TILE * DKP + i, in ? wt + (size_t)(ta + tt) * ld_w + (size_t)head * dk + row : wt, in);
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < PER_THREAD; ++e) {
                    const int i = threadIdx.x + e * RET_THREADS, tt = i / DKP, row = i % DKP;
                    const bool in = tt < n && row < dk;
                    const size_t at = in ? (size_t)(ta + tt) * ld + (size_t)head * dk + row : 0;
                    ret_copy(qs + b * RET_TILE * DKP + i, qp + at, in);
                    ret_copy(ks + b * RET_TILE * DKP + i, kp + at, in);
                    if (TM) ret_copy(ws + b * RET_TILE * DKP + i, in ? wt + (size_t)(ta + tt) * ld_w + (size_t)head * dk + row : wt, in);
                }
            }
            if (threadIdx.x < RET_TILE * RET_COLS) {
                const int tt = threadIdx.x / RET_COLS, cc = c0 + threadIdx.x % RET_COLS;
                const bool in = tt < n && cc < dv;
                ret_copy(vs + b * RET_TILE * RET_COLS + threadIdx.x, in ? vp + (size_t)(ta + tt) * ld + (size_t)head * dv + cc : vp, in);
            }
            if (TM && threadIdx.x >= RET_THREADS - RET_TILE) {
                const int tt = threadIdx.x - (RET_THREADS - RET_TILE);
                ret_copy(bs + b * RET_TILE + tt, tt < n ? bonus + (size_t)(ta + tt) * H + head : bonus, tt < n);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto finish = [&](int ta, int b2) {       // the warps' sums of one (token, column), in the warps' order
        if (threadIdx.x < RET_TILE * RET_COLS) {
            const int tt = threadIdx.x / RET_COLS, cc = threadIdx.x % RET_COLS;
            if (ta + tt < t1 && c0 + cc < dv) {
                const float* src = red + (b2 * RET_TILE + tt) * RET_WARPS * RET_COLS + cc;
                float sum = src[0];
#pragma unroll
                for (int w = 1; w < RET_WARPS; ++w) sum += src[w * RET_COLS];
                o[((size_t)(ta + tt) * H + head) * dv + c0 + cc] = sum;
            }
        }
    };
#pragma unroll
    for (int st = 0; st < STAGES - 1; ++st) fetch(t0 + st * RET_TILE, st);
    int b = 0, b2 = 0;
    for (int ta = t0; ta < t1; ta += RET_TILE, b = b + 1 == STAGES ? 0 : b + 1, b2 ^= 1) {
        const int n = min(RET_TILE, t1 - ta);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                      // this tile has landed for everyone; the tile before it is done with
        if (ta > t0) finish(ta - RET_TILE, b2 ^ 1);
        fetch(ta + (STAGES - 1) * RET_TILE, b == 0 ? STAGES - 1 : b - 1);
        const float* qb = qs + b * RET_TILE * DKP + row0;
        const float* kb = ks + b * RET_TILE * DKP + row0;
        const float* wb = ws + b * RET_TILE * DKP + row0;
        const float* vb = vs + b * RET_TILE * RET_COLS + cl;
        const float* bb = bs + b * RET_TILE;
        const bool starts = warp == 0 && lane < RET_COLS;    // TM: the thread whose sum starts with the bonus
        auto element = [&](float& st, float kx, float qx, float wx, float v, float& acc) {
            if (TM) {
                acc = fmaf(st, qx, acc);
                st = fmaf(wx, st, kx * v);
            } else {
                st = fmaf(d, st, kx * v);
                acc = fmaf(st, qx, acc);
            }
        };
        float* rb = red + (b2 * RET_TILE * RET_WARPS + warp) * RET_COLS + cl;
        auto token = [&](int tt) {
            const float v = vb[tt * RET_COLS];
            float acc = TM && starts ? bb[tt] * v : 0.0f;
#pragma unroll
            for (int i = 0; i < RPT; i += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kb + tt * DKP + i);
                const float4 q4 = *reinterpret_cast<const float4*>(qb + tt * DKP + i);
                const float4 w4 = TM ? *reinterpret_cast<const float4*>(wb + tt * DKP + i) : k4;
                element(s[i], k4.x, q4.x, w4.x, v, acc);
                element(s[i + 1], k4.y, q4.y, w4.y, v, acc);
                element(s[i + 2], k4.z, q4.z, w4.z, v, acc);
                element(s[i + 3], k4.w, q4.w, w4.w, v, acc);
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, RET_COLS);       // the lane with the same column and the warp's other rows
            if (lane < RET_COLS) rb[tt * RET_WARPS * RET_COLS] = acc;
        };
        if (n == RET_TILE) {                  // a full tile: the next token's rows are read while this one's are summed
            float4 kk[2][RPT / 4], qq[2][RPT / 4], ww[2][TM ? RPT / 4 : 1];
            float vv[RET_TILE];
#pragma unroll
            for (int tt = 0; tt < RET_TILE; ++tt) vv[tt] = vb[tt * RET_COLS];
#pragma unroll
            for (int i = 0; i < RPT / 4; ++i) {
                kk[0][i] = *reinterpret_cast<const float4*>(kb + 4 * i);
                qq[0][i] = *reinterpret_cast<const float4*>(qb + 4 * i);
                if (TM) ww[0][TM ? i : 0] = *reinterpret_cast<const float4*>(wb + 4 * i);
            }
#pragma unroll
            for (int tt = 0; tt < RET_TILE; ++tt) {
                if (tt + 1 < RET_TILE) {
#pragma unroll
                    for (int i = 0; i < RPT / 4; ++i) {
                        kk[(tt + 1) & 1][i] = *reinterpret_cast<const float4*>(kb + (tt + 1) * DKP + 4 * i);
                        qq[(tt + 1) & 1][i] = *reinterpret_cast<const float4*>(qb + (tt + 1) * DKP + 4 * i);
                        if (TM) ww[(tt + 1) & 1][TM ? i : 0] = *reinterpret_cast<const float4*>(wb + (tt + 1) * DKP + 4 * i);
                    }
                }
                const float v = vv[tt];
                float acc = TM && starts ? bb[tt] * v : 0.0f;
#pragma unroll
                for (int i = 0; i < RPT / 4; ++i) {
                    const float4 k4 = kk[tt & 1][i], q4 = qq[tt & 1][i], w4 = TM ? ww[tt & 1][TM ? i : 0] : k4;
                    element(s[4 * i], k4.x, q4.x, w4.x, v, acc);
                    element(s[4 * i + 1], k4.y, q4.y, w4.y, v, acc);
                    element(s[4 * i + 2], k4.z, q4.z, w4.z, v, acc);
                    element(s[4 * i + 3], k4.w, q4.w, w4.w, v, acc);
                }
                acc += __shfl_xor_sync(0xffffffffu, acc, RET_COLS);
                if (lane < RET_COLS) rb[tt * RET_WARPS * RET_COLS] = acc;
            }
        } else {
#pragma unroll
            for (int tt = 0; tt < RET_TILE; ++tt)
                if (tt < n) token(tt);
        }
    }
    __syncthreads();
    finish(t0 + (t1 - t0 - 1) / RET_TILE * RET_TILE, b2 ^ 1);
    if (col < dv) {
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if (row0 + i < dk) mine[(size_t)(row0 + i) * dv] = s[i];
    }
}

template <int RPT, int STAGES, bool WIDE, bool TM>
int launch_retention(dim3 grid, cudaStream_t st, const float* q, const float* k, const float* v, int ld, const float* decay, const float* wt, int ld_w,
                     const float* bonus, float* state, const int* q_start, const int* slot_ids, float* o, int H, int dk, int dv, int most) {
    const size_t smem = (size_t)(STAGES * RET_TILE * ((TM ? 3 : 2) * RET_CHUNKS * RPT + RET_COLS + (TM ? 1 : 0)) + 2 * RET_TILE * RET_WARPS * RET_COLS) * sizeof(float);
    auto kernel = retention_kernel<RPT, STAGES, WIDE, TM>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    q6k_launch(kernel, grid, RET_THREADS, smem, st, q, k, v, ld, decay, wt, ld_w, bonus, state, q_start, slot_ids, o, H, dk, dv, most);
    return 0;
}

// One block per token: the n mixes of its row with the row before it, out[j, t] = T(x + (x' - x) mu[j]).  prev: FP32 [slots, D], the
// last row of the request's earlier portions (zeros at its start); the block of a portion's first row reads it, then leaves
// the portion's last row there.
template <typename T>
__global__ void __launch_bounds__(256) token_shift_kernel(const T* x, const float* mu, int n, float* prev, const int* req_of_token, const int* q_start,
                                                          const int* slot_ids, T* out, int T_, int D) {
    pdl_enter();
    const int t = blockIdx.x, r = req_of_token[t], first = q_start[r], last = q_start[r + 1] - 1;
    float* mine = prev + (size_t)slot_ids[r] * D;
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
        const float v = to_f32(x[(size_t)t * D + i]);
        float before;
        if (t == first) {
            before = mine[i];
            mine[i] = to_f32(x[(size_t)last * D + i]);
        } else {
            before = to_f32(x[(size_t)(t - 1) * D + i]);
        }
        for (int j = 0; j < n; ++j) out[((size_t)j * T_ + t) * D + i] = from_f32<T>(fmaf(before - v, mu[(size_t)j * D + i], v));
    }
}

// Eight values at a time as FP32 (16 bytes of bfloat16, 32 of FP32), and back.
template <typename T> __device__ __forceinline__ void load8(const T* p, float* v);
template <> __device__ __forceinline__ void load8<float>(const float* p, float* v) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float* v) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[2 * i] = __uint_as_float(w[i] << 16), v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
}
__device__ __forceinline__ void store8(float* p, const float* v) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* v) {
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const unsigned*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// The same for rows of a multiple of eight entries that start on 16 bytes: grid (T, ceil(D / 8 / 128)), eight entries a thread.
template <typename T>
__global__ void __launch_bounds__(128) token_shift8_kernel(const T* x, const float* mu, int n, float* prev, const int* req_of_token, const int* q_start,
                                                           const int* slot_ids, T* out, int T_, int D) {
    pdl_enter();
    const int t = blockIdx.x, i = (blockIdx.y * 128 + threadIdx.x) * 8;
    if (i >= D) return;
    const int r = req_of_token[t], first = q_start[r];
    float v[8], before[8];
    load8<T>(x + (size_t)t * D + i, v);
    if (t == first) {
        float* mine = prev + (size_t)slot_ids[r] * D + i;
        float last[8];
        load8<float>(mine, before);
        load8<T>(x + (size_t)(q_start[r + 1] - 1) * D + i, last);
        store8(mine, last);
    } else {
        load8<T>(x + (size_t)(t - 1) * D + i, before);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) before[e] -= v[e];
    for (int j = 0; j < n; ++j) {
        float m[8], o[8];
        load8<float>(mu + (size_t)j * D + i, m);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = fmaf(before[e], m[e], v[e]);
        store8(out + ((size_t)j * T_ + t) * D + i, o);
    }
}

// A warp per (token, head): w <- exp(-exp(w + w0)) in place, bonus = sum_x u[x] k[x] r[x].
__global__ void __launch_bounds__(128) time_mix_prep_kernel(const float* r, const float* k, int ld, float* w, const float* w0, const float* u, float* bonus,
                                                            int rows, int H, int dk) {
    pdl_enter();
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const int t = row / H, h = row % H;
    const float* rr = r + (size_t)t * ld + h * dk;
    const float* kr = k + (size_t)t * ld + h * dk;
    float* wr = w + ((size_t)t * H + h) * dk;
    float sum = 0.0f;
    for (int x = lane; x < dk; x += 32) {
        sum = fmaf(u[h * dk + x] * kr[x], rr[x], sum);
        wr[x] = expf(-expf(wr[x] + w0[h * dk + x]));
    }
    sum = warp_sum(sum);
    if (lane == 0) bonus[row] = sum;
}

// ---------------------------------------------------------------------------------------- long portions, chunk by chunk
//
// The walk above takes 200 ns a token whatever runs beside it.  Over a chunk of C = 64 tokens, with S the state before it and d the head's
// decay,
//
//   O_i = d^(i+1) S^T q_i + sum_(m <= i) M[i][m] v_m,   M[i][m] = d^(i-m) (q_i . k_m);      S <- d^C S + sum_m d^(C-1-m) k_m v_m^T
//
// so only a sum of matrices goes from chunk to chunk.  ret_outer_kernel makes every chunk's sum of k v^T, all at once; ret_fold_kernel
// walks a request's chunks entry by entry and leaves in each one's place the state it starts from; ret_out_kernel makes every
// chunk's results, [d^(i+1) Q | M] times [S | V] as one product of 64 x 128 outputs whose second factor comes by in slices of 32 rows.
// FP32 throughout; powers of d are made in double precision.  C = 64: 32 would double the bytes of the states (one per chunk and head).
// 2,550 tokens in three portions, 16 heads of 128 x 128: 202 us token by token, 41 + 14 + 95 us so.  What bounds the two products: reads of
// shared memory beside the FP32 pipe, each about half of the time.  Heads of 65 to 128 keys take chunks of 128 on the tensor cores instead (retention_tc.cuh).
constexpr int RC = 64;

__device__ __forceinline__ float ret_power(float d, int n) {
    double p = 1.0, x = (double)d;
    for (; n > 0; n >>= 1, x *= x)
        if (n & 1) p *= x;
    return (float)p;
}

}  // namespace
#include "retention_tc.cuh"
namespace {

// grid (H, chunks, ceil(dk / 128) ceil(dv / 128)) (blocks of chunks that there are not come last), 256 threads, 64 KB of dynamic shared memory; KV: FP32 [chunks, H, dk, dv].
__global__ void __launch_bounds__(256) ret_outer_kernel(const float* kp, const float* vp, int ld, const float* decay, const int* q_start, int R, int beyond, float* KV, int H, int dk,
                                                        int dv) {
    pdl_enter();
    extern __shared__ __align__(16) float sm[];
    float *ks = sm, *vs = sm + RC * 128;                    // [64][128] each, k times its token's power of d
    const int head = blockIdx.x, tid = threadIdx.x, cols = (dv + 127) / 128, row0 = blockIdx.z / cols * 128, col0 = blockIdx.z % cols * 128;
    int first = 0, n = 0;
    chunk_of<RC>(q_start, R, beyond, blockIdx.y, first, n);
    if (n == 0) return;
    const float d = decay[head];
    const int at = (tid & 31) * 4;
    float4 k4[8], v4[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int t = (tid >> 5) + 8 * e;
        const size_t row = (size_t)(first + t) * ld;
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        k4[e] = t < n && row0 + at < dk ? *reinterpret_cast<const float4*>(kp + row + (size_t)head * dk + row0 + at) : zero;
        v4[e] = t < n && col0 + at < dv ? *reinterpret_cast<const float4*>(vp + row + (size_t)head * dv + col0 + at) : zero;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int t = (tid >> 5) + 8 * e;
        const float p = ret_power(d, t < n ? n - 1 - t : 0);
        *reinterpret_cast<float4*>(ks + t * 128 + at) = make_float4(k4[e].x * p, k4[e].y * p, k4[e].z * p, k4[e].w * p);
        *reinterpret_cast<float4*>(vs + t * 128 + at) = v4[e];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, row = (warp >> 1) * 32 + (lane >> 3) * 4, col = (warp & 1) * 64 + (lane & 7) * 4;
    unsigned long long acc[8][4] = {};                      // rows row .. row + 3 and row + 16 .. row + 19; columns col .. and col + 32 ..
#pragma unroll 2
    for (int m = 0; m < n; ++m) {
        const float4 a0 = *reinterpret_cast<const float4*>(ks + m * 128 + row), a1 = *reinterpret_cast<const float4*>(ks + m * 128 + row + 16);
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(vs + m * 128 + col), b1 = *reinterpret_cast<const ulonglong2*>(vs + m * 128 + col + 32);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned long long aa = both(a[i]);
            fma_pair(acc[i][0], aa, b0.x), fma_pair(acc[i][1], aa, b0.y), fma_pair(acc[i][2], aa, b1.x), fma_pair(acc[i][3], aa, b1.y);
        }
    }
    float* out = KV + ((size_t)blockIdx.y * H + head) * dk * dv;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rr = row0 + row + (i & 3) + (i >> 2) * 16;
        if (rr >= dk) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (col0 + col + 32 * j < dv) *reinterpret_cast<ulonglong2*>(out + (size_t)rr * dv + col0 + col + 32 * j) = make_ulonglong2(acc[i][2 * j], acc[i][2 * j + 1]);
    }
}

// The state every chunk starts from, in its sum's place, and the state a portion leaves.  grid (long requests * blocks), blocks = ceil(H dk dv / 1024).
template <int CT>
__global__ void __launch_bounds__(256) ret_fold_kernel(float* KV, const float* decay, float* state, const int* q_start, int R, int beyond, const int* slot_ids, int H, int cells) {
    pdl_enter();
    const size_t all = (size_t)H * cells;                   // cells = dk dv, a multiple of 4
    const unsigned blocks = (unsigned)((all + 1023) / 1024);
    int chunk0;
    const int r = long_request<CT>(q_start, R, beyond, blockIdx.x / blocks, chunk0);
    if (r < 0) return;
    const int n = q_start[r + 1] - q_start[r], count = (n + CT - 1) / CT;
    const size_t i = ((size_t)(blockIdx.x % blocks) * 256 + threadIdx.x) * 4;
    if (i >= all) return;
    const float d = decay[i / cells], full = ret_power(d, CT), rest = ret_power(d, n - (count - 1) * CT);
    float4* mine = reinterpret_cast<float4*>(state + (size_t)slot_ids[r] * all + i);
    float4 S = *mine;
    float* at = KV + (size_t)chunk0 * all + i;
    for (int c0 = 0; c0 < count; c0 += 4) {
        float4 built[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (c0 + e < count) built[e] = *reinterpret_cast<const float4*>(at + (size_t)(c0 + e) * all);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (c0 + e < count) {
                *reinterpret_cast<float4*>(at + (size_t)(c0 + e) * all) = S;
                const float p = c0 + e + 1 == count ? rest : full;
                S = make_float4(fmaf(p, S.x, built[e].x), fmaf(p, S.y, built[e].y), fmaf(p, S.z, built[e].z), fmaf(p, S.w, built[e].w));
            }
    }
    *mine = S;
}

constexpr int RO_SLICE = 32, RO_STAGES = 3, RO_MLD = RC + 4;
__host__ __device__ constexpr int ret_out_slices(int dkp) { return RC * (dkp + 4) > RO_STAGES * RO_SLICE * 128 ? RC * (dkp + 4) : RO_STAGES * RO_SLICE * 128; }
__host__ __device__ constexpr int ret_out_floats(int dkp) { return RC * (dkp + 4) + RC * RO_MLD + ret_out_slices(dkp) + RC + 4; }

// grid (H, chunks, ceil(dv / 128)), 256 threads.  dkp: dk rounded up to a multiple of 32.
__global__ void __launch_bounds__(256, 2) ret_out_kernel(const float* qp, const float* kp, const float* vp, int ld, const float* decay, const float* KV, const int* q_start,
                                                         int R, int beyond, float* o, int H, int dk, int dv, int dkp) {
    pdl_enter();
    extern __shared__ __align__(16) float sm[];
    const int ldq = dkp + 4;
    float* Q = sm;                                          // [64][ldq]
    float* M = Q + RC * ldq;                                // [64][68]
    float* B = M + RC * RO_MLD;                             // K [64][ldq], then the slices [3][32][128] of S and V
    float* pw = B + ret_out_slices(dkp);                    // [65]
    const int head = blockIdx.x, col0 = blockIdx.z * 128, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int first = 0, n = 0;
    chunk_of<RC>(q_start, R, beyond, blockIdx.y, first, n);
    if (n == 0) return;
    if (tid <= RC) pw[tid] = ret_power(decay[head], tid);
    for (int t = warp; t < RC; t += 8)
        for (int d = lane * 4; d < dkp; d += 128) {
            const bool in = t < n && d < dk;
            const size_t at = (size_t)(first + (in ? t : 0)) * ld + (size_t)head * dk + (in ? d : 0);
            copy16((uint32_t)__cvta_generic_to_shared(Q + t * ldq + d), qp + at, in);
            copy16((uint32_t)__cvta_generic_to_shared(B + t * ldq + d), kp + at, in);
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int row = (warp >> 2) * 32 + (lane >> 3);         // rows row + 4 i
    {   // M: columns mc and mc + 8
        const int mc = (warp & 3) * 16 + (lane & 7);
        unsigned long long acc[8][2] = {};
#pragma unroll 2
        for (int d = 0; d < dkp; d += 4) {
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(B + mc * ldq + d), b1 = *reinterpret_cast<const ulonglong2*>(B + (mc + 8) * ldq + d);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(Q + (row + 4 * i) * ldq + d);
                fma_pair(acc[i][0], a.x, b0.x), fma_pair(acc[i][0], a.y, b0.y);
                fma_pair(acc[i][1], a.x, b1.x), fma_pair(acc[i][1], a.y, b1.y);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int t = row + 4 * i, m = mc + 8 * j;
                M[t * RO_MLD + m] = m <= t ? pw[t - m] * (low(acc[i][j]) + high(acc[i][j])) : 0.0f;
            }
    }
    __syncthreads();                                        // K is done with, M whole
    const int state_slices = dkp / RO_SLICE, slices = state_slices + (n + RO_SLICE - 1) / RO_SLICE;
    const float* S = KV + ((size_t)blockIdx.y * H + head) * dk * dv;
    auto fetch = [&](int s) {
        if (s < slices) {
            const int c = col0 + lane * 4;
#pragma unroll
            for (int e = 0; e < RO_SLICE / 8; ++e) {
                const int rr = warp + 8 * e, x = (s < state_slices ? s : s - state_slices) * RO_SLICE + rr;
                const bool in = c < dv && x < (s < state_slices ? dk : n);
                const float* from = s < state_slices ? S + (size_t)x * dv + c : vp + (size_t)(first + x) * ld + (size_t)head * dv + c;
                copy16((uint32_t)__cvta_generic_to_shared(B + ((s % RO_STAGES) * RO_SLICE + rr) * 128 + lane * 4), in ? from : vp, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    fetch(1);
    for (int t = warp; t < RC; t += 8)                      // d^(i+1) Q, seen by all at the first slice's barrier
        for (int d = lane; d < dkp; d += 32) Q[t * ldq + d] *= pw[t + 1];
    const int col = (warp & 3) * 32 + (lane & 7) * 4;
    unsigned long long acc[8][2] = {};
    for (int s = 0; s < slices; ++s) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                    // the slice has landed for everyone; the one before it is done with
        fetch(s + 2);
        const float* b = B + (s % RO_STAGES) * RO_SLICE * 128 + col;
        if (s < state_slices) {
            const float* a = Q + row * ldq + s * RO_SLICE;
#pragma unroll 2
            for (int d = 0; d < RO_SLICE; d += 4) {
                float4 x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(a + 4 * i * ldq + d);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(b + (d + e) * 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const unsigned long long aa = both(e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w);
                        fma_pair(acc[i][0], aa, w.x), fma_pair(acc[i][1], aa, w.y);
                    }
                }
            }
        } else {
            const int m0 = (s - state_slices) * RO_SLICE;
            const float* a = M + row * RO_MLD + m0;
#pragma unroll 1
            for (int d = 0; d < RO_SLICE; d += 4) {
                float4 x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(a + 4 * i * RO_MLD + d);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(b + (d + e) * 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (m0 + d + e <= row + 4 * i) {    // no value of a later token, were it infinite, reaches an earlier one
                            const unsigned long long aa = both(e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w);
                            fma_pair(acc[i][0], aa, w.x), fma_pair(acc[i][1], aa, w.y);
                        }
                }
            }
        }
    }
    if (col0 + col < dv) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = row + 4 * i;
            if (t < n) *reinterpret_cast<ulonglong2*>(o + ((size_t)(first + t) * H + head) * dv + col0 + col) = make_ulonglong2(acc[i][0], acc[i][1]);
        }
    }
}

}  // namespace

Q6K_API int q6k_retention_max_dim() { return RET_MAX_DK; }

// Rotates q and k of every head in place and scales k.
Q6K_API int q6k_retention_prep(float* p, int ld, int T_, int H, int dk, int q_col, int k_col,
                               const float* inv_freq, int rd, int neighbours, float k_scale, const int* positions, int act_cols,
                               cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && H > 0 && dk > 0 && 2 * H <= 65535, "retention_prep: bad sizes T=%d H=%d dk=%d", T_, H, dk);
    Q6K_REQUIRE(rd >= 0 && rd % 2 == 0 && rd <= dk && (rd == 0 || inv_freq), "retention_prep: %d turning dimensions of %d", rd, dk);
    Q6K_REQUIRE(act_cols >= 0 && act_cols <= ld, "retention_prep: %d activated columns of %d", act_cols, ld);
    if (rd == 0 && k_scale == 1.0f && act_cols == 0) return 0;
    if (rd > 0 && rd % 8 == 0 && !neighbours && act_cols == 0 && dk % 4 == 0 && ld % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && ((uintptr_t)p & 15) == 0) {
        q6k_launch(retention_turn4_kernel, dim3(T_), 256, (size_t)rd * sizeof(float), st, p, ld, H, dk, q_col, k_col, inv_freq, rd, k_scale, positions);
        return q6k_check_launch("retention_prep");
    }
    q6k_launch(retention_prep_kernel, dim3(T_), 256, (size_t)rd * sizeof(float), st, p, ld, H, dk, q_col, k_col,
               inv_freq, rd, neighbours, k_scale, positions, act_cols);
    return q6k_check_launch("retention_prep");
}

// most: requests of up to so many tokens (the others are left alone).
Q6K_API int q6k_retention(const float* p, int ld, int q_col, int k_col, int v_col, const float* decay, float* state, const int* q_start,
                          const int* slot_ids, int R, float* o, int H, int dk, int dv, int most, cudaStream_t st) {
    if (R == 0) return 0;
    Q6K_REQUIRE(R > 0 && H > 0 && dk > 0 && dv > 0 && dk <= RET_MAX_DK, "retention: bad sizes R=%d H=%d dk=%d (at most %d) dv=%d", R, H, dk, RET_MAX_DK, dv);
    const int zb = (dv + RET_COLS - 1) / RET_COLS;
    Q6K_REQUIRE(H <= 65535 && zb <= 65535, "retention: grid too large");
    const dim3 grid(R, H, zb);
    auto on16 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
    const bool wide = dk % 4 == 0 && ld % 4 == 0 && on16(p + q_col) && on16(p + k_col);
#define RET_LAUNCH(RPT)                                                                                                               \
    do {                                                                                                                              \
        if (wide) launch_retention<RPT, RET_STAGES, true, false>(grid, st, p + q_col, p + k_col, p + v_col, ld, decay, nullptr, 0, nullptr, state, q_start, slot_ids, o, H, dk, dv, most); \
        else launch_retention<RPT, RET_STAGES, false, false>(grid, st, p + q_col, p + k_col, p + v_col, ld, decay, nullptr, 0, nullptr, state, q_start, slot_ids, o, H, dk, dv, most);     \
    } while (0)
    if (dk <= 64) RET_LAUNCH(4);
    else if (dk <= 128) RET_LAUNCH(8);
    else RET_LAUNCH(16);
#undef RET_LAUNCH
    return q6k_check_launch("retention");
}

// Floats of scratch for the same walk chunk by chunk.
// Heads of more than 64 and up to 128 keys go on the tensor cores, in chunks of 128: narrower ones would fill half of their tiles (a head of 64 x 64,
// 1,024 tokens of 16: 47 us in FP32, 37 us for the tiles of twice its size), wider ones do not fit.
static bool retention_tc(int dk) { return dk > 64 && dk <= 128; }
Q6K_API long long q6k_retention_chunk_floats(int T_, int R, int H, int dk, int dv, int beyond) {
    return (long long)(retention_tc(dk) ? most_chunks<RT>(T_, R, beyond) : most_chunks<RC>(T_, R, beyond)) * H * dk * dv;
}
Q6K_API int q6k_retention_tc_status() {
    int v = -1;
    if (cudaMemcpyFromSymbol(&v, g_retention_tc_status, sizeof v) != cudaSuccess) return -1;
    return v;
}

// Requests of more than `beyond` tokens in chunks of 64 (T_: rows of the step): rows and heads of q, k and v that start on 16 bytes,
// dk and dv multiples of 4.
Q6K_API int q6k_retention_chunked(const float* p, int ld, int q_col, int k_col, int v_col, const float* decay, float* chunks, float* state, const int* q_start,
                                  const int* slot_ids, int T_, int R, float* o, int H, int dk, int dv, int beyond, cudaStream_t st) {
    if (R == 0 || T_ == 0) return 0;
    Q6K_REQUIRE(R > 0 && beyond >= 0 && H > 0 && dk > 0 && dv > 0 && dk <= RET_MAX_DK, "retention: bad sizes R=%d H=%d dk=%d (at most %d) dv=%d", R, H, dk, RET_MAX_DK, dv);
    Q6K_REQUIRE(dk % 4 == 0 && dv % 4 == 0 && ld % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && v_col % 4 == 0 && (((uintptr_t)p | (uintptr_t)chunks | (uintptr_t)state) & 15) == 0,
                "retention: chunks take rows and heads that start on 16 bytes");
    const int n_long = most_long(T_, R, beyond), n_chunks = most_chunks<RC>(T_, R, beyond), cols = (dv + 127) / 128, dkp = (dk + 31) / 32 * 32;
    if (n_long == 0) return 0;
    const unsigned folds = (unsigned)(n_long * (((size_t)H * dk * dv + 1023) / 1024));
    if (retention_tc(dk)) {
        const long long tasks = (long long)most_chunks<RT>(T_, R, beyond) * H * cols;
        Q6K_REQUIRE(tasks < 0x7fffffff - 1024, "retention: %lld tasks", tasks);
        const unsigned grid = (unsigned)(tasks < 148 ? tasks : 148);
        if (cudaFuncSetAttribute(ret_outer_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RT_SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(ret_out_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RT_SMEM) != cudaSuccess)
            return q6k_check_launch("retention: shared memory attribute");
        q6k_launch(ret_outer_tc_kernel, grid, RT_THREADS, RT_SMEM, st, p + k_col, p + v_col, ld, decay, q_start, R, beyond, chunks, H, dk, dv, (int)tasks);
        if (int rc = q6k_check_launch("ret_outer_tc")) return rc;
        q6k_launch(ret_fold_kernel<RT>, dim3(folds), 256, 0, st, chunks, decay, state, q_start, R, beyond, slot_ids, H, dk * dv);
        if (int rc = q6k_check_launch("ret_fold")) return rc;
        q6k_launch(ret_out_tc_kernel, grid, RT_THREADS, RT_SMEM, st, p + q_col, p + k_col, p + v_col, ld, decay, chunks, q_start, R, beyond, o, H, dk, dv, (int)tasks);
        return q6k_check_launch("ret_out_tc");
    }
    const size_t smem1 = (size_t)2 * RC * 128 * sizeof(float), smem2 = (size_t)ret_out_floats(dkp) * sizeof(float);
    if (cudaFuncSetAttribute(ret_outer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1) != cudaSuccess ||
        cudaFuncSetAttribute(ret_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2) != cudaSuccess)
        return q6k_check_launch("retention: shared memory attribute");
    q6k_launch(ret_outer_kernel, dim3(H, n_chunks, (dk + 127) / 128 * cols), 256, smem1, st, p + k_col, p + v_col, ld, decay, q_start, R, beyond, chunks, H, dk, dv);
    if (int rc = q6k_check_launch("ret_outer")) return rc;
    q6k_launch(ret_fold_kernel<RC>, dim3(folds), 256, 0, st, chunks, decay, state, q_start, R, beyond, slot_ids, H, dk * dv);
    if (int rc = q6k_check_launch("ret_fold")) return rc;
    q6k_launch(ret_out_kernel, dim3(H, n_chunks, cols), 256, smem2, st, p + q_col, p + k_col, p + v_col, ld, decay, chunks, q_start, R, beyond, o, H, dk, dv, dkp);
    return q6k_check_launch("ret_out");
}

// x: [T, D] in the storage type; mu: FP32 [n, D]; prev: FP32 [slots, D]; out: [n, T, D] in the storage type.
Q6K_API int q6k_token_shift(const void* x, const float* mu, int n, float* prev, const int* req_of_token, const int* q_start, const int* slot_ids, void* out,
                            int T_, int D, int dtype, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && D > 0 && n > 0, "token_shift: bad sizes T=%d D=%d n=%d", T_, D, n);
    auto on16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (D % 8 == 0 && on16(x) && on16(mu) && on16(prev) && on16(out)) {
        Q6K_DISPATCH(dtype, q6k_launch(token_shift8_kernel<T>, dim3(T_, (D / 8 + 127) / 128), 128, 0, st, (const T*)x, mu, n, prev, req_of_token, q_start, slot_ids,
                                       (T*)out, T_, D););
        return q6k_check_launch("token_shift");
    }
    Q6K_DISPATCH(dtype, q6k_launch(token_shift_kernel<T>, dim3(T_), 256, 0, st, (const T*)x, mu, n, prev, req_of_token, q_start, slot_ids, (T*)out, T_, D););
    return q6k_check_launch("token_shift");
}

// r, k: FP32, a token's heads side by side, rows ld apart; w: FP32 [T, H dk] (in: the decay projection, out: the decays); w0, u: FP32 [H dk];
// bonus: FP32 [T, H].
Q6K_API int q6k_time_mix_prep(const float* r, const float* k, int ld, float* w, const float* w0, const float* u, float* bonus, int T_, int H, int dk, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && H > 0 && dk > 0 && (long long)T_ * H <= 0x7fffffffLL, "time_mix_prep: bad sizes T=%d H=%d dk=%d", T_, H, dk);
    q6k_launch(time_mix_prep_kernel, dim3((unsigned)(((long long)T_ * H + 3) / 4)), 128, 0, st, r, k, ld, w, w0, u, bonus, T_ * H, H, dk);
    return q6k_check_launch("time_mix_prep");
}

// The second recurrence: r, k, v FP32, rows ld apart; w: FP32 [T, H dk] decays; bonus: FP32 [T, H]; state: FP32 [slots, H, dk, dv]; o: FP32 [T, H dv].
Q6K_API int q6k_time_mix(const float* r, const float* k, const float* v, int ld, const float* w, const float* bonus, float* state, const int* q_start,
                         const int* slot_ids, int R, float* o, int H, int dk, int dv, cudaStream_t st) {
    if (R == 0) return 0;
    Q6K_REQUIRE(R > 0 && H > 0 && dk > 0 && dv > 0 && dk <= RET_MAX_DK, "time_mix: bad sizes R=%d H=%d dk=%d (at most %d) dv=%d", R, H, dk, RET_MAX_DK, dv);
    const int zb = (dv + RET_COLS - 1) / RET_COLS;
    Q6K_REQUIRE(H <= 65535 && zb <= 65535, "time_mix: grid too large");
    const dim3 grid(R, H, zb);
    auto on16 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
    const bool wide = dk % 4 == 0 && ld % 4 == 0 && on16(r) && on16(k) && on16(w);
#define RET_LAUNCH(RPT)                                                                                                               \
    do {                                                                                                                              \
        if (wide) launch_retention<RPT, RET_STAGES, true, true>(grid, st, r, k, v, ld, nullptr, w, H * dk, bonus, state, q_start, slot_ids, o, H, dk, dv, 0x7fffffff); \
        else launch_retention<RPT, RET_STAGES, false, true>(grid, st, r, k, v, ld, nullptr, w, H * dk, bonus, state, q_start, slot_ids, o, H, dk, dv, 0x7fffffff);     \
    } while (0)
    if (dk <= 64) RET_LAUNCH(4);
    else if (dk <= 128) RET_LAUNCH(8);
    else RET_LAUNCH(16);
#undef RET_LAUNCH
    return q6k_check_launch("time_mix");
}
