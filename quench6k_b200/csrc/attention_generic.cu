// Attention over the paged cache for any mix of rows (prompt portions beside decode tokens), any
// head size that is a multiple of 16 up to 256, any number of heads and groups, in FP32 or
// bfloat16 storage with FP32 arithmetic.  This is the kernel of the true 32-bit path and the
// fallback of the bfloat16 path.
//
// Formulas: crates/cuda/kernels/flint.cu:211-529 (query head h reads KV head h / G; score
// q.k/sqrt(hd); key j visible to position p iff j <= p and, with a window W, j > p - W; online
// softmax; probabilities rounded to the storage type before they are summed, :409-415) and
// :531-561 (a sink adds exp(sink_h - m) to the denominator only).
//
// A block takes one (token, KV head); its warps take the G query heads in turn.  Keys are walked
// in tiles of 32 aligned to multiples of 32 of the key index, so the order of the sums for a
// given (position, head) never depends on how the tokens were cut into steps or batched.
#include "common.cuh"

namespace {

constexpr int MAX_HD = 256, DPL = MAX_HD / 32;   // head dims per lane

// One query head h of row t, by a warp; qw: hd floats of shared memory of its own.
template <typename T>
__device__ __forceinline__ void attention_row(const T* q, const T* k_pages, const T* v_pages, const int* bt, int page_size, size_t head_base, int pos, int lo,
                                              const float* sinks, float scale, T* out, int t, int h, int Hq, int hd, float* qw) {
    const int lane = threadIdx.x & 31;
    for (int d = lane; d < hd; d += 32) qw[d] = to_f32(q[((size_t)t * Hq + h) * hd + d]);
    __syncwarp();
    float m = -INFINITY, l = 0.0f, o[DPL];
#pragma unroll
    for (int i = 0; i < DPL; ++i) o[i] = 0.0f;
    for (int j0 = lo & ~31; j0 <= pos; j0 += 32) {
        const int j = j0 + lane;
        const bool ok = j >= lo && j <= pos;
        float s = -INFINITY;
        size_t row = 0;
        if (ok) {
            const int page = bt[j / page_size];
            row = ((head_base + page) * page_size + j % page_size) * hd;
            const T* kr = k_pages + row;
            float acc = 0.0f;
            for (int d = 0; d < hd; ++d) acc = fmaf(qw[d], to_f32(kr[d]), acc);
            s = acc * scale;
        }
        const float mt = warp_max(s);
        const float mn = fmaxf(m, mt);          // finite: the tile holds at least one visible key
        const float corr = m == -INFINITY ? 0.0f : expf(m - mn);
        float p = ok ? round_to<T>(expf(s - mn)) : 0.0f;
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < DPL; ++i) o[i] *= corr;
        const int nk = min(32, pos - j0 + 1);
        for (int jj = 0; jj < nk; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const unsigned long long rj = __shfl_sync(0xffffffffu, (unsigned long long)row, jj);
            if (pj == 0.0f) continue;           // uniform across the warp
            const T* vr = v_pages + rj;
#pragma unroll
            for (int i = 0; i < DPL; ++i) {
                const int d = lane + 32 * i;
                if (d < hd) o[i] = fmaf(pj, to_f32(vr[d]), o[i]);
            }
        }
        m = mn;
    }
    float den = l;
    float osc = 1.0f;
    if (sinks) {
        const float sk = sinks[h];
        const float M = fmaxf(m, sk);
        osc = expf(m - M);
        den = l * osc + expf(sk - M);
    }
    const float inv = osc / den;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
        const int d = lane + 32 * i;
        if (d < hd) out[((size_t)t * Hq + h) * hd + d] = from_f32<T>(o[i] * inv);
    }
    __syncwarp();
}

// Whether fewer than `least` rows of the step, one after the other, belong to row t's request (rows [ta, tb) around t are known to).
__device__ __forceinline__ bool few_rows(const int* req_of_token, int ta, int tb, int T_, int least) {
    const int req = req_of_token[ta];
    while (tb - ta < least && ta > 0 && req_of_token[ta - 1] == req) --ta;
    while (tb - ta < least && tb < T_ && req_of_token[tb] == req) ++tb;
    return tb - ta < least;
}

// least > 0: requests of at least so many rows belong to the launch of row tiles.
template <typename T>
__global__ void __launch_bounds__(128) attention_generic_kernel(const T* q, const T* k_pages, const T* v_pages,
                                                                const int* block_table, int max_blocks, int page_size,
                                                                int num_pages, const int* req_of_token, const int* positions, int window,
                                                                const float* sinks, float scale, T* out, int T_, int Hq, int Hkv,
                                                                int hd, int least) {
    pdl_enter();
    extern __shared__ float qs[];             // [warps][hd]
    const int t = blockIdx.x, kh = blockIdx.y, G = Hq / Hkv;
    if (least > 0 && !few_rows(req_of_token, t, t + 1, T_, least)) return;
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int pos = positions[t];
    const int* bt = block_table + (size_t)req_of_token[t] * max_blocks;
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    for (int g = warp; g < G; g += nwarps)       // pools are [Hkv, num_pages, page_size, hd]
        attention_row(q, k_pages, v_pages, bt, page_size, (size_t)kh * num_pages, pos, lo, sinks, scale, out, t, kh * G + g, Hq, hd, qs + warp * hd);
}

// The same for steps that bring several tokens per request: the same sums in the same order (a row's scores are summed over ascending
// dimensions, its keys come in tiles of 32 whose weights a warp adds with the same butterfly, values are added in ascending order
// of the keys), so a row's result is the same bit for bit whichever of the two kernels runs it.
//
// The kernel above reads a key row per lane and a value row per (head, key) from global memory: 500 us for 509 tokens of 8 heads
// over 509 keys, waiting for loads.  Here a block takes up to 32 rows (the query heads of a KV head for consecutive tokens of the step)
// and brings each key tile into shared memory once; 8 threads share a row: each makes the scores of four keys and owns every
// eighth group of four dimensions of the result, so that a 16-byte read of keys or values serves four rows and a warp's reads fall into
// different banks: 92 us.  Tokens of several requests in one block are taken request by request, so where a block could meet many,
// requests of fewer than `least` tokens are left to the kernel above.  8 heads on 8 KV heads, 509 tokens beside 32 requests of 4,000 keys: a
// block walked the contexts of 32 tokens one after the other, 15,700 us; all rows in the kernel above 4,470; so 2,830.
constexpr int GT_ROWS = 32, GT_KEYS = 32, GT_THREADS = 256;

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}

template <typename T, int NI>          // NI: groups of 32 dimensions (hd <= 32 NI)
__global__ void __launch_bounds__(GT_THREADS) attention_tiled_kernel(const T* q, const T* k_pages, const T* v_pages, const int* block_table, int max_blocks,
                                                                     int page_size, int num_pages, const int* req_of_token, const int* positions,
                                                                     int window, const float* sinks, float scale, T* out, int T_, int Hq, int Hkv, int hd,
                                                                     int tokens, int heads, int least) {
    pdl_enter();
    extern __shared__ __align__(16) float gt_smem[];
    const int ld = hd + 4;
    float* qs = gt_smem;                              // [GT_ROWS][ld]
    float* ks = qs + GT_ROWS * ld;                    // [GT_KEYS][ld]
    float* vs = ks + GT_KEYS * ld;                    // [GT_KEYS][ld]
    float* ss = vs + GT_KEYS * ld;                    // [GT_ROWS][GT_KEYS + 4]: scores, then weights
    float* corr_s = ss + GT_ROWS * (GT_KEYS + 4);     // [GT_ROWS]: what a row's result is multiplied by before the tile, at the end by
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = Hq / Hkv;
    const int kh = blockIdx.y, g0 = blockIdx.z * heads, here = min(heads, G - g0);
    const size_t head_base = (size_t)kh * num_pages;
    const int t0 = blockIdx.x * tokens, t1 = min(T_, t0 + tokens);
    const int row = tid >> 3, c = tid & 7;            // this thread's row and place in it; row = token * heads + head
    for (int ta = t0; ta < t1;) {
        const int req = req_of_token[ta];
        int tb = ta + 1, pos_min = positions[ta], pos_max = pos_min;        // the rows' positions may come in any order
        for (; tb < t1 && req_of_token[tb] == req; ++tb) pos_min = min(pos_min, positions[tb]), pos_max = max(pos_max, positions[tb]);
        if (least > 0 && few_rows(req_of_token, ta, tb, T_, least)) {
            ta = tb;
            continue;
        }
        const int* bt = block_table + (size_t)req * max_blocks;
        const int rows = (tb - ta) * heads, k_end = pos_max + 1;
        const int lo_first = window > 0 ? max(0, pos_min - window + 1) : 0;
        __syncthreads();                              // the rows before are done with
        for (int i = tid; i < rows * (hd / 4); i += GT_THREADS) {
            const int r = i / (hd / 4), d = (i % (hd / 4)) * 4, g = g0 + r % heads;
            *reinterpret_cast<float4*>(qs + r * ld + d) = load4(q + ((size_t)(ta + r / heads) * Hq + kh * G + (g < G ? g : 0)) * hd + d);
        }
        // the softmax state of rows 4 warp .. 4 warp + 3, the same in every lane
        float m[4], l[4];
        int pos4[4], lo4[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int r = warp * 4 + x;
            m[x] = -INFINITY, l[x] = 0.0f;
            pos4[x] = r < rows ? positions[ta + r / heads] : -1;
            lo4[x] = window > 0 ? max(0, pos4[x] - window + 1) : 0;
        }
        float4 o[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) o[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int j0 = lo_first & ~(GT_KEYS - 1); j0 < k_end; j0 += GT_KEYS) {
            __syncthreads();                          // the tile before is done with
            for (int i = tid; i < GT_KEYS * (hd / 4); i += GT_THREADS) {
                const int kk = i / (hd / 4), d = (i % (hd / 4)) * 4, j = j0 + kk;
                float4 kv = make_float4(0.0f, 0.0f, 0.0f, 0.0f), vv = kv;
                const int page = j >= lo_first && j < k_end ? bt[j / page_size] : -1;
                if (page >= 0) {                      // a page between the rows' windows may be gone
                    const size_t at = ((head_base + page) * page_size + j % page_size) * hd + d;
                    kv = load4(k_pages + at);
                    vv = load4(v_pages + at);
                }
                *reinterpret_cast<float4*>(ks + kk * ld + d) = kv;
                *reinterpret_cast<float4*>(vs + kk * ld + d) = vv;
            }
            __syncthreads();
            if (row < rows) {
                float s[4] = {};
                const float* qr = qs + row * ld;
                const float* kr = ks + c * ld;
#pragma unroll 4
                for (int d = 0; d < hd; d += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(qr + d);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const float4 b = *reinterpret_cast<const float4*>(kr + x * 8 * ld + d);
                        s[x] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s[x]))));
                    }
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) ss[row * (GT_KEYS + 4) + c + 8 * x] = s[x];
            }
            __syncwarp();                             // a row's eight threads, its state and its weights belong to one warp
            // softmax: a lane per key, the warp's four rows in turn
            const int j = j0 + lane;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int r = warp * 4 + x;
                if (j0 > pos4[x] || j0 + GT_KEYS <= lo4[x]) {              // no key of this tile for the row: it does not see the tile at all
                    if (lane == 0) corr_s[r] = -1.0f;
                    continue;
                }
                const bool ok = j >= lo4[x] && j <= pos4[x];
                const float s = ok ? ss[r * (GT_KEYS + 4) + lane] * scale : -INFINITY;
                const float mn = fmaxf(m[x], warp_max(s));
                const float corr = m[x] == -INFINITY ? 0.0f : expf(m[x] - mn);
                const float p = ok ? round_to<T>(expf(s - mn)) : 0.0f;
                l[x] = l[x] * corr + warp_sum(p);
                m[x] = mn;
                ss[r * (GT_KEYS + 4) + lane] = p;
                if (lane == 0) corr_s[r] = corr;
            }
            __syncwarp();
            const float corr = row < rows ? corr_s[row] : -1.0f;
            if (corr != -1.0f) {
#pragma unroll
                for (int i = 0; i < NI; ++i) o[i].x *= corr, o[i].y *= corr, o[i].z *= corr, o[i].w *= corr;
                const float* pr = ss + row * (GT_KEYS + 4);
#pragma unroll 4
                for (int kk = 0; kk < GT_KEYS; ++kk) {
                    const float p = pr[kk];
                    if (p != 0.0f) {
                        const float* vr = vs + kk * ld + c * 4;
#pragma unroll
                        for (int i = 0; i < NI; ++i)
                            if (NI * 32 == hd || c * 4 + 32 * i < hd) {
                                const float4 b = *reinterpret_cast<const float4*>(vr + 32 * i);
                                o[i].x = fmaf(p, b.x, o[i].x), o[i].y = fmaf(p, b.y, o[i].y), o[i].z = fmaf(p, b.z, o[i].z), o[i].w = fmaf(p, b.w, o[i].w);
                            }
                    }
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int r = warp * 4 + x;
            if (lane == 0 && r < rows) {
                float den = l[x], osc = 1.0f;
                if (sinks && g0 + r % heads < G) {
                    const float sk = sinks[kh * G + g0 + r % heads], M = fmaxf(m[x], sk);
                    osc = expf(m[x] - M);
                    den = l[x] * osc + expf(sk - M);
                }
                corr_s[r] = osc / den;
            }
        }
        __syncwarp();
        if (row < rows && row % heads < here) {
            const float inv = corr_s[row];
            T* dst = out + ((size_t)(ta + row / heads) * Hq + kh * G + g0 + row % heads) * hd + c * 4;
#pragma unroll
            for (int i = 0; i < NI; ++i)
                if (NI * 32 == hd || c * 4 + 32 * i < hd) {
                    dst[32 * i] = from_f32<T>(o[i].x * inv), dst[32 * i + 1] = from_f32<T>(o[i].y * inv);
                    dst[32 * i + 2] = from_f32<T>(o[i].z * inv), dst[32 * i + 3] = from_f32<T>(o[i].w * inv);
                }
        }
        ta = tb;
    }
}

}  // namespace

// q: [T, Hq, hd]; pages: [Hkv, num_pages, page_size, hd]; block_table: [R, max_blocks];
// window 0: every earlier key is visible; sinks: FP32 [Hq] or null; out: [T, Hq*hd].  requests: how many the step's rows belong to
// (0: not said); shortest: the rows of the one with the fewest (0: not said).
Q6K_API int q6k_attention_generic(const void* q, const void* k_pages, const void* v_pages, int num_pages, const int* block_table,
                                  int max_blocks, int page_size, const int* req_of_token, const int* positions, int window,
                                  const float* sinks, float scale, void* out, int T_, int Hq, int Hkv, int hd, int dtype, int requests, int shortest,
                                  cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0, "attention: bad head counts Hq=%d Hkv=%d", Hq, Hkv);
    Q6K_REQUIRE(hd > 0 && hd % 16 == 0 && hd <= MAX_HD, "attention: head_dim %d is not a multiple of 16 in 16..%d", hd, MAX_HD);
    Q6K_REQUIRE(page_size > 0 && max_blocks > 0 && window >= 0, "attention: bad page_size %d / max_blocks %d / window %d",
                page_size, max_blocks, window);
    Q6K_REQUIRE(Hkv <= 65535, "attention: %d KV heads exceed the grid limit", Hkv);
    const int G = Hq / Hkv;
    // Several tokens per request: row tiles (92 us against 500 where a step brings 509 tokens of one request).  A decode step (a token
    // each) would leave most of a tile's rows empty and keeps a block per token.  A tile takes 0.30 us a key for each request it
    // meets in turn, a warp of the other kernel 0.70 for a fourth of the heads: tiles of up to 4 tokens take every request; larger ones those that
    // fill half of one, so that none meets more than three.  The others then wait for a launch of their own, which pays where they are
    // few beside the rows of long portions (8 heads on 2, window of 128: 509 tokens beside 32 of one 315 -> 150 us, 60 beside 8 95 -> 114).
    const int heads = G < GT_ROWS ? G : GT_ROWS, tokens = GT_ROWS / heads;
    int least = tokens > 4 && requests > 1 && shortest < tokens / 2 ? tokens / 2 : 0;
    if (requests > 0 && T_ >= (least > 0 ? 16 : 4) * requests && (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0) {
        const size_t smem = (size_t)((GT_ROWS + 2 * GT_KEYS) * (hd + 4) + GT_ROWS * (GT_KEYS + 4) + GT_ROWS) * sizeof(float);
        const dim3 tiles((T_ + tokens - 1) / tokens, Hkv, (G + heads - 1) / heads);
#define TILED(NI)                                                                                                                                       \
    do {                                                                                                                                                \
        if (cudaFuncSetAttribute(attention_tiled_kernel<T, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)                 \
            return q6k_check_launch("attention_tiled: shared memory attribute");                                                                        \
        q6k_launch(attention_tiled_kernel<T, NI>, tiles, GT_THREADS, smem, st, (const T*)q, (const T*)k_pages, (const T*)v_pages, block_table,          \
                   max_blocks, page_size, num_pages, req_of_token, positions, window, sinks, scale, (T*)out, T_, Hq, Hkv, hd, tokens, heads, least);    \
    } while (0)
        Q6K_DISPATCH(dtype, {
            if (hd <= 32) TILED(1);
            else if (hd <= 64) TILED(2);
            else if (hd <= 128) TILED(4);
            else TILED(8);
        });
#undef TILED
        const int rc = q6k_check_launch("attention_tiled");
        if (rc || least == 0) return rc;
    } else {
        least = 0;
    }
    const int warps = G < 4 ? G : 4;
    dim3 grid(T_, Hkv);
    Q6K_DISPATCH(dtype, q6k_launch(attention_generic_kernel<T>, grid, warps * 32, warps * hd * sizeof(float), st, 
                            (const T*)q, (const T*)k_pages, (const T*)v_pages, block_table, max_blocks, page_size,
                            num_pages, req_of_token, positions, window, sinks, scale, (T*)out, T_, Hq, Hkv, hd, least););
    return q6k_check_launch("attention_generic");
}
