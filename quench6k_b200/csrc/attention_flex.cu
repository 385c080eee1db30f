// Attention over the paged cache with the shapes and masks the fixed-shape kernels do not take:
// keys and values of different widths (any width), values that are a leading slice of the key rows
// (a cached latent shared by all heads), a query given as an FP32 part followed by a part in the
// storage type, a causal mask narrowed by a sliding window and/or by chunks of positions, and,
// optionally, the heads' softmax weights mixed by a matrix before they meet the values.
// FP32 arithmetic on FP32 or bfloat16 storage: the kernels of the true 32-bit path for these
// shapes, and of the bfloat16 path where no tensor-core kernel covers the shape.
//
// Also here: the kernels that prepare q, k and v for them.
//
// Keys are walked in tiles of 32 aligned to multiples of 32 of the key index, so the order of
// every sum for a (position, head) depends neither on how the tokens were cut into steps nor on
// what else is in the batch.  Scores, softmax weights and their sums are FP32.
#include "common.cuh"

namespace {

constexpr int MAX_DV = 512, DPL = MAX_DV / 32;

// First visible key of position pos: causal, then the window (last `window` keys), then the chunk (keys of pos's own
// block of `chunk` positions, blocks counted from position 0).
__device__ __forceinline__ int first_visible(int pos, int window, int chunk) {
    int lo = 0;
    if (window > 0) lo = max(lo, pos - window + 1);
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    return lo;
}

template <typename T> struct Vec;
template <> struct Vec<float> { static constexpr int n = 4; };
template <> struct Vec<__nv_bfloat16> { static constexpr int n = 8; };

// q (FP32, shared memory) . row (storage type, global), dk elements; vec: the row starts on 16 bytes and dk is a multiple of the vector.
template <typename T>
__device__ __forceinline__ float dot_row(const float* q, const T* row, int dk, bool vec) {
    float acc = 0.0f;
    if (vec) {
        constexpr int V = Vec<T>::n;
        for (int d = 0; d < dk; d += V) {
            const uint4 raw = *reinterpret_cast<const uint4*>(row + d);
            const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int i = 0; i < V; ++i) acc = fmaf(q[d + i], to_f32(e[i]), acc);
        }
    } else {
        for (int d = 0; d < dk; ++d) acc = fmaf(q[d], to_f32(row[d]), acc);
    }
    return acc;
}

struct FlexArgs {
    const float* qa; int da;            // FP32 leading part of a query row (or null)
    const void* qb; int db;             // the rest, in the storage type (or null)
    int q_head_major;                   // row of (t, h): h * T + t, else t * H + h
    const void* k_pages; long long k_head_stride; int k_ld;
    const void* v_pages; long long v_head_stride; int v_ld; int dv;
    const int* block_table; int max_blocks; int page_size;
    const int* req_of_token; const int* positions;
    int window, chunk; float scale;
    const float* talk;                  // [H, H] or null
    void* out; int out_head_major;
    int T_, H, Hkv;
    const float* sinks;                 // [H] or null: exp(sinks[h]) joins head h's softmax denominator (no key, no value, not scaled)
    float softcap;                      // > 0: a scaled score s becomes softcap * tanh(s / softcap)
    int maps;                           // > 1: every head attends `maps` times with keys of its own over the same values: q holds
                                        // heads x maps rows per token (a head's maps side by side), the key pages Hkv = groups x maps
                                        // heads (a group's maps side by side), the value pages one head per group
    float* out_f32;                     // not null: the result leaves as FP32 here instead of through `out`
};

// The query row (of H per token) that key head kh serves as the g-th of its G, and the value head that goes with kh.
__device__ __forceinline__ int flex_query_head(int kh, int g, int G, int maps) { return maps > 1 ? ((kh / maps) * G + g) * maps + kh % maps : kh * G + g; }

template <typename T>
__device__ __forceinline__ void load_query(const FlexArgs& a, int t, int h, float* q) {
    const size_t row = a.q_head_major ? (size_t)h * a.T_ + t : (size_t)t * a.H + h;
    const int lane = threadIdx.x & 31;
    for (int d = lane; d < a.da; d += 32) q[d] = a.qa[row * a.da + d];
    const T* qb = (const T*)a.qb;
    for (int d = lane; d < a.db; d += 32) q[a.da + d] = to_f32(qb[row * a.db + d]);
}

// A block takes one (token, KV head); its warps take the G query heads of the group in turn.
template <typename T>
__global__ void __launch_bounds__(128) attention_flex_kernel(const FlexArgs a) {
    pdl_enter();
    extern __shared__ float qs[];             // [warps][dk]
    const int t = blockIdx.x, kh = blockIdx.y, G = a.H / a.Hkv, dk = a.da + a.db;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int pos = a.positions[t];
    const int* bt = a.block_table + (size_t)a.req_of_token[t] * a.max_blocks;
    const int lo = first_visible(pos, a.window, a.chunk);
    float* qw = qs + warp * dk;
    const T* kp = (const T*)a.k_pages + (size_t)kh * a.k_head_stride;
    const T* vp = (const T*)a.v_pages + (size_t)(a.maps > 1 ? kh / a.maps : kh) * a.v_head_stride;
    const bool vec = dk % Vec<T>::n == 0 && ((size_t)a.k_ld * sizeof(T)) % 16 == 0 && ((size_t)kp % 16) == 0;
    T* out = (T*)a.out;

    for (int g = warp; g < G; g += nwarps) {
        const int h = flex_query_head(kh, g, G, a.maps);
        load_query<T>(a, t, h, qw);
        __syncwarp();
        float m = -INFINITY, l = 0.0f, o[DPL];
#pragma unroll
        for (int i = 0; i < DPL; ++i) o[i] = 0.0f;
        for (int j0 = lo & ~31; j0 <= pos; j0 += 32) {
            const int j = j0 + lane;
            const bool ok = j >= lo && j <= pos;
            float s = -INFINITY;
            int rowi = 0;
            if (ok) {
                rowi = bt[j / a.page_size] * a.page_size + j % a.page_size;
                s = dot_row<T>(qw, kp + (size_t)rowi * a.k_ld, dk, vec) * a.scale;
                if (a.softcap > 0.0f) s = a.softcap * tanhf(s / a.softcap);
            }
            const float mn = fmaxf(m, warp_max(s));     // finite: the tile holds at least one visible key
            const float corr = m == -INFINITY ? 0.0f : expf(m - mn);
            const float p = ok ? expf(s - mn) : 0.0f;
            l = l * corr + warp_sum(p);
#pragma unroll
            for (int i = 0; i < DPL; ++i) o[i] *= corr;
            const int nk = min(32, pos - j0 + 1);
            for (int jj = max(0, lo - j0); jj < nk; ++jj) {
                const float pj = __shfl_sync(0xffffffffu, p, jj);
                const int rj = __shfl_sync(0xffffffffu, rowi, jj);
                if (pj == 0.0f) continue;               // uniform across the warp
                const T* vr = vp + (size_t)rj * a.v_ld;
#pragma unroll
                for (int i = 0; i < DPL; ++i) {
                    const int d = lane + 32 * i;
                    if (d < a.dv) o[i] = fmaf(pj, to_f32(vr[d]), o[i]);
                }
            }
            m = mn;
        }
        if (a.sinks) {                                  // the sink counts once in the denominator
            const float sk = a.sinks[h], mn = fmaxf(m, sk), corr = expf(m - mn);
            l = l * corr + expf(sk - mn);
#pragma unroll
            for (int i = 0; i < DPL; ++i) o[i] *= corr;
        }
        const float inv = 1.0f / l;
        const size_t orow = a.out_head_major ? (size_t)h * a.T_ + t : (size_t)t * a.H + h;
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            const int d = lane + 32 * i;
            if (d < a.dv) {
                if (a.out_f32) a.out_f32[orow * a.dv + d] = o[i] * inv;
                else out[orow * a.dv + d] = from_f32<T>(o[i] * inv);
            }
        }
        __syncwarp();
    }
}

// The heads' weights mixed before the values: w'_h(j) = sum_g talk[h, g] * softmax_g(j); head h applies w'_h to the values
// of its own KV head.  A block takes one token and all heads.  First every head's maximum and denominator over the
// visible keys, then, tile by tile, the normalised weights of all heads into shared memory, their mixture, and the
// weighted sum of the values.
template <typename T>
__global__ void __launch_bounds__(256) attention_talk_kernel(const FlexArgs a) {
    pdl_enter();
    extern __shared__ float sm[];             // q [H][dk] | max [H] | 1/den [H] | weights [H][32] | talk [H][H]
    const int t = blockIdx.x, H = a.H, G = H / a.Hkv, dk = a.da + a.db;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    float* q = sm;
    float* mx = q + (size_t)H * dk;
    float* rden = mx + H;
    float* pw = rden + H;
    float* tk = pw + H * 32;
    const int pos = a.positions[t];
    const int* bt = a.block_table + (size_t)a.req_of_token[t] * a.max_blocks;
    const int lo = first_visible(pos, a.window, a.chunk);
    const bool vec = dk % Vec<T>::n == 0 && ((size_t)a.k_ld * sizeof(T)) % 16 == 0 && ((size_t)a.k_pages % 16) == 0 &&
                     ((size_t)a.k_head_stride * sizeof(T)) % 16 == 0;
    T* out = (T*)a.out;
    for (int i = threadIdx.x; i < H * H; i += blockDim.x) tk[i] = a.talk[i];
    for (int g = warp; g < H; g += nwarps) {
        load_query<T>(a, t, g, q + (size_t)g * dk);
        __syncwarp();
        const T* kp = (const T*)a.k_pages + (size_t)(g / G) * a.k_head_stride;
        float m = -INFINITY, l = 0.0f;
        for (int j0 = lo & ~31; j0 <= pos; j0 += 32) {
            const int j = j0 + lane;
            const bool ok = j >= lo && j <= pos;
            float s = -INFINITY;
            if (ok) {
                const int rowi = bt[j / a.page_size] * a.page_size + j % a.page_size;
                s = dot_row<T>(q + (size_t)g * dk, kp + (size_t)rowi * a.k_ld, dk, vec) * a.scale;
            }
            const float mn = fmaxf(m, warp_max(s));
            const float corr = m == -INFINITY ? 0.0f : expf(m - mn);
            l = l * corr + warp_sum(ok ? expf(s - mn) : 0.0f);
            m = mn;
        }
        if (lane == 0) {
            mx[g] = m;
            rden[g] = 1.0f / l;
        }
    }
    __syncthreads();
    // each warp keeps the running sums of the heads it owns: heads warp, warp + nwarps, ... (at most MAX_OWN of them)
    constexpr int MAX_OWN = 8, DPLT = 8;       // at most 64 heads, value widths up to 256 here
    float o[MAX_OWN][DPLT];
#pragma unroll
    for (int u = 0; u < MAX_OWN; ++u)
#pragma unroll
        for (int i = 0; i < DPLT; ++i) o[u][i] = 0.0f;
    for (int j0 = lo & ~31; j0 <= pos; j0 += 32) {
        const int j = j0 + lane;
        const bool ok = j >= lo && j <= pos;
        const int rowi = ok ? bt[j / a.page_size] * a.page_size + j % a.page_size : 0;
        for (int g = warp; g < H; g += nwarps) {
            const T* kp = (const T*)a.k_pages + (size_t)(g / G) * a.k_head_stride;
            float p = 0.0f;
            if (ok) p = expf(dot_row<T>(q + (size_t)g * dk, kp + (size_t)rowi * a.k_ld, dk, vec) * a.scale - mx[g]) * rden[g];
            pw[g * 32 + lane] = p;
        }
        __syncthreads();
        const int nk = min(32, pos - j0 + 1);
#pragma unroll
        for (int u = 0; u < MAX_OWN; ++u) {
            const int h = warp + u * nwarps;
            if (h < H) {
                float mixed = 0.0f;
                for (int g = 0; g < H; ++g) mixed = fmaf(tk[h * H + g], pw[g * 32 + lane], mixed);
                const T* vp = (const T*)a.v_pages + (size_t)(h / G) * a.v_head_stride;
                for (int jj = max(0, lo - j0); jj < nk; ++jj) {
                    const float pj = __shfl_sync(0xffffffffu, mixed, jj);
                    const int rj = __shfl_sync(0xffffffffu, rowi, jj);
                    const T* vr = vp + (size_t)rj * a.v_ld;
#pragma unroll
                    for (int i = 0; i < DPLT; ++i) {
                        const int d = lane + 32 * i;
                        if (d < a.dv) o[u][i] = fmaf(pj, to_f32(vr[d]), o[u][i]);
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < MAX_OWN; ++u) {
        const int h = warp + u * nwarps;
        if (h < H) {
            const size_t orow = a.out_head_major ? (size_t)h * a.T_ + t : (size_t)t * H + h;
#pragma unroll
            for (int i = 0; i < DPLT; ++i) {
                const int d = lane + 32 * i;
                if (d < a.dv) out[orow * a.dv + d] = from_f32<T>(o[u][i]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ preparation
// The first `rd` of n values in shared memory x turn by pos * inv_freq[pair]; returns element d's new value.
__device__ __forceinline__ float rotated(const float* x, int d, int rd, int neighbours, int pos, const float* inv_freq) {
    if (d >= rd) return x[d];
    const int half = rd / 2;
    const int i = neighbours ? d >> 1 : (d < half ? d : d - half);
    const bool first = neighbours ? !(d & 1) : d < half;
    const int partner = neighbours ? d ^ 1 : (first ? d + half : d - half);
    float sn, cs;
    sincosf((float)pos * inv_freq[i], &sn, &cs);
    return first ? x[d] * cs - x[partner] * sn : x[d] * cs + x[partner] * sn;
}

// qkv: FP32 [T, ld] = [Hq heads of hd | Hkv heads of hd | Hv heads of vd].  Per-head RMS norm of q and k (weights or
// null), rotation of their first rd dimensions (inv_freq or null), q -> q_out [T, Hq, hd]; k, v -> pages
// [Hkv, num_pages, page_size, hd] and [Hv, .., vd].  Grid (T, Hq + Hkv + Hv) (or (T, Hq) when nothing is written).
// bias: one entry per column of a row, added to the summed slices, or null.  v_is_k: the rows hold no v heads; a value is its
// key as projected (bias included, before norm and rotation).  v_norm: a value is divided by its root mean square (no weight).
template <typename T>
__global__ void __launch_bounds__(128) qkv_pages_kernel(const float* qkv, int ld, int splits, size_t split_stride, int Hq, int Hkv, int hd, int vd,
                                                        const float* q_norm, const float* k_norm, float eps, const float* inv_freq, int rd,
                                                        int neighbours, const int* positions, const int* req_of_token,
                                                        const int* block_table, int max_blocks, int page_size, int num_pages, T* q_out,
                                                        T* k_pages, T* v_pages, int Hv, const float* bias, int v_is_k, int v_norm) {
    pdl_enter();
    extern __shared__ float xs[];            // max(hd, vd) floats
    __shared__ float red[32];
    const int t = blockIdx.x, h = blockIdx.y;
    const int kind = h < Hq ? 0 : h < Hq + Hkv ? 1 : 2;
    const int pos = positions[t];
    const int n = kind == 2 ? vd : hd;
    // a value head of a layer whose values are its keys reads the key head of its number (as projected)
    const size_t col = kind == 0 ? (size_t)h * hd : kind == 1 ? (size_t)Hq * hd + (size_t)(h - Hq) * hd
                     : v_is_k    ? (size_t)Hq * hd + (size_t)(h - Hq - Hkv) * hd
                                 : (size_t)(Hq + Hkv) * hd + (size_t)(h - Hq - Hkv) * vd;
    const float* src = qkv + (size_t)t * ld + col;
    float ss = 0.0f;
    for (int d = threadIdx.x; d < n; d += blockDim.x) {
        float v = src[d];
        for (int s = 1; s < splits; ++s) v += src[s * split_stride + d];
        if (bias) v += bias[col + d];
        xs[d] = v;
        ss = fmaf(v, v, ss);
    }
    const float* nw = kind == 0 ? q_norm : kind == 1 ? k_norm : nullptr;
    if (nw || (kind == 2 && v_norm)) {
        const float inv = rsqrtf(block_sum(ss, red) / (float)n + eps);
        for (int d = threadIdx.x; d < n; d += blockDim.x) xs[d] = xs[d] * inv * (nw ? nw[d] : 1.0f);
    }
    __syncthreads();
    T* dst;
    if (kind == 0) {
        dst = q_out + ((size_t)t * Hq + h) * hd;
    } else {
        const int page = block_table[(size_t)req_of_token[t] * max_blocks + pos / page_size];
        if (page < 0) return;
        const int kh = kind == 1 ? h - Hq : h - Hq - Hkv;
        dst = (kind == 1 ? k_pages : v_pages) + (((size_t)kh * num_pages + page) * page_size + pos % page_size) * n;
    }
    const bool turns = inv_freq && kind != 2;
    for (int d = threadIdx.x; d < n; d += blockDim.x) dst[d] = from_f32<T>(turns ? rotated(xs, d, rd, neighbours, pos, inv_freq) : xs[d]);
}

// The same with a warp per (token, head), eight heads a block, for heads of at most 256 entries: a lane keeps its entries
// (lane, lane + 32, ...) in registers, the head passes through the warp's stretch of shared memory once for the rotation's
// partners, and the sums of squares are a warp's shuffles.  Same arithmetic and order of sums per head as the block kernel
// has for one warp's share; which of the two runs depends on the head widths alone.
template <typename T>
__global__ void __launch_bounds__(256) qkv_pages_warp_kernel(const float* qkv, int ld, int splits, size_t split_stride, int Hq, int Hkv, int hd, int vd,
                                                             const float* q_norm, const float* k_norm, float eps, const float* inv_freq, int rd,
                                                             int neighbours, const int* positions, const int* req_of_token,
                                                             const int* block_table, int max_blocks, int page_size, int num_pages, T* q_out,
                                                             T* k_pages, T* v_pages, int heads, const float* bias, int v_is_k, int v_norm) {
    pdl_enter();
    __shared__ float stage[8][256];
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y * 8 + warp;
    if (h >= heads) return;
    const int kind = h < Hq ? 0 : h < Hq + Hkv ? 1 : 2;
    const int pos = positions[t];
    const int n = kind == 2 ? vd : hd;
    // a value head of a layer whose values are its keys reads the key head of its number (as projected)
    const size_t col = kind == 0 ? (size_t)h * hd : kind == 1 ? (size_t)Hq * hd + (size_t)(h - Hq) * hd
                     : v_is_k    ? (size_t)Hq * hd + (size_t)(h - Hq - Hkv) * hd
                                 : (size_t)(Hq + Hkv) * hd + (size_t)(h - Hq - Hkv) * vd;
    const float* src = qkv + (size_t)t * ld + col;
    float x[8];
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int d = lane + 32 * j;
        float v = 0.0f;
        if (d < n) {
            v = src[d];
            for (int s = 1; s < splits; ++s) v += src[s * split_stride + d];
            if (bias) v += bias[col + d];
        }
        x[j] = v;
        ss = fmaf(v, v, ss);
    }
    const float* nw = kind == 0 ? q_norm : kind == 1 ? k_norm : nullptr;
    if (nw || (kind == 2 && v_norm)) {
        const float inv = rsqrtf(warp_sum(ss) / (float)n + eps);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int d = lane + 32 * j;
            if (d < n) x[j] = x[j] * inv * (nw ? nw[d] : 1.0f);
        }
    }
    T* dst;
    if (kind == 0) {
        dst = q_out + ((size_t)t * Hq + h) * hd;
    } else {
        const int page = block_table[(size_t)req_of_token[t] * max_blocks + pos / page_size];
        if (page < 0) return;
        const int kh = kind == 1 ? h - Hq : h - Hq - Hkv;
        dst = (kind == 1 ? k_pages : v_pages) + (((size_t)kh * num_pages + page) * page_size + pos % page_size) * n;
    }
    const bool turns = inv_freq && kind != 2 && rd > 0;
    if (turns) {
        float* xs = stage[warp];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int d = lane + 32 * j;
            if (d < n) xs[d] = x[j];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int d = lane + 32 * j;
            if (d < n) dst[d] = from_f32<T>(rotated(xs, d, rd, neighbours, pos, inv_freq));
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int d = lane + 32 * j;
        if (d < n) dst[d] = from_f32<T>(x[j]);
    }
}

__device__ __forceinline__ void store4(float* out, float4 v) { *reinterpret_cast<float4*>(out) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* out, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(out) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// The same again for heads of 16 to 128 entries (powers of two) that fill rows of 128 columns evenly: a warp takes stretches of 128
// columns, 16 bytes a lane, asks for two of them first, and a head's lanes add its squares among themselves.  The kernel
// above, which reads 4 bytes a lane and starts a warp per head, took 45 us for 2,465 tokens of 44 heads (30 MB), waiting
// for its chain of loads; this one takes 20 (16 for 23 where 2,048 tokens have 24 heads of 128).
constexpr int QR_WARPS = 8, QR_EACH = 2;

// grid (T, ceil(stretches / 16)), 256 threads.
template <typename T>
__global__ void __launch_bounds__(QR_WARPS * 32) qkv_rows_kernel(const float* qkv, int ld, int splits, size_t split_stride, int Hq, int Hkv, int Hv, int hd, int vd,
                                                                 const float* q_norm, const float* k_norm, float eps, const float* inv_freq, int rd,
                                                                 int neighbours, const int* positions, const int* req_of_token, const int* block_table,
                                                                 int max_blocks, int page_size, int num_pages, T* q_out, T* k_pages, T* v_pages,
                                                                 int write_kv, const float* bias, int v_is_k, int v_norm) {
    pdl_enter();
    __shared__ float stage[QR_WARPS][128];
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pos = positions[t];
    const int q_end = Hq * hd / 128, k_end = q_end + (write_kv ? Hkv * hd / 128 : 0), end = k_end + (write_kv ? Hv * vd / 128 : 0);
    const int page = write_kv ? block_table[(size_t)req_of_token[t] * max_blocks + pos / page_size] : -1;
    float4 x[QR_EACH];
#pragma unroll
    for (int e = 0; e < QR_EACH; ++e) {
        const int s = blockIdx.y * QR_WARPS * QR_EACH + e * QR_WARPS + warp;
        const int from = (s < k_end || !v_is_k ? s : s - k_end + q_end) * 128 + lane * 4;       // v_is_k: a value head reads the key head of its number
        x[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (s >= end) continue;
        const float* src = qkv + (size_t)t * ld + from;
        x[e] = *reinterpret_cast<const float4*>(src);
        for (int i = 1; i < splits; ++i) {
            const float4 y = *reinterpret_cast<const float4*>(src + i * split_stride);
            x[e].x += y.x, x[e].y += y.y, x[e].z += y.z, x[e].w += y.w;
        }
        if (bias) {
            const float4 y = *reinterpret_cast<const float4*>(bias + from);
            x[e].x += y.x, x[e].y += y.y, x[e].z += y.z, x[e].w += y.w;
        }
    }
#pragma unroll
    for (int e = 0; e < QR_EACH; ++e) {
        const int s = blockIdx.y * QR_WARPS * QR_EACH + e * QR_WARPS + warp;
        if (s >= end) break;
        const int kind = s < q_end ? 0 : s < k_end ? 1 : 2, n = kind == 2 ? vd : hd;
        const int col = (s - (kind == 0 ? 0 : kind == 1 ? q_end : k_end)) * 128 + lane * 4, h = col / n, d = col % n;     // head of its kind, entry in it
        const float* nw = kind == 0 ? q_norm : kind == 1 ? k_norm : nullptr;
        if (nw || (kind == 2 && v_norm)) {
            float ss = fmaf(x[e].w, x[e].w, fmaf(x[e].z, x[e].z, fmaf(x[e].y, x[e].y, x[e].x * x[e].x)));
            for (int o = n / 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float inv = rsqrtf(ss / (float)n + eps);
            const float4 w = nw ? make_float4(nw[d], nw[d + 1], nw[d + 2], nw[d + 3]) : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
            x[e] = make_float4(x[e].x * inv * w.x, x[e].y * inv * w.y, x[e].z * inv * w.z, x[e].w * inv * w.w);
        }
        if (inv_freq && kind != 2 && rd > 0) {
            *reinterpret_cast<float4*>(&stage[warp][lane * 4]) = x[e];
            __syncwarp();
            const float* xs = &stage[warp][lane * 4 - d];
            x[e] = make_float4(rotated(xs, d, rd, neighbours, pos, inv_freq), rotated(xs, d + 1, rd, neighbours, pos, inv_freq),
                               rotated(xs, d + 2, rd, neighbours, pos, inv_freq), rotated(xs, d + 3, rd, neighbours, pos, inv_freq));
            __syncwarp();
        }
        if (kind == 0) store4(q_out + ((size_t)t * Hq + h) * hd + d, x[e]);
        else if (page >= 0) store4((kind == 1 ? k_pages : v_pages) + (((size_t)h * num_pages + page) * page_size + pos % page_size) * n + d, x[e]);
    }
}

// The inputs of attention over a cached latent.  x: FP32 [T, ld] = [H query heads of (dim + rd) | latent of `rank` | rd].
// Block (t, h < H): the head's first `dim` values -> qn[(h T + t) dim] (they go through the key up-projection next), its
// last rd values, the first `turn` of them rotated -> qr[(h T + t) rd].  Block (t, H): the latent, RMS-normed with weight
// cw -> the page row's first `rank` values; the shared rotated key part -> the row's last rd.  neighbours: the rotation
// pairs 2i with 2i+1 instead of i with i + turn/2.  A layer that reads another layer's pages has no block (t, H) (and x no
// latent columns).  The latent (and the shared key part after it) is read from rows of its own: xc + t ldc.
template <typename T>
__global__ void __launch_bounds__(128) latent_prep_kernel(const float* x, int ld, const float* xc, int ldc, int H, int dim, int rd, int rank, const float* cw, float eps,
                                                          const float* inv_freq, int turn, int neighbours, const int* positions,
                                                          const int* req_of_token, const int* block_table, int max_blocks, int page_size,
                                                          T* qn, T* qr, T* pages, int T_) {
    pdl_enter();
    extern __shared__ float xs[];            // rd floats (the part that turns)
    __shared__ float red[32];
    const int t = blockIdx.x, h = blockIdx.y, pos = positions[t];
    if (h < H) {
        const float* src = x + (size_t)t * ld + (size_t)h * (dim + rd);
        const size_t row = (size_t)h * T_ + t;
        for (int d = threadIdx.x; d < dim; d += blockDim.x) qn[row * dim + d] = from_f32<T>(src[d]);
        for (int d = threadIdx.x; d < rd; d += blockDim.x) xs[d] = src[dim + d];
        __syncthreads();
        for (int d = threadIdx.x; d < rd; d += blockDim.x) qr[row * rd + d] = from_f32<T>(rotated(xs, d, turn, neighbours, pos, inv_freq));
        return;
    }
    const float* src = xc + (size_t)t * ldc;
    float ss = 0.0f;
    for (int d = threadIdx.x; d < rank; d += blockDim.x) ss = fmaf(src[d], src[d], ss);
    const float inv = rsqrtf(block_sum(ss, red) / (float)rank + eps);
    for (int d = threadIdx.x; d < rd; d += blockDim.x) xs[d] = src[rank + d];
    __syncthreads();
    const int page = block_table[(size_t)req_of_token[t] * max_blocks + pos / page_size];
    if (page < 0) return;
    T* dst = pages + ((size_t)page * page_size + pos % page_size) * (rank + rd);
    for (int d = threadIdx.x; d < rank; d += blockDim.x) dst[d] = from_f32<T>(src[d] * inv * cw[d]);
    for (int d = threadIdx.x; d < rd; d += blockDim.x) dst[rank + d] = from_f32<T>(rotated(xs, d, turn, neighbours, pos, inv_freq));
}

// The same with a block for all of a token's heads, 16 bytes a read (dim, rd and ld multiples of 4), and the sines and cosines of a
// token's angles made once: a block of 128 threads per (token, head) took 39 us for 2,048 tokens of 16 heads of 128 + 64;
// this one takes 17.  The second block of a token is the latent's, as above.
// grid (T, pages ? 2 : 1), 256 threads; dynamic shared memory: cos [turn / 2] | sin [turn / 2] | the rotated parts [H][rd].
template <typename T>
__global__ void __launch_bounds__(256) latent_rows_kernel(const float* x, int ld, const float* xc, int ldc, int H, int dim, int rd, int rank, const float* cw, float eps,
                                                          const float* inv_freq, int turn, int neighbours, const int* positions,
                                                          const int* req_of_token, const int* block_table, int max_blocks, int page_size,
                                                          T* qn, T* qr, T* pages, int T_) {
    pdl_enter();
    extern __shared__ __align__(16) float sm[];
    __shared__ float red[32];
    const int t = blockIdx.x, pos = positions[t], half = turn / 2;
    float *xs = sm, *cs = sm + (blockIdx.y == 0 ? H : 1) * rd, *sn = cs + half;
    auto turned = [&](const float* v, int d) {              // rotated() with the angles' table
        if (d >= turn) return v[d];
        const int i = neighbours ? d >> 1 : (d < half ? d : d - half);
        const bool first = neighbours ? !(d & 1) : d < half;
        const int partner = neighbours ? d ^ 1 : (first ? d + half : d - half);
        return first ? v[d] * cs[i] - v[partner] * sn[i] : v[d] * cs[i] + v[partner] * sn[i];
    };
    for (int i = threadIdx.x; i < half; i += 256) sincosf((float)pos * inv_freq[i], &sn[i], &cs[i]);
    if (blockIdx.y == 0) {
        const float* src = x + (size_t)t * ld;
        const int head4 = (dim + rd) / 4;
#pragma unroll 4
        for (int i = threadIdx.x; i < H * head4; i += 256) {
            const float4 v = *reinterpret_cast<const float4*>(src + 4 * i);
            const int h = i / head4, d = (i - h * head4) * 4;
            if (d < dim) store4(qn + ((size_t)h * T_ + t) * dim + d, v);
            else *reinterpret_cast<float4*>(xs + h * rd + d - dim) = v;
        }
        __syncthreads();
        for (int i = threadIdx.x * 4; i < H * rd; i += 1024) {
            const int h = i / rd, d = i - h * rd;
            const float* v = xs + h * rd;
            store4(qr + ((size_t)h * T_ + t) * rd + d, make_float4(turned(v, d), turned(v, d + 1), turned(v, d + 2), turned(v, d + 3)));
        }
        return;
    }
    const float* src = xc + (size_t)t * ldc;
    float ss = 0.0f;
    for (int d = threadIdx.x; d < rank; d += 256) ss = fmaf(src[d], src[d], ss);
    for (int d = threadIdx.x; d < rd; d += 256) xs[d] = src[rank + d];
    const float inv = rsqrtf(block_sum(ss, red) / (float)rank + eps);
    __syncthreads();
    const int page = block_table[(size_t)req_of_token[t] * max_blocks + pos / page_size];
    if (page < 0) return;
    T* dst = pages + ((size_t)page * page_size + pos % page_size) * (rank + rd);
    for (int d = threadIdx.x; d < rank; d += 256) dst[d] = from_f32<T>(src[d] * inv * cw[d]);
    for (int d = threadIdx.x; d < rd; d += 256) dst[rank + d] = from_f32<T>(turned(xs, d));
}

// The latents that prompt portions see, for the product that expands them: every position of every request, a request after the other, each from a
// multiple of 64 rows on, from its page into lat [rows, rank] (zeros in the rows between), its rotated part behind each of the H heads' expanded keys,
// whose rows of dim entries lie `pitch` apart, [H, rows, pitch].  16 bytes at a time: everything a multiple of 8 entries.  Which request and position a
// row is follows from q_start and pos_start (32 requests a look: a warp sums their blocks of 64 rows); blocks [R, wide] receives every request's blocks,
// the last one in the places beyond.  (As lists made on the host this took two uploads of a step, which waited for the GPU.)  grid (rows), 128 threads.
__global__ void __launch_bounds__(128) latent_context_kernel(const uint4* pages, const int* q_start, const int* pos_start, int R, const int* block_table, int max_blocks, int page_size,
                                                             uint4* lat, uint4* keys, int* blocks, int wide, int rank8, int rd8, int dim8, int pitch8, int H) {
    pdl_enter();
    const int row = blockIdx.x, block = row >> 6, lane = threadIdx.x & 31;
    int r = -1, first = 0, count = 0, reach = 0;                                  // of this row's request: its first block, its blocks, its positions
    for (int r0 = 0, before = 0; r0 < R && r < 0; r0 += 32) {
        const int q = r0 + lane, sees = q < R ? pos_start[q] + q_start[q + 1] - q_start[q] : 0, n = (sees + 63) >> 6;
        int sum = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        const unsigned beyond = __ballot_sync(0xffffffffu, before + sum > block);
        if (beyond) {
            const int l = __ffs(beyond) - 1;
            r = r0 + l, count = __shfl_sync(0xffffffffu, n, l), reach = __shfl_sync(0xffffffffu, sees, l);
            first = before + __shfl_sync(0xffffffffu, sum, l) - count;
        }
        before += __shfl_sync(0xffffffffu, sum, 31);
    }
    const int pos = row - first * 64, page = r >= 0 && pos < reach ? block_table[(size_t)r * max_blocks + pos / page_size] : -1;
    if (r >= 0 && (row & 63) == 0)
        for (int i = block - first + threadIdx.x; i < (block - first + 1 < count ? min(block - first + 1, wide) : wide); i += 128) blocks[(size_t)r * wide + i] = block;
    const uint4* src = pages + ((size_t)max(page, 0) * page_size + pos % page_size) * (rank8 + rd8);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < rank8; i += 128) lat[(size_t)row * rank8 + i] = page >= 0 ? src[i] : zero;
    for (int i = threadIdx.x; i < H * rd8; i += 128) {
        const int h = i / rd8, c = i - h * rd8;
        keys[((size_t)h * gridDim.x + row) * pitch8 + dim8 + c] = page >= 0 ? src[rank8 + c] : zero;
    }
}

// src: FP32 [H, T, n] -> out: [T, H n] in the storage type, four values a thread (n4 = n / 4; a value a thread took 19 us for 2,048 rows
// of 16 x 128, 25 MB; so 6).
template <typename T>
__global__ void __launch_bounds__(256) heads_to_rows4_kernel(const float4* src, T* out, int H, int T_, int n4, int total) {
    pdl_enter();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const int th = i / n4, t = th / H, h = th - t * H;
    store4(out + 4 * (size_t)i, src[((size_t)h * T_ + t) * n4 + (i - th * n4)]);
}

// The same for any n.
template <typename T>
__global__ void heads_to_rows_kernel(const float* src, T* out, int H, int T_, int n) {
    pdl_enter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)H * T_ * n) return;
    const int d = i % n;
    const size_t th = i / n;
    const int h = th % H;
    const size_t t = th / H;
    out[i] = from_f32<T>(src[((size_t)h * T_ + t) * n + d]);
}

// The two maps of a head combined: a FP32 [T, H, 2, dv] (a head's maps side by side) -> out [T, H dv] in the storage type,
// o = a1 - lambda a2, then o / sqrt(mean(o^2) + eps) * mult over the head's dv values.  A warp per (token, head).
template <typename T>
__global__ void __launch_bounds__(128) map_difference_kernel(const float* a, T* out, int rows, int dv, float lambda, float eps, float mult) {
    pdl_enter();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* a1 = a + (size_t)row * 2 * dv;
    const float* a2 = a1 + dv;
    float ss = 0.0f;
    for (int d = lane; d < dv; d += 32) {
        const float o = a1[d] - lambda * a2[d];
        ss = fmaf(o, o, ss);
    }
    const float inv = rsqrtf(warp_sum(ss) / (float)dv + eps) * mult;
    for (int d = lane; d < dv; d += 32) out[(size_t)row * dv + d] = from_f32<T>((a1[d] - lambda * a2[d]) * inv);
}

// The same, 16 bytes a read (dv a multiple of 4).
template <typename T>
__global__ void __launch_bounds__(128) map_difference4_kernel(const float* a, T* out, int rows, int dv, float lambda, float eps, float mult) {
    pdl_enter();
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* a1 = a + (size_t)row * 2 * dv;
    auto at = [&](int d) {
        const float4 x = *reinterpret_cast<const float4*>(a1 + d), y = *reinterpret_cast<const float4*>(a1 + dv + d);
        return make_float4(x.x - lambda * y.x, x.y - lambda * y.y, x.z - lambda * y.z, x.w - lambda * y.w);
    };
    float ss = 0.0f;
    for (int d = lane * 4; d < dv; d += 128) {
        const float4 o = at(d);
        ss = fmaf(o.w, o.w, fmaf(o.z, o.z, fmaf(o.y, o.y, fmaf(o.x, o.x, ss))));
    }
    const float inv = rsqrtf(warp_sum(ss) / (float)dv + eps) * mult;
    for (int d = lane * 4; d < dv; d += 128) {
        const float4 o = at(d);
        store4(out + (size_t)row * dv + d, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
    }
}

// Every head's result times the sigmoid of its number: a [T, H, n] in the storage type, in place; the numbers are columns
// col .. col + H of p, FP32 [slices, T, ld], the slices added in order.  A warp per (token, head).
template <typename T>
__global__ void __launch_bounds__(128) gate_heads_kernel(T* a, const float* p, int slices, size_t slice_stride, int ld, int col, int rows, int H, int n) {
    pdl_enter();
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* src = p + (size_t)(row / H) * ld + col + row % H;
    float z = src[0];
    for (int s = 1; s < slices; ++s) z += src[s * slice_stride];
    const float g = 1.0f / (1.0f + expf(-z));
    T* mine = a + (size_t)row * n;
    for (int d = lane; d < n; d += 32) mine[d] = from_f32<T>(to_f32(mine[d]) * g);
}

// The same for bfloat16 heads of a multiple of eight entries: a thread takes eight (16 bytes) and reads its head's number at
// the same time.
__global__ void __launch_bounds__(256) gate_heads8_kernel(__nv_bfloat16* a, const float* p, int slices, size_t slice_stride, int ld, int col, long long count,
                                                          int H, int n8) {
    pdl_enter();
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    if (idx >= count) return;
    const int row = (int)(idx / n8);
    uint4* at = reinterpret_cast<uint4*>(a) + idx;
    uint4 u = *at;
    const float* src = p + (size_t)(row / H) * ld + col + row % H;
    float z = src[0];
    for (int s = 1; s < slices; ++s) z += src[s * slice_stride];
    const float g = 1.0f / (1.0f + expf(-z));
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        h[i] = __floats2bfloat162_rn(f.x * g, f.y * g);
    }
    *at = u;
}

// out[t] = T(x[t, col : col + n] over its root mean square times w): n columns of FP32 rows, normed on their own.  A block per row.
template <typename T>
__global__ void __launch_bounds__(128) norm_columns_kernel(const float* x, int ld, int col, int n, const float* w, float eps, T* out) {
    pdl_enter();
    __shared__ float red[32];
    const float* src = x + (size_t)blockIdx.x * ld + col;
    constexpr int KEEP = 8;                    // entries a thread keeps between the two passes; wider rows are read again
    float v[KEEP], ss = 0.0f;
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        const int d = threadIdx.x + 128 * j;
        v[j] = d < n ? src[d] : 0.0f;
        ss = fmaf(v[j], v[j], ss);
    }
    for (int d = threadIdx.x + 128 * KEEP; d < n; d += 128) ss = fmaf(src[d], src[d], ss);
    const float inv = rsqrtf(block_sum(ss, red) / (float)n + eps);
    T* dst = out + (size_t)blockIdx.x * n;
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        const int d = threadIdx.x + 128 * j;
        if (d < n) dst[d] = from_f32<T>(v[j] * inv * w[d]);
    }
    for (int d = threadIdx.x + 128 * KEEP; d < n; d += 128) dst[d] = from_f32<T>(src[d] * inv * w[d]);
}

// The same for at most 1,024 columns that come in fours and start on 16 bytes: a thread takes four.
template <typename T>
__global__ void __launch_bounds__(256) norm_columns4_kernel(const float* x, int ld, int col, int n, const float* w, float eps, T* out) {
    pdl_enter();
    __shared__ float red[32];
    const int d = threadIdx.x * 4;
    const float4 v = d < n ? *reinterpret_cast<const float4*>(x + (size_t)blockIdx.x * ld + col + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 g = d < n ? *reinterpret_cast<const float4*>(w + d) : v;
    const float inv = rsqrtf(block_sum(fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))), red) / (float)n + eps);
    if (d >= n) return;
    T* dst = out + (size_t)blockIdx.x * n + d;
    dst[0] = from_f32<T>(v.x * inv * g.x), dst[1] = from_f32<T>(v.y * inv * g.y), dst[2] = from_f32<T>(v.z * inv * g.z), dst[3] = from_f32<T>(v.w * inv * g.w);
}

}  // namespace

Q6K_API int q6k_gate_heads(void* a, const float* p, int slices, long long slice_stride, int ld, int col, int T_, int H, int n, int dtype, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && H > 0 && n > 0 && slices >= 1 && col >= 0 && col + H <= ld && (long long)T_ * H <= 0x7fffffffLL, "gate_heads: bad sizes T=%d H=%d n=%d", T_, H, n);
    if (dtype == Q6K_BF16 && n % 8 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0) {
        const long long count = (long long)T_ * H * (n / 8);
        q6k_launch(gate_heads8_kernel, dim3((unsigned)((count + 255) / 256)), 256, 0, st, (__nv_bfloat16*)a, p, slices, (size_t)slice_stride, ld, col, count, H, n / 8);
        return q6k_check_launch("gate_heads");
    }
    Q6K_DISPATCH(dtype, q6k_launch(gate_heads_kernel<T>, dim3((unsigned)(((long long)T_ * H + 3) / 4)), 128, 0, st, (T*)a, p, slices, (size_t)slice_stride, ld, col,
                                   T_ * H, H, n););
    return q6k_check_launch("gate_heads");
}

Q6K_API int q6k_norm_columns(const float* x, int ld, int col, int n, const float* w, float eps, void* out, int T_, int dtype, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && n > 0 && col >= 0 && col + n <= ld && w, "norm_columns: bad sizes T=%d n=%d", T_, n);
    if (n % 4 == 0 && n <= 1024 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(x + col) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
        Q6K_DISPATCH(dtype, q6k_launch(norm_columns4_kernel<T>, dim3(T_), (n / 4 + 31) / 32 * 32, 0, st, x, ld, col, n, w, eps, (T*)out););
        return q6k_check_launch("norm_columns");
    }
    Q6K_DISPATCH(dtype, q6k_launch(norm_columns_kernel<T>, dim3(T_), 128, 0, st, x, ld, col, n, w, eps, (T*)out););
    return q6k_check_launch("norm_columns");
}

Q6K_API int q6k_map_difference(const float* a, void* out, int T_, int H, int dv, float lambda, float eps, float mult, int dtype, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && H > 0 && dv > 0, "map_difference: bad sizes T=%d H=%d dv=%d", T_, H, dv);
    const long long rows = (long long)T_ * H;
    Q6K_REQUIRE(rows <= 0x7fffffffLL, "map_difference: too many rows");
    if (dv % 4 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)out & (dtype == Q6K_F32 ? 15 : 7)) == 0) {
        Q6K_DISPATCH(dtype, q6k_launch(map_difference4_kernel<T>, dim3((unsigned)((rows + 3) / 4)), 128, 0, st, a, (T*)out, (int)rows, dv, lambda, eps, mult););
        return q6k_check_launch("map_difference");
    }
    Q6K_DISPATCH(dtype, q6k_launch(map_difference_kernel<T>, dim3((unsigned)((rows + 3) / 4)), 128, 0, st, a, (T*)out, (int)rows, dv, lambda, eps, mult););
    return q6k_check_launch("map_difference");
}

Q6K_API int q6k_attention_flex(const float* qa, int da, const void* qb, int db, int q_head_major, const void* k_pages,
                               long long k_head_stride, int k_ld, const void* v_pages, long long v_head_stride, int v_ld, int dv,
                               const int* block_table, int max_blocks, int page_size, const int* req_of_token, const int* positions,
                               int window, int chunk, float scale, const float* talk, const float* sinks, void* out, int out_head_major,
                               int T_, int H, int Hkv, int dtype, float softcap, int maps, float* out_f32, cudaStream_t st) {
    if (T_ == 0) return 0;
    const int dk = da + db;
    Q6K_REQUIRE(maps >= 1 && Hkv % maps == 0 && softcap >= 0.0f, "attention: %d maps over %d key heads, softcap %f", maps, Hkv, softcap);
    Q6K_REQUIRE(!talk || (maps == 1 && softcap == 0.0f && !out_f32), "attention with mixed heads takes neither maps, a cap nor FP32 results");
    Q6K_REQUIRE(T_ > 0 && H > 0 && Hkv > 0 && H % Hkv == 0, "attention: bad head counts H=%d Hkv=%d", H, Hkv);
    Q6K_REQUIRE(da >= 0 && db >= 0 && dk > 0 && (da == 0 || qa) && (db == 0 || qb), "attention: bad query parts %d + %d", da, db);
    Q6K_REQUIRE(dv > 0 && dv <= MAX_DV, "attention: value width %d outside 1..%d", dv, MAX_DV);
    Q6K_REQUIRE(page_size > 0 && max_blocks > 0 && window >= 0 && chunk >= 0, "attention: bad page_size %d / max_blocks %d / window %d / chunk %d",
                page_size, max_blocks, window, chunk);
    FlexArgs a{qa, da, qb, db, q_head_major, k_pages, k_head_stride, k_ld, v_pages, v_head_stride, v_ld, dv, block_table, max_blocks,
               page_size, req_of_token, positions, window, chunk, scale, talk, out, out_head_major, T_, H, Hkv, sinks, softcap, maps, out_f32};
    if (talk) {
        Q6K_REQUIRE(!sinks, "attention with mixed heads takes no sinks");
        Q6K_REQUIRE(dv <= 256 && H <= 64, "attention with mixed heads: value width %d (at most 256), %d heads (at most 64)", dv, H);
        const int warps = H < 8 ? H : 8;
        const size_t smem = ((size_t)H * dk + 2 * H + (size_t)H * 32 + (size_t)H * H) * sizeof(float);
        Q6K_REQUIRE(smem <= 200 * 1024, "attention with mixed heads: %d heads of %d do not fit shared memory", H, dk);
        Q6K_DISPATCH(dtype, {
            if (smem > 48 * 1024) cudaFuncSetAttribute(attention_talk_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            q6k_launch(attention_talk_kernel<T>, dim3(T_), warps * 32, smem, st, a);
        });
        return q6k_check_launch("attention_talk");
    }
    Q6K_REQUIRE(Hkv <= 65535, "attention: %d KV heads exceed the grid limit", Hkv);
    const int G = H / Hkv;
    const int warps = G < 4 ? G : 4;
    const size_t smem = (size_t)warps * dk * sizeof(float);
    Q6K_REQUIRE(smem <= 48 * 1024, "attention: keys of %d do not fit shared memory", dk);
    Q6K_DISPATCH(dtype, q6k_launch(attention_flex_kernel<T>, dim3(T_, Hkv), warps * 32, smem, st, a););
    return q6k_check_launch("attention_flex");
}

Q6K_API int q6k_qkv_pages(const float* qkv, int ld, int splits, long long split_stride, int T_, int Hq, int Hkv, int hd, int vd,
                          const float* q_norm, const float* k_norm, float eps, const float* inv_freq, int rotary_dim, int neighbours,
                          const int* positions, const int* req_of_token, const int* block_table, int max_blocks, int page_size,
                          int num_pages, void* q_out, void* k_pages, void* v_pages, int write_kv, int dtype, int Hv, const float* bias, int v_is_k,
                          int v_norm, cudaStream_t st) {
    if (T_ == 0) return 0;
    if (Hv <= 0) Hv = Hkv;
    Q6K_REQUIRE(!v_is_k || (Hv == Hkv && vd == hd), "qkv_pages: values that are the keys have the keys' heads and width");
    Q6K_REQUIRE(T_ > 0 && Hq > 0 && Hkv > 0 && hd > 0 && vd > 0 && splits >= 1, "qkv_pages: bad sizes T=%d Hq=%d Hkv=%d hd=%d vd=%d", T_, Hq, Hkv, hd, vd);
    Q6K_REQUIRE(!inv_freq || (rotary_dim > 0 && rotary_dim % 2 == 0 && rotary_dim <= hd), "qkv_pages: %d rotating dimensions of a head of %d", rotary_dim, hd);
    Q6K_REQUIRE(!write_kv || (page_size > 0 && max_blocks > 0), "qkv_pages: bad page_size %d / max_blocks %d", page_size, max_blocks);
    const int heads = write_kv ? Hq + Hkv + Hv : Hq;
    Q6K_REQUIRE(heads <= 65535, "qkv_pages: %d heads exceed the grid limit", heads);
    const size_t smem = (size_t)(hd > vd ? hd : vd) * sizeof(float);
    Q6K_REQUIRE(smem <= 48 * 1024, "qkv_pages: heads of %d do not fit shared memory", hd > vd ? hd : vd);
    const auto fills = [](int n, int count) { return n >= 16 && n <= 128 && (n & (n - 1)) == 0 && (long long)n * count % 128 == 0; };
    const size_t align = dtype == Q6K_F32 ? 15 : 7;
    if (fills(hd, Hq) && (!write_kv || (fills(hd, Hkv) && fills(vd, Hv))) && ld % 4 == 0 && split_stride % 4 == 0 && (((uintptr_t)qkv | (uintptr_t)bias) & 15) == 0 &&
        (((uintptr_t)q_out | (uintptr_t)(write_kv ? k_pages : nullptr) | (uintptr_t)(write_kv ? v_pages : nullptr)) & align) == 0) {
        const long long stretches = ((long long)Hq * hd + (write_kv ? (long long)Hkv * hd + (long long)Hv * vd : 0)) / 128;
        if ((stretches + 15) / 16 <= 65535) {
            Q6K_DISPATCH(dtype, q6k_launch(qkv_rows_kernel<T>, dim3(T_, (unsigned)((stretches + 15) / 16)), QR_WARPS * 32, 0, st, qkv, ld, splits, (size_t)split_stride, Hq, Hkv, Hv,
                                           hd, vd, q_norm, k_norm, eps, inv_freq, inv_freq ? rotary_dim : 0, neighbours, positions, req_of_token,
                                           block_table, max_blocks, page_size, num_pages, (T*)q_out, (T*)k_pages, (T*)v_pages, write_kv, bias, v_is_k, v_norm););
            return q6k_check_launch("qkv_pages");
        }
    }
    if (hd <= 256 && vd <= 256 && (heads + 7) / 8 <= 65535) {                 // narrow heads: a warp per head
        Q6K_DISPATCH(dtype, q6k_launch(qkv_pages_warp_kernel<T>, dim3(T_, (heads + 7) / 8), 256, 0, st, qkv, ld, splits, (size_t)split_stride, Hq, Hkv,
                                       hd, vd, q_norm, k_norm, eps, inv_freq, inv_freq ? rotary_dim : 0, neighbours, positions, req_of_token,
                                       block_table, max_blocks, page_size, num_pages, (T*)q_out, (T*)k_pages, (T*)v_pages, heads, bias, v_is_k, v_norm););
        return q6k_check_launch("qkv_pages");
    }
    Q6K_DISPATCH(dtype, q6k_launch(qkv_pages_kernel<T>, dim3(T_, heads), 128, smem, st, qkv, ld, splits, (size_t)split_stride, Hq, Hkv, hd, vd,
                                   q_norm, k_norm, eps, inv_freq, inv_freq ? rotary_dim : 0, neighbours, positions, req_of_token, block_table,
                                   max_blocks, page_size, num_pages, (T*)q_out, (T*)k_pages, (T*)v_pages, Hv, bias, v_is_k, v_norm););
    return q6k_check_launch("qkv_pages");
}

Q6K_API int q6k_latent_prep(const float* x, int ld, const float* xc, int ldc, int T_, int H, int dim, int rd, int rank, const float* cw, float eps,
                            const float* inv_freq, int turn, int neighbours, const int* positions, const int* req_of_token,
                            const int* block_table, int max_blocks, int page_size, void* qn, void* qr, void* pages, int dtype, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && H > 0 && dim > 0 && rd >= 0 && ((rank > 0 && xc) || !pages), "latent_prep: bad sizes T=%d H=%d dim=%d rd=%d rank=%d", T_, H, dim, rd, rank);
    Q6K_REQUIRE(turn >= 0 && turn % 2 == 0 && turn <= rd && (turn == 0 || inv_freq), "latent_prep: %d turning dimensions of %d", turn, rd);
    Q6K_REQUIRE(H + 1 <= 65535 && (!pages || (page_size > 0 && max_blocks > 0 && cw)), "latent_prep: bad grid or pages");
    const size_t smem = (size_t)(rd > 0 ? rd : 1) * sizeof(float), smem_rows = ((size_t)H * rd + turn) * sizeof(float), align = dtype == Q6K_F32 ? 15 : 7;
    if (dim % 4 == 0 && rd % 4 == 0 && ld % 4 == 0 && ((uintptr_t)x & 15) == 0 && (((uintptr_t)qn | (uintptr_t)qr) & align) == 0 && smem_rows <= 40 * 1024 &&
        (long long)H * (dim + rd) <= 0x7fffffffLL) {
        Q6K_DISPATCH(dtype, q6k_launch(latent_rows_kernel<T>, dim3(T_, pages ? 2 : 1), 256, smem_rows, st, x, ld, xc, ldc, H, dim, rd, rank, cw, eps, inv_freq, turn,
                                       neighbours, positions, req_of_token, block_table, max_blocks, page_size, (T*)qn, (T*)qr, (T*)pages, T_););
        return q6k_check_launch("latent_prep");
    }
    Q6K_DISPATCH(dtype, q6k_launch(latent_prep_kernel<T>, dim3(T_, pages ? H + 1 : H), 128, smem, st, x, ld, xc, ldc, H, dim, rd, rank, cw, eps, inv_freq, turn,
                                   neighbours, positions, req_of_token, block_table, max_blocks, page_size, (T*)qn, (T*)qr, (T*)pages, T_););
    return q6k_check_launch("latent_prep");
}

// pages: bfloat16 [pages, page_size, rank + rd]; rows: 64 for every 64 positions (or part of them) that one of the R requests sees; lat: bfloat16 [rows, rank];
// keys: bfloat16 [H, rows, pitch] (columns dim .. dim + rd are written); blocks: int32 [R, wide], wide the most blocks of a request.
Q6K_API int q6k_latent_context(const void* pages, const int* q_start, const int* pos_start, int R, int rows, const int* block_table, int max_blocks, int page_size, void* lat,
                               void* keys, int* blocks, int wide, int rank, int rd, int dim, int pitch, int H, cudaStream_t st) {
    if (rows == 0) return 0;
    Q6K_REQUIRE(rows > 0 && R > 0 && wide > 0 && rank > 0 && rank % 8 == 0 && rd >= 0 && rd % 8 == 0 && dim % 8 == 0 && pitch % 8 == 0 && pitch >= dim + rd && H > 0 &&
                    page_size > 0 && (((uintptr_t)pages | (uintptr_t)lat | (uintptr_t)keys) & 15) == 0,
                "latent_context: bad sizes rows=%d rank=%d rd=%d dim=%d", rows, rank, rd, dim);
    q6k_launch(latent_context_kernel, dim3(rows), 128, 0, st, (const uint4*)pages, q_start, pos_start, R, block_table, max_blocks, page_size, (uint4*)lat, (uint4*)keys, blocks, wide,
               rank / 8, rd / 8, dim / 8, pitch / 8, H);
    return q6k_check_launch("latent_context");
}

Q6K_API int q6k_heads_to_rows(const float* src, void* out, int H, int T_, int n, int dtype, cudaStream_t st) {
    if (T_ == 0) return 0;
    const size_t total = (size_t)H * T_ * n;
    if (n % 4 == 0 && total / 4 < 0x7fffff00 && ((uintptr_t)src & 15) == 0 && ((uintptr_t)out & (dtype == Q6K_F32 ? 15 : 7)) == 0) {
        Q6K_DISPATCH(dtype, q6k_launch(heads_to_rows4_kernel<T>, dim3((unsigned)((total / 4 + 255) / 256)), 256, 0, st, (const float4*)src, (T*)out, H, T_, n / 4, (int)(total / 4)););
        return q6k_check_launch("heads_to_rows");
    }
    Q6K_DISPATCH(dtype, q6k_launch(heads_to_rows_kernel<T>, dim3((unsigned)((total + 255) / 256)), 256, 0, st, src, (T*)out, H, T_, n););
    return q6k_check_launch("heads_to_rows");
}
