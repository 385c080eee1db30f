// The flexible attention for prompt portions on the 5th-generation tensor cores: bfloat16 pages, key rows up to 576 wide, values
// of their own or the leading entries of the key rows, a query given in two parts, causal mask narrowed by a
// window and/or chunks, sinks, a cap on the scores, several maps per head, and every head against every value head for the mixing
// kernel.  The scores, maxima, exponentials, sums and accumulators are FP32 and the weights enter the value product as two
// bfloat16 terms (16 bits of them), as in attention_flex_mma.cu, which keeps the steps of short portions and the shapes this one does not
// take.  Groups of more than 32 query heads, values beyond 512 and whatever else that kernel does not take stay on CUDA cores with
// FP32 weights.
//
// A CTA takes 128 query rows (the G query heads of one key head for 128 / G consecutive tokens of one request) and up to 256
// value columns (FP32 accumulators in tensor memory: a latent of 512 is two CTAs per row tile, which both make the scores: the
// 576-wide score product is half of a CTA's work, and a 512-wide accumulator would leave no tensor memory for scores), and walks
// the keys in tiles of 64.
//   warp 0      producer: the tile's [64 keys x 64 columns] chunks as TMA boxes of a page's rows, in two groups: A is read by the
//               score product only, B is what the value product reads (the value columns of this CTA; with shared values they
//               are key columns as well), so that A's shared memory is refilled while the softmax runs
//   warp 1      one thread issues S(j+1) = Q K^T and O += P(j) V(j): the next tile's scores run under this tile's softmax
//   warps 2-5   softmax, one thread per row: 64 scores from tensor memory, weights back over them (32 columns of rounded weights,
//               32 of what rounding left), O rescaled only when the running maximum grew by more than 2^8
//   warps 6-9   help to bring Q in, then to send for the key tiles (with narrow values two CTAs of an SM hide each other's softmax and loads instead)
// Where the query is wide, four of its 64-wide chunks live in tensor memory (A operand of the score product): that leaves shared
// memory for two key tiles, and those products read half as much of it.
// Tensor memory: O at column 0, S/P buffers at 256 and 320 (two CTAs to an SM: 128 and 192), Q chunks from 384.
// What bounds it: chains, not a unit (tensor pipe 30 % active): a tile is its loads, its scores, its softmax and its value product, each
// 700 to 1,900 clocks, overlapped two tiles deep for the widest rows and four for others; then the boxes of shuffled pages (a TMA
// box of 16 rows takes about 60 clocks).  B200, 2,048 tokens, pages in shuffled order: latent of 512 + 64 under 16 heads 941 us on
// mma.sync, 194 us here; 16 heads on 4 value heads of 128 in chunks of 1,024, mixed, 564 -> 107 us; two maps of 64, 2,465 tokens
// in chunks of 1,024, 326 -> 77 us.
// Every wait is bounded; one that runs out records a code that q6k_attention_flex_tc_status() returns.
#include "umma.cuh"

namespace {

constexpr int FT_ROWS = 128, FT_KEYS = 64, FT_GROUP = 32;   // FT_GROUP: query heads of a key head, at most (as in attention_flex_mma.cu)
constexpr uint32_t FT_CHUNK = FT_KEYS * 128;           // bytes of a [64 keys x 64 columns] chunk
constexpr uint32_t FT_QCHUNK = FT_ROWS * 128;          // bytes of a [128 rows x 64 columns] chunk of Q
constexpr int FT_STAGES = 4;
constexpr float FT_LOG2E = 1.4426950408889634f;

__device__ int g_flex_tc_status = 0;

struct FlexTc {
    const __nv_bfloat16* qa; int da;    // a query row: da entries of one tensor, then db of another
    const __nv_bfloat16* qb; int db;
    int q_head_major;
    int dkb, qt;                        // chunks of a key row; how many of Q's lie in tensor memory
    int nvc, shared_v;                  // value chunks of a CTA; values are the leading columns of the key rows
    int stages, parts;                  // stages of the ring; CTAs that share a row tile's value columns
    int per_tile;                       // CTAs of a row tile: key heads x parts
    int k_head_rows, v_head_rows;       // page rows of a head
    const int* block_table; int max_blocks, page_size, box;
    int oob_k, oob_v;                   // a row beyond the pages: reads zeros
    const int* req_of_token; const int* positions;
    const int* tile_tok0; const int* tile_ntok;
    int window, chunk;
    float scale_log2, softcap;          // scale * log2 e (softcap > 0: the scale alone)
    __nv_bfloat16* out; float* out_f32;
    float* part_o; float* part_ml;
    int out_head_major, T_, H, G, maps, dv, v_heads;       // v_heads > 0: mixed heads
    int nsplit, split_keys;
    const float* sinks;
    uint32_t tmem_cols, s_col;          // columns to allocate; where the first score buffer lies
};

__device__ __forceinline__ int ft_query_head(int kh, int g, int G, int maps) { return maps > 1 ? ((kh / maps) * G + g) * maps + kh % maps : kh * G + g; }

// Whether the phase of the given parity has completed (no wait beyond the instruction's own).
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// 16-byte piece c (0..7) of row r in a chunk of 128-byte rows with the 128-byte swizzle.
__device__ __forceinline__ uint32_t ft_swz(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

__device__ __forceinline__ uint32_t ft_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// CAP: scores pass softcap * tanh(s / softcap).  WARPS4: groups of four warps that bring Q in (the first one is the softmax).
template <bool CAP, int WARPS4>
__global__ void __launch_bounds__(64 + 128 * WARPS4, WARPS4 == 1 ? 2 : 1) attention_flex_tc_kernel(
    const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_k_run,
    const __grid_constant__ CUtensorMap tm_v_run, const FlexTc p) {
    pdl_wait();
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int n_q = p.dkb - p.qt;                               // Q chunks in shared memory: chunks qt .. dkb-1
    const int n_chunks = p.shared_v ? p.dkb : p.dkb + p.nvc;     // chunks of a stage
    const uint32_t q_s = smem_u32(smem), k_s = q_s + n_q * FT_QCHUNK, stage_bytes = n_chunks * FT_CHUNK;
    __shared__ __align__(8) uint64_t bars[4 * FT_STAGES + 7];
    __shared__ uint32_t tmem_slot;
    const uint32_t fullA = smem_u32(&bars[0]), emptyA = fullA + 8 * FT_STAGES, fullB = fullA + 16 * FT_STAGES, emptyB = fullA + 24 * FT_STAGES;
    const uint32_t s_full = fullA + 32 * FT_STAGES, p_full = s_full + 16, pv_done = s_full + 32, q_full = s_full + 48;

    // every (key head, part of the values) of a row tile side by side, the tiles in the order of the list (those with the most keys first)
    const int tile = blockIdx.x / p.per_tile, of_tile = blockIdx.x % p.per_tile, kh = of_tile / p.parts, part = of_tile % p.parts, split = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, G = p.G;
    const int tok0 = p.tile_tok0[tile], ntok = min(p.tile_ntok[tile], FT_ROWS / G);
    const int pos0 = p.positions[tok0], pos_last = pos0 + ntok - 1;
    const int* bt = p.block_table + (size_t)p.req_of_token[tok0] * p.max_blocks;
    // keys [k_begin, k_end) matter to some row
    int k_begin = q6k_first_seen(pos0, p.window, p.chunk), k_end = pos_last + 1;
    if (p.nsplit > 1) {
        k_begin = max(k_begin, split * p.split_keys);
        k_end = min(k_end, (split + 1) * p.split_keys);
    }
    const int j_first = k_begin & ~(FT_KEYS - 1), n = k_end > k_begin ? (k_end - j_first + FT_KEYS - 1) / FT_KEYS : 0;
    const int b0 = p.shared_v ? part * p.nvc : p.dkb;            // first chunk of group B in a stage

    if (tid == 0) {
        for (int s = 0; s < FT_STAGES; ++s) {
            mbar_init(fullA + 8 * s, 1);
            mbar_init(emptyA + 8 * s, 1);
            mbar_init(fullB + 8 * s, 1);
            mbar_init(emptyB + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(s_full + 8 * s, 1);
            mbar_init(p_full + 8 * s, 128);
            mbar_init(pv_done + 8 * s, 1);
        }
        mbar_init(q_full, 128 * WARPS4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_v) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_k_run) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_v_run) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, q_col = 384;
    pdl_launch();                                               // this block holds its tensor memory: a successor may come

    // The producers.  Unit u is group u & 1 of key tile u / 2.  Warp 0 fills the ring, then the warps that are done with Q share
    // the units: a tile of shuffled 16-row pages is up to 36 boxes, and sending for them takes one warp longer than their products.
    // A (stage, group) always has the same warp: only a warp that has waited for every one of a barrier's phases in turn may go by
    // the parity of the next (two warps taking turns on a stage let the second run two phases ahead and overwrite tiles in use).
    auto produce = [&](int first, int last, int who, int warps) {
        auto next = [&](int u) {                                     // the first unit from u on that is this warp's
            while (u < last && (((u >> 1) % p.stages) * 2 + (u & 1)) % warps != who) ++u;
            return u;
        };
        const int ps = p.page_size, boxes = FT_KEYS / p.box, mine = lane & (boxes - 1);
        // the page row of this lane's box of a unit's tile (-1: no key of this block in it)
        auto find = [&](int u) {
            const int j = j_first + (u >> 1) * FT_KEYS + mine * p.box;
            if (j + p.box <= k_begin || j >= k_end) return -1;
            const int page = bt[j / ps];
            return page < 0 ? -1 : page * ps + j % ps;
        };
        int u = next(first), row_next = u < last ? find(u) : -1;
        while (u < last) {
            const int i = u >> 1, grp = u & 1, s = i % p.stages, row = row_next;
            u = next(u + 1);
            if (u < last) row_next = find(u);                        // on its way while this unit's boxes are sent for
            // pages with consecutive numbers lie next to each other and come in as one box of 64 rows
            const int row0 = __shfl_sync(0xffffffffu, row, 0);
            const bool run = boxes > 1 && __all_sync(0xffffffffu, row >= 0 && row == row0 + mine * p.box);
            const uint32_t dst = k_s + s * stage_bytes, fb = (grp ? fullB : fullA) + 8 * s;
            if (!mbar_wait((grp ? emptyB : emptyA) + 8 * s, ((i / p.stages) & 1) ^ 1)) {
                if (lane == 0) atomicExch(&g_flex_tc_status, 1);
                break;
            }
            const int count = grp ? p.nvc : n_chunks - p.nvc;
            if (lane == 0) {
                if (count > 0) mbar_expect_tx(fb, count * FT_CHUNK);
                else mbar_arrive(fb);                                // every key column is a value column of this CTA: nothing in A
            }
            __syncwarp();
            int at[8];                                               // the boxes' page rows, for the one thread that sends for them
#pragma unroll
            for (int b = 0; b < 8; ++b) at[b] = __shfl_sync(0xffffffffu, row, b & (boxes - 1));
            if (elect_one()) {
                for (int e = 0; e < count; ++e) {
                    const int c = grp ? b0 + e : (p.shared_v && e >= b0 ? e + p.nvc : e);
                    const bool is_v = c >= p.dkb;
                    int x = c * 64, head = kh * p.k_head_rows;
                    if (is_v) {                                      // mixed heads have their value heads' columns side by side
                        const int vcol = (part * p.nvc + (c - p.dkb)) * 64, vh = p.v_heads > 0 ? vcol / p.dv : p.maps > 1 ? kh / p.maps : kh;
                        x = p.v_heads > 0 ? vcol % p.dv : vcol;
                        head = vh * p.v_head_rows;
                    }
                    const uint32_t to = dst + c * FT_CHUNK;
                    if (run) {
                        tma_load_2d(to, is_v ? &tm_v_run : &tm_k_run, x, head + row0, fb);
                    } else {
                        const CUtensorMap* map = is_v ? &tm_v : &tm_k;
                        const int oob = is_v ? p.oob_v : p.oob_k;
#pragma unroll
                        for (int b = 0; b < 8; ++b)
                            if (b < boxes) tma_load_2d(to + b * p.box * 128, map, x, at[b] >= 0 ? head + at[b] : oob, fb);
                    }
                }
            }
        }
    };
    const int filled = WARPS4 == 1 ? 2 * n : 2 * min(n, p.stages);   // units of warp 0 alone
    if (warp == 0) {
        produce(0, filled, 0, 1);
        if (WARPS4 > 1) produce(filled, 2 * n, 0, 5);
    } else if (warp == 1) {
        if (n > 0 && elect_one()) {
            const uint32_t idesc_s = umma_idesc_m128(FT_KEYS, false), idesc_o = umma_idesc_m128(p.nvc * 64, true);
            bool ok = mbar_wait(q_full, 0);
            if (!ok) atomicExch(&g_flex_tc_status, 2);
            tc_fence_after();
            auto wait = [&](uint32_t bar, uint32_t parity, int code) {
                if (ok && !mbar_wait(bar, parity)) {
                    atomicExch(&g_flex_tc_status, code);
                    ok = false;
                }
            };
            auto scores = [&](int i, int grp) {                      // one group's share of S(i)
                const int s = i % p.stages;
                const uint32_t src = k_s + s * stage_bytes, d = tmem + p.s_col + (i & 1) * FT_KEYS;
                tc_fence_after();
                const int count = grp ? p.nvc : p.shared_v ? p.dkb - p.nvc : p.dkb;
                uint32_t acc = grp && p.dkb > p.nvc;
                for (int e = 0; e < count; ++e) {
                    const int c = grp ? b0 + e : (p.shared_v && e >= b0 ? e + p.nvc : e);
                    const uint64_t db = umma_desc_k(src + c * FT_CHUNK);
                    if (c < p.qt) {
#pragma unroll
                        for (int k = 0; k < 4; ++k, acc = 1) umma_ts(d, tmem + q_col + c * 32 + k * 8, db + 2 * k, idesc_s, acc);
                    } else {
                        const uint64_t da = umma_desc_k(q_s + (c - p.qt) * FT_QCHUNK);
#pragma unroll
                        for (int k = 0; k < 4; ++k, acc = 1) umma_ss(d, da + 2 * k, db + 2 * k, idesc_s, acc);
                    }
                }
                if (!grp) umma_commit(emptyA + 8 * s);
                if (grp || !p.shared_v) umma_commit(s_full + 8 * (i & 1));
            };
            auto values = [&](int i) {                               // O += P(i) V(i)
                const int s = i % p.stages;
                tc_fence_after();
                const uint32_t pa = tmem + p.s_col + (i & 1) * FT_KEYS, v = k_s + s * stage_bytes + b0 * FT_CHUNK;
#pragma unroll
                for (int t = 0; t < 2; ++t)                       // the rounded weights, then what rounding left
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_ts(tmem, pa + t * 32 + k * 8, umma_desc_mn(v + k * 2048, FT_CHUNK), idesc_o, (i | t | k) != 0);
                umma_commit(emptyB + 8 * s);
                umma_commit(pv_done + 8 * (i & 1));
            };
            const int groups = p.shared_v ? 2 : 1;
            for (int grp = 0; grp < groups && ok; ++grp) {
                wait((grp ? fullB : fullA), 0, 3);
                if (ok) scores(0, grp);
            }
            // Whichever is ready first: the next part of S(i + 1) (its chunks have landed) or O += P(i) V(i) (the weights are out).
            // With a fixed order each waits for the other's loads: 4,700 clocks a tile of the widest latent.  A buffer of scores is
            // free for S(i + 1) since P(i - 1), which lay there, was multiplied before this tile's turn.
            for (int i = 0; i < n && ok; ++i) {
                int grp = i + 1 < n ? 0 : groups;
                bool pv = false, v_in = p.shared_v != 0;
                const int s1 = (i + 1) % p.stages, ph1 = ((i + 1) / p.stages) & 1;
                long long t0 = 0;
                for (uint32_t spin = 0; ok && (grp < groups || !pv); ++spin) {
                    if (grp < groups && mbar_test((grp ? fullB : fullA) + 8 * s1, ph1)) {
                        scores(i + 1, grp++);
                        continue;
                    }
                    if (!pv && !v_in) v_in = mbar_test(fullB + 8 * (i % p.stages), (i / p.stages) & 1);
                    if (!pv && v_in && mbar_test(p_full + 8 * (i & 1), (i >> 1) & 1)) {
                        values(i);
                        pv = true;
                        continue;
                    }
                    if ((spin & 255u) == 255u) {
                        const long long now = clock64();
                        if (t0 == 0) t0 = now;
                        else if (now - t0 > WAIT_LIMIT_CYCLES) {
                            atomicExch(&g_flex_tc_status, 4);
                            ok = false;
                        }
                    }
                }
            }
        }
    } else {
        // A barrier's parity tells a phase from the one before and the one after it only, and these warps do not wait for every value
        // product.  So the products take turns on two barriers: when a row has seen the scores of tile i, the product of tile i - 2
        // is done (the scores were issued behind it), and no product beyond i - 1 can end before the row's weights of tile i are
        // out.  Product i - 1 is thus the last phase of its barrier that ended or the one at hand, whenever the row comes to ask.
        // With one barrier product i - 1 could be taken for i - 3, and a row that came late to ask for i - 2 would wait for i.
        // ---- Q (zeros in rows without a token)
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const int ht = tid - 64;
        auto fetch_q = [&](int c0, int count) {                     // chunks c0 .. c0 + count - 1 into the first chunks of Q's shared memory
            for (int i = ht; i < FT_ROWS * count * 8; i += 128 * WARPS4) {
                const int c = i & 7, r = (i >> 3) & (FT_ROWS - 1), ch = i >> 10, tk = r / G, d = (c0 + ch) * 64 + c * 8;
                const int h = ft_query_head(kh, r - tk * G, G, p.maps), t = tok0 + tk;
                const size_t row_of = p.q_head_major ? (size_t)h * p.T_ + t : (size_t)t * p.H + h;
                const __nv_bfloat16* src = d < p.da ? p.qa + row_of * p.da + d : p.qb + row_of * p.db + (d - p.da);
                const bool have = tk < ntok && d < p.da + p.db;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(q_s + ch * FT_QCHUNK + ft_swz(r, c)), "l"(have ? src : (const __nv_bfloat16*)p.positions),
                             "r"(have ? 16 : 0)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        };
        // the chunks for tensor memory pass through the shared memory of the others
        for (int c0 = 0; c0 < p.qt; c0 += n_q) {
            const int count = min(n_q, p.qt - c0);
            fetch_q(c0, count);
            asm volatile("bar.sync 1, %0;" ::"n"(128 * WARPS4) : "memory");
            for (int c = (warp - 2) >> 2; c < count; c += WARPS4) {
                uint32_t v[32];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint4 x = *reinterpret_cast<const uint4*>(smem + c * FT_QCHUNK + ft_swz(row, e));
                    v[4 * e] = x.x, v[4 * e + 1] = x.y, v[4 * e + 2] = x.z, v[4 * e + 3] = x.w;
                }
                tmem_st32(tmem + lane_base + q_col + (c0 + c) * 32, v);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(128 * WARPS4) : "memory");
        }
        tmem_st_wait();
        fetch_q(p.qt, n_q);
        const int tk = row / G, h = ft_query_head(kh, row % G, G, p.maps), t = tok0 + tk;
        const bool valid = tk < ntok;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        mbar_arrive(q_full);
        if (warp >= 6) {
            produce(filled, 2 * n, warp - 5, 5);
        } else {
            // ---- softmax, one thread per row
            const int pos = pos0 + tk, lim_hi = valid ? pos : -1, lim_lo = valid ? max(k_begin, q6k_first_seen(pos, p.window, p.chunk)) : 0;
            const int all_lo = max(k_begin, q6k_first_seen(pos_last, p.window, p.chunk));
            const float cap2 = p.softcap * FT_LOG2E, inv_cap = CAP ? p.scale_log2 / p.softcap : 0.0f;
            const float mult = CAP ? 1.0f : p.scale_log2;           // what a value in v[] is multiplied by to be a base-2 exponent
            float m = -INFINITY, l = 0.0f;                          // the reference point (base 2) and the sum of weights
            bool ok = true;
            for (int i = 0; i < n; ++i) {
                const int j0 = j_first + i * FT_KEYS, st = i % p.stages;
                const uint32_t s_addr = tmem + lane_base + p.s_col + (i & 1) * FT_KEYS;
                if (!mbar_wait(s_full + 8 * (i & 1), (i >> 1) & 1)) {
                    if (lane == 0) atomicExch(&g_flex_tc_status, 6);
                    ok = false;
                    break;
                }
                tc_fence_after();
                float v[FT_KEYS];
                tmem_ld32_issue(s_addr, v);
                tmem_ld32_issue(s_addr + 32, v + 32);
                tmem_ld_wait();
                if (CAP) {
                    // cap * tanh(s / cap).  Scores far below the cap (the usual case) take the odd Taylor series up to y^9, whose
                    // error below |y| = 1/4 is 1e-8 of the value, on the FMA pipe; else 1 - 2 / (1 + e^2y) on the special-function
                    // unit, which the weights' exponentials already keep busy.
                    float most = 0.0f;
#pragma unroll
                    for (int x = 0; x < FT_KEYS; ++x) {
                        v[x] *= inv_cap;
                        most = fmaxf(most, fabsf(v[x]));
                    }
                    if (__any_sync(0xffffffffu, !(most < 0.25f))) {
#pragma unroll
                        for (int x = 0; x < FT_KEYS; ++x) v[x] = cap2 * (1.0f - __fdividef(2.0f, 1.0f + ex2_approx(v[x] * (2.0f * FT_LOG2E))));
                    } else {
#pragma unroll
                        for (int x = 0; x < FT_KEYS; ++x) {
                            const float y = v[x], z = y * y;
                            v[x] = cap2 * fmaf(y * z, fmaf(z, fmaf(z, fmaf(z, 62.0f / 2835.0f, -17.0f / 315.0f), 2.0f / 15.0f), -1.0f / 3.0f), y);
                        }
                    }
                }
                if (!(j0 + FT_KEYS - 1 <= pos0 && j0 >= all_lo && j0 + FT_KEYS <= k_end)) {
                    // the keys of this tile that the row sees, as offsets into it
                    const int lo = lim_lo - j0, hi = min(lim_hi, k_end - 1) - j0;
#pragma unroll
                    for (int x = 0; x < FT_KEYS; ++x) v[x] = (x >= lo && x <= hi) ? v[x] : -INFINITY;
                }
                float mx[8];
#pragma unroll
                for (int x = 0; x < 8; ++x) mx[x] = fmaxf(v[x], v[x + 8]);
#pragma unroll
                for (int y = 16; y < FT_KEYS; y += 8)
#pragma unroll
                    for (int x = 0; x < 8; ++x) mx[x] = fmaxf(mx[x], v[y + x]);
#pragma unroll
                for (int w = 4; w >= 1; w >>= 1)
#pragma unroll
                    for (int x = 0; x < w; ++x) mx[x] = fmaxf(mx[x], mx[x + w]);
                const float top = mx[0] * mult;                   // the scale is positive
                float ref = m, corr = 1.0f;
                if (top > m + 8.0f || m == -INFINITY) {
                    ref = fmaxf(m, top);
                    corr = m == -INFINITY ? 1.0f : ex2_approx(m - ref);
                }
                if (i > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
                    if (!mbar_wait(pv_done + 8 * ((i - 1) & 1), ((i - 1) >> 1) & 1)) {
                        if (lane == 0) atomicExch(&g_flex_tc_status, 7);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < p.nvc * 2; ++c) {
                        float o[32];
                        tmem_ld32_issue(tmem + lane_base + c * 32, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int x = 0; x < 32; ++x) o[x] *= corr;
                        tmem_st32(tmem + lane_base + c * 32, reinterpret_cast<uint32_t*>(o));
                    }
                }
                const float neg_ref = ref == -INFINITY ? 0.0f : -ref;
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                uint32_t hi[32], lo[32];
#pragma unroll
                for (int x = 0; x < FT_KEYS; x += 2) {
                    const float e0 = ex2_approx(fmaf(v[x], mult, neg_ref)), e1 = ex2_approx(fmaf(v[x + 1], mult, neg_ref));
                    sum[(x >> 1) & 3] += e0 + e1;
                    const uint32_t w = ft_pack(e0, e1);
                    hi[x >> 1] = w;
                    lo[x >> 1] = ft_pack(e0 - __uint_as_float(w << 16), e1 - __uint_as_float(w & 0xffff0000u));
                }
                tmem_st32(s_addr, hi);
                tmem_st32(s_addr + 32, lo);
                l = l * corr + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
                m = ref;
                if (j0 + FT_KEYS > k_end) {
                    // the last page came in whole: value rows past the last key are cleared (0 * what was never written)
                    if (!p.shared_v && !mbar_wait(fullB + 8 * st, (i / p.stages) & 1)) {
                        if (lane == 0) atomicExch(&g_flex_tc_status, 8);
                        ok = false;
                        break;
                    }
                    const uint32_t base = (k_s - q_s) + st * stage_bytes + b0 * FT_CHUNK;
                    const int r0 = k_end - j0, rows = FT_KEYS - r0;
                    for (int e = ht; e < rows * p.nvc * 8; e += 128) {
                        const int c = e / (rows * 8), r = r0 + (e / 8) % rows;
                        *reinterpret_cast<uint4*>(smem + base + c * FT_CHUNK + r * 128 + (e & 7) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(p_full + 8 * (i & 1));
            }
            if (ok && n > 0) {
                if (!mbar_wait(pv_done + 8 * ((n - 1) & 1), ((n - 1) >> 1) & 1)) {      // the products before it are done when it is
                    if (lane == 0) atomicExch(&g_flex_tc_status, 9);
                    ok = false;
                }
                tc_fence_after();
            }
            // ---- results: every lane takes part in the loads from tensor memory, rows of real tokens store
            if (ok) {
                const int col0 = part * p.nvc * 64;
                float mulo = l > 0.0f ? 1.0f / l : 0.0f;
                float* f32 = nullptr;
                __nv_bfloat16* b16 = nullptr;
                const size_t row_of = p.out_head_major ? (size_t)h * p.T_ + t : (size_t)t * p.H + h;
                if (p.v_heads > 0) {
                    f32 = p.part_o + ((size_t)t * p.H + h) * p.v_heads * p.dv + col0;
                } else if (p.nsplit > 1) {
                    const size_t prow = ((size_t)split * p.T_ + t) * p.H + h;
                    f32 = p.part_o + prow * p.dv + col0;
                    if (part == 0 && valid) {
                        p.part_ml[prow * 2] = m * 0.6931471805599453f;
                        p.part_ml[prow * 2 + 1] = l;
                    }
                    mulo = 1.0f;
                } else {
                    if (p.sinks) {                                // the sink counts once in the denominator
                        const float sk = valid ? p.sinks[h] * FT_LOG2E : 0.0f, top = fmaxf(m, sk);
                        const float c = m == -INFINITY ? 0.0f : exp2f(m - top), den = l * c + exp2f(sk - top);
                        mulo = den > 0.0f ? c / den : 0.0f;
                    }
                    if (p.out_f32) f32 = p.out_f32 + row_of * p.dv + col0;
                    else b16 = p.out + row_of * p.dv + col0;
                }
                // through shared memory (no product reads it any more), 32 columns of the warp's 32 rows at a time, so that rows
                // leave in whole 128-byte lines (a thread storing its own row 16 bytes at a time took 10,000 clocks for 256 FP32 columns)
                const bool store = valid && (n > 0 || p.nsplit == 1);
                const unsigned stores = __ballot_sync(0xffffffffu, store);
                float* stage = reinterpret_cast<float*>(smem) + (warp - 2) * 32 * 36;
#pragma unroll 1
                for (int c = 0; c < p.nvc * 2; ++c) {
                    float o[32];
                    if (n > 0) {
                        tmem_ld32_issue(tmem + lane_base + c * 32, o);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int x = 0; x < 32; ++x) o[x] = 0.0f;
                    }
#pragma unroll
                    for (int x = 0; x < 32; x += 4)
                        *reinterpret_cast<float4*>(stage + lane * 36 + x) = make_float4(o[x] * mulo, o[x + 1] * mulo, o[x + 2] * mulo, o[x + 3] * mulo);
                    __syncwarp();
#pragma unroll
                    for (int r0 = 0; r0 < 32; r0 += 4) {
                        const int r = r0 + (lane >> 3), x = (lane & 7) * 4;
                        const unsigned long long at = __shfl_sync(0xffffffffu, f32 ? (unsigned long long)f32 : (unsigned long long)b16, r);
                        const float4 y = *reinterpret_cast<const float4*>(stage + r * 36 + x);
                        if ((stores >> r) & 1) {
                            if (f32) *reinterpret_cast<float4*>((float*)at + c * 32 + x) = y;
                            else *reinterpret_cast<uint2*>((__nv_bfloat16*)at + c * 32 + x) = make_uint2(ft_pack(y.x, y.y), ft_pack(y.z, y.w));
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
    }
}

// What a launch needs for these sizes; false: not taken.
struct FlexTcPlan {
    int dkb, qt, parts, nvc, stages;
    bool two;                            // two CTAs to an SM
    uint32_t cols, s_col;
    size_t smem;
};

bool flex_tc_plan(int H, int Hkv, int dk, int dv, int da, int db, int v_heads, bool shared_v, int page_size, FlexTcPlan* o) {
    if (Hkv <= 0 || H <= 0 || H % Hkv || H / Hkv > FT_GROUP || dv > 512) return false;
    if (page_size < 8 || (page_size < FT_KEYS ? FT_KEYS % page_size : page_size % FT_KEYS)) return false;
    const int total = v_heads > 0 ? v_heads * dv : dv;
    if (dk % 8 || da % 8 || db % 8 || dv <= 0 || dv % 64 || total > 2048) return false;
    o->parts = (total + 255) / 256;
    if (total % (o->parts * 64)) return false;
    o->nvc = total / o->parts / 64;
    o->dkb = (dk + 63) / 64;
    const size_t chunks = shared_v ? o->dkb : o->dkb + o->nvc, stage = chunks * FT_CHUNK;
    if (shared_v && dv > dk) return false;
    const size_t most = 225 * 1024, half = 111 * 1024;      // without the alignment, the static and the reserved part
    o->qt = 0;
    // narrow values: half of an SM's tensor memory and shared memory, so that two CTAs hide each other's softmax
    o->two = o->nvc <= 2 && o->dkb * FT_QCHUNK + 2 * stage <= half;
    if (!o->two && o->dkb * FT_QCHUNK + 2 * stage > most) {
        if (o->dkb <= 4) return false;   // some of Q stays in shared memory: what goes to tensor memory passes through its place
        o->qt = 4;
    }
    const size_t q_bytes = (size_t)(o->dkb - o->qt) * FT_QCHUNK, room = o->two ? half : most;
    if (q_bytes + 2 * stage > room) return false;
    o->stages = (int)((room - q_bytes) / stage);
    if (o->stages > FT_STAGES) o->stages = FT_STAGES;
    o->cols = o->two ? 256 : 512, o->s_col = o->two ? 128 : 256;
    o->smem = q_bytes + o->stages * stage + 1024;
    return true;
}

// A pool of pages as a matrix of rows, cut into boxes of [box_rows x 64].
int flex_tc_map(CUtensorMap* m, const void* base, long long rows, int cols, int ld, int box_rows) {
    return make_bf16_map(m, base, rows, cols, ld, box_rows, true, "attention_flex_tc");
}

}  // namespace

Q6K_API int q6k_attention_flex_tc_status() {
    int v = -1;
    if (cudaMemcpyFromSymbol(&v, g_flex_tc_status, sizeof v) != cudaSuccess) return -1;
    return v;
}

// CTAs that share a row tile's values for these sizes, or 0 where the kernel does not take them.  v_heads: value heads every head
// meets (mixed heads), else 0.
Q6K_API int q6k_attention_flex_tc_parts(int H, int Hkv, int da, int db, int dv, int v_heads, int shared_v, int page_size) {
    FlexTcPlan o;
    return flex_tc_plan(H, Hkv, da + db, dv, da, db, v_heads, shared_v != 0, page_size, &o) ? o.parts : 0;
}

// Tokens of one request a row tile holds.
Q6K_API int q6k_attention_flex_tc_tile_tokens(int H, int Hkv) { return Hkv > 0 && H % Hkv == 0 && H / Hkv <= FT_GROUP ? FT_ROWS / (H / Hkv) : 0; }

// Arguments as q6k_attention_flex_tc's (attention_flex_mma.cu).  talk != 0: mixed heads; the result is part_o FP32
// [T, H, Hkv, dv], for the mixing kernel.  nsplit > 1: part_o [nsplit, T, H, dv] unnormalised and part_ml [nsplit, T, H, 2], for
// the merging kernel.
int q6k_attention_flex_tc_launch(const void* qa, int da, const void* qb, int db, int q_head_major, const void* k_pages, int k_ld, const void* v_pages,
                                 int v_ld, int dv, int num_pages, const int* block_table, int max_blocks, int page_size, const int* req_of_token,
                                 const int* positions, const int* tile_tok0, const int* tile_ntok, int n_tiles, int window, int chunk, float scale, void* out,
                                 int out_head_major, int T_, int H, int Hkv, int nsplit, int split_keys, float* part_o, float* part_ml, int talk,
                                 const float* sinks, float softcap, int maps, float* out_f32, cudaStream_t st) {
    const bool shared_v = v_pages == k_pages;
    FlexTcPlan pl;
    Q6K_REQUIRE(flex_tc_plan(H, Hkv, da + db, dv, da, db, talk ? Hkv : 0, shared_v, page_size, &pl), "attention_flex_tc: shapes H=%d Hkv=%d dk=%d dv=%d not taken", H,
                Hkv, da + db, dv);
    const int Hv = maps > 1 ? Hkv / maps : Hkv;
    const long long k_rows = (long long)Hkv * num_pages * page_size, v_rows = (long long)Hv * num_pages * page_size;
    Q6K_REQUIRE(k_rows < (1LL << 31) && (long long)n_tiles * Hkv * pl.parts < (1LL << 31) && nsplit <= 65535 && ((uintptr_t)k_pages & 15) == 0 && ((uintptr_t)v_pages & 15) == 0 && k_ld % 8 == 0 &&
                    v_ld % 8 == 0 && ((uintptr_t)qa & 15) == 0 && ((uintptr_t)qb & 15) == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)part_o & 15) == 0 && scale > 0.0f,
                "attention_flex_tc: too many rows or operands not 16-byte aligned");
    const int box = page_size < FT_KEYS ? page_size : FT_KEYS;
    CUtensorMap tk, tv, tkr, tvr;
    if (int rc = flex_tc_map(&tk, k_pages, k_rows, da + db, k_ld, box)) return rc;
    if (int rc = flex_tc_map(&tkr, k_pages, k_rows, da + db, k_ld, FT_KEYS)) return rc;
    tv = tk, tvr = tkr;
    if (!shared_v) {
        if (int rc = flex_tc_map(&tv, v_pages, v_rows, dv, v_ld, box)) return rc;
        if (int rc = flex_tc_map(&tvr, v_pages, v_rows, dv, v_ld, FT_KEYS)) return rc;
    }
    FlexTc p{};
    p.qa = (const __nv_bfloat16*)qa, p.da = da, p.qb = (const __nv_bfloat16*)qb, p.db = db, p.q_head_major = q_head_major;
    p.dkb = pl.dkb, p.qt = pl.qt, p.nvc = pl.nvc, p.shared_v = shared_v, p.stages = pl.stages, p.parts = pl.parts, p.per_tile = Hkv * pl.parts;
    p.k_head_rows = p.v_head_rows = num_pages * page_size, p.oob_k = (int)k_rows, p.oob_v = (int)v_rows;
    p.block_table = block_table, p.max_blocks = max_blocks, p.page_size = page_size, p.box = box;
    p.req_of_token = req_of_token, p.positions = positions, p.tile_tok0 = tile_tok0, p.tile_ntok = tile_ntok;
    p.window = window, p.chunk = chunk, p.scale_log2 = softcap > 0.0f ? scale : scale * FT_LOG2E, p.softcap = softcap;
    p.out = (__nv_bfloat16*)out, p.out_f32 = out_f32, p.part_o = part_o, p.part_ml = part_ml;
    p.out_head_major = out_head_major, p.T_ = T_, p.H = H, p.G = H / Hkv, p.maps = maps, p.dv = dv, p.v_heads = talk ? Hkv : 0;
    p.nsplit = nsplit, p.split_keys = split_keys, p.sinks = sinks, p.tmem_cols = pl.cols, p.s_col = pl.s_col;
    auto* kernel = pl.two ? (softcap > 0.0f ? attention_flex_tc_kernel<true, 1> : attention_flex_tc_kernel<false, 1>)
                          : (softcap > 0.0f ? attention_flex_tc_kernel<true, 2> : attention_flex_tc_kernel<false, 2>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem) != cudaSuccess) return q6k_check_launch("attention_flex_tc: shared memory attribute");
    q6k_launch(kernel, dim3(n_tiles * Hkv * pl.parts, nsplit), pl.two ? 192 : 320, pl.smem, st, tk, tv, tkr, tvr, p);
    return q6k_check_launch("attention_flex_tc");
}
