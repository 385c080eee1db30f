// The recurrent half of a selective state-space mixer (Mamba, first form), for any mix of prompt
// portions and single tokens, with the state of every request in its slot:
//
//   conv:  u[t, c] = silu(bias[c] + sum_k w[c, k] * x[t - (taps-1-k), c])      inputs before the portion come from the slot's
//                                                                              tail of the last taps-1 inputs, zeros at the start
//   scan:  dt = softplus(dt_raw[t, c] + dt_bias[c])
//          S[c, n] <- exp(dt * A[c, n]) * S[c, n] + dt * u[t, c] * B[t, n]
//          y[t, c] = (sum_n S[c, n] * C[t, n] + D[c] * u[t, c]) * silu(z[t, c])
//
// The state S, dt, the decay and every sum of the recurrence are FP32; u leaves the convolution in
// the operand dtype (it is the next product's input) and enters the recurrence as stored.  A group of
// L lanes owns a channel, each lane eight states side by side (B and C come to them 16 bytes at a time); the sum over n is
// a lane's own and then a butterfly over those lanes, so its order depends on nothing but N.  Tokens of a request are walked in order, so a prompt
// cut anywhere leaves the same state as the whole prompt.
//
// A long portion is walked in segments of `seg_len` tokens by different blocks (the recurrence is linear in S, so a
// segment's effect on the state is a pair: the state it builds from zero and the sum of dt over it, from which follows
// the decay it applies to what came before).  A first launch (MODE 1) leaves that pair per segment; a small kernel walks a
// request's pairs in order and puts the state that each segment starts from in its state's place; the last launch (MODE 2)
// runs as the single launch (MODE 0) does.  This only regroups the sums of the recurrence: the result differs by rounding.
// 2,048 tokens, 4,096 channels of 16 states: the launches were 545 us when each segment folded all of its predecessors
// itself (254 MB of pairs) and a lane read its states' B and C one by one.  Now 135 + 20 + 216 us.  What bounds it: issue slots,
// about 16 a token and state in either launch, and the special-function unit (an exponential each).
#include "short_conv.cuh"

#include <type_traits>

namespace {

constexpr int MAX_TAPS = 16;
constexpr int SCAN_TILE = 32;      // tokens whose inputs are staged in shared memory at a time
constexpr int MAX_PER_LANE = 8;    // states per lane

__device__ __forceinline__ float silu_f(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.0f ? v : log1pf(expf(v)); }
// exp(x) - 1 for x <= 0 with a relative error near 1e-7: down to -1/4 the Taylor series in x (its truncation is below
// x^7 / 40320), beyond that expf(x) - 1, where the exponential's rounding is small beside its distance from 1.
// FAST (bfloat16 operands, whose own rounding is four orders of magnitude above it): the hardware exponential beyond -1/4
// (a few units in the last place of the exponential) and two terms fewer in the series.
template <bool FAST>
__device__ __forceinline__ float decay_minus_one(float x) {
    float p = FAST ? fmaf(x, 1.0f / 120.0f, 1.0f / 24.0f) : fmaf(x, fmaf(x, fmaf(x, 1.0f / 5040.0f, 1.0f / 720.0f), 1.0f / 120.0f), 1.0f / 24.0f);
    p = fmaf(x, p, 1.0f / 6.0f);
    p = fmaf(x, p, 0.5f);
    p = fmaf(x, p, 1.0f);
    const float near = x * p, far = (FAST ? __expf(x) : expf(x)) - 1.0f;      // both, so that no warp splits over it
    return x > -0.25f ? near : far;
}

// grid (T, ceil(C / 256)); x: FP32 [T, ldx] (first C columns); tail: FP32 [slots, taps-1, C].
template <typename T>
__global__ void __launch_bounds__(256) conv_silu_kernel(const float* x, int ldx, const float* w, const float* bias, const float* tail,
                                                        const int* req_of_token, const int* q_start, const int* slot_ids, T* out,
                                                        int C, int taps) {
    pdl_enter();
    const int t = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int r = req_of_token[t], first = q_start[r], i = t - first;
    const float* old = tail + (size_t)slot_ids[r] * (taps - 1) * C;
    float acc = bias[c];
    for (int k = 0; k < taps; ++k) {
        const int j = i - (taps - 1 - k);                        // index within the portion; negative: before it
        const float v = j >= 0 ? x[(size_t)(first + j) * ldx + c] : old[(size_t)(taps - 1 + j) * C + c];
        acc = fmaf(w[(size_t)c * taps + k], v, acc);
    }
    out[(size_t)t * C + c] = from_f32<T>(silu_f(acc));
}

// The state every segment of request r starts from, in place of the state it builds from zero.  grid (R * blocks), blocks = ceil(C N / 256).
__global__ void __launch_bounds__(256) scan_fold_kernel(float* ws, const float* A, const float* state, const int* q_start, const int* slot_ids,
                                                        const int* seg_base, int seg_len, int seg_slots, int C, int N) {
    pdl_enter();
    const size_t CN = (size_t)C * N;
    const unsigned blocks = (unsigned)((CN + 255) / 256);
    const int r = blockIdx.x / blocks, n_req = q_start[r + 1] - q_start[r];
    const size_t i = (size_t)(blockIdx.x % blocks) * 256 + threadIdx.x;
    if (i >= CN) return;
    const float a = A[i];
    float S = state[(size_t)slot_ids[r] * CN + i];
    float* at = ws + (size_t)seg_base[r] * CN + i;
    const float* sums = ws + (size_t)seg_slots * CN + (size_t)seg_base[r] * C + i / N;
    const int segments = (n_req + seg_len - 1) / seg_len;
#pragma unroll 4
    for (int q = 0; q < segments; ++q, at += CN, sums += C) {
        const bool more = q + 1 < segments;                                     // the last segment leaves no pair
        const float built = more ? *at : 0.0f, dts = more ? *sums : 0.0f;
        *at = S;
        S = fmaf(expm1f(dts * a), S, S) + built;
    }
}

// The last taps - 1 inputs of a channel's convolution: the end of a portion of n tokens, preceded by what is left of the old tail.
__device__ __forceinline__ void scan_move_tail(float* tl, const float* x, int ldx, int C, int n, int taps) {
    float keep[MAX_TAPS];
#pragma unroll
    for (int j = 0; j < MAX_TAPS; ++j)
        if (j < taps - 1) {
            const int src = n - (taps - 1) + j;              // index within the portion
            keep[j] = src >= 0 ? x[(size_t)src * ldx] : tl[(size_t)(j + n) * C];
        }
#pragma unroll
    for (int j = 0; j < MAX_TAPS; ++j)
        if (j < taps - 1) tl[(size_t)j * C] = keep[j];
}

// grid (R, ceil(C / (128 / L)), segments), 128 threads; dynamic shared memory SCAN_TILE * (16 L + 4 * 128 / L) floats.
// ws (MODE 1, 2): per segment slot q = seg_base[r] + segment, [q][C][N] the state built from zero (MODE 2: the state to start
// from), then [q][C] the sum of dt.
template <typename T, int MODE>
__global__ void __launch_bounds__(128) selective_scan_kernel(const T* u, const float* dt_raw, const float* dt_bias, const float* proj, int ldp,
                                                             int b_col, int c_col, const float* A, const float* Dskip, const float* xz,
                                                             int ldx, int z_col, float* state, float* tail, const int* q_start,
                                                             const int* slot_ids, T* out, int C, int N, int L, int taps, float* ws,
                                                             const int* seg_base, int seg_len, int seg_slots) {
    pdl_enter();
    extern __shared__ __align__(16) float bc[];    // [SCAN_TILE][8 L] of B, the same of C, then four [SCAN_TILE][channels of the block]
    const int r = blockIdx.x, seg = MODE == 0 ? 0 : blockIdx.z;
    const int per_block = blockDim.x / L;
    const int c = blockIdx.y * per_block + threadIdx.x / L, sub = threadIdx.x % L;
    const bool live = c < C;
    const int first_req = q_start[r], n_req = q_start[r + 1] - first_req, slot = slot_ids[r];
    const int t_begin = MODE == 0 ? 0 : seg * seg_len;
    if (MODE != 0 && t_begin >= n_req) return;
    const int n_tok = MODE == 0 ? n_req : min(n_req - t_begin, seg_len);       // this block's tokens
    const int first = first_req + t_begin;
    const bool last_segment = t_begin + n_tok == n_req;
    if (MODE == 1 && last_segment) return;     // no later segment follows this one
    const size_t CN = (size_t)C * N, own = ((size_t)(live ? c : 0)) * N;
    const int n0 = sub * MAX_PER_LANE, NP = L * MAX_PER_LANE;                  // this lane's first state; states with padding
    float S[MAX_PER_LANE], a[MAX_PER_LANE], dt_sum = 0.0f;
    float* Sg = state + (size_t)slot * CN + own;
    float* seg_state = MODE == 0 ? Sg : ws + (size_t)(seg_base[r] + seg) * CN + own;
#pragma unroll
    for (int k = 0; k < MAX_PER_LANE; ++k) {
        const bool has = live && n0 + k < N;   // a state beyond N has A = B = C = 0 and stays zero
        a[k] = has ? A[(size_t)c * N + n0 + k] : 0.0f;
        S[k] = has && MODE != 1 ? seg_state[n0 + k] : 0.0f;
    }
    // Per tile of SCAN_TILE tokens the block first makes, once per (token, channel) and with coalesced loads, what the
    // recurrence needs of them: dt = softplus(dt_raw + bias), dt u, the gate silu(z) and the skip D u; then B and C.
    float* s_dt = bc + 2 * SCAN_TILE * NP;         // [SCAN_TILE][per_block]
    float* s_du = s_dt + SCAN_TILE * per_block;
    float* s_gate = s_du + SCAN_TILE * per_block;
    float* s_skip = s_gate + SCAN_TILE * per_block;
    const int c0 = blockIdx.y * per_block, cc = threadIdx.x / L;
    for (int t0 = 0; t0 < n_tok; t0 += SCAN_TILE) {
        const int nt = min(SCAN_TILE, n_tok - t0);
        __syncthreads();
        for (int i = threadIdx.x; i < nt * NP; i += blockDim.x) {
            const int tt = i / NP, n = i % NP;
            const float* pr = proj + (size_t)(first + t0 + tt) * ldp;
            bc[i] = n < N ? pr[b_col + n] : 0.0f;
            bc[SCAN_TILE * NP + i] = n < N ? pr[c_col + n] : 0.0f;
        }
        for (int i = threadIdx.x; i < nt * per_block; i += blockDim.x) {
            const int tt = i / per_block, ch = c0 + i % per_block;
            if (ch < C) {
                const size_t row = (size_t)(first + t0 + tt);
                const float dt = softplus_f(dt_raw[row * C + ch] + dt_bias[ch]);
                const float uu = to_f32(u[row * C + ch]);
                s_dt[i] = dt;
                s_du[i] = dt * uu;
                if (MODE != 1) {
                    s_gate[i] = silu_f(xz[row * ldx + z_col + ch]);
                    s_skip[i] = Dskip[ch] * uu;
                }
            }
        }
        __syncthreads();
#pragma unroll 2
        for (int tt = 0; tt < nt; ++tt) {
            const float dt = s_dt[tt * per_block + cc], du = s_du[tt * per_block + cc];
            const float4* Bt = reinterpret_cast<const float4*>(bc + tt * NP + n0);
            const float4* Ct = reinterpret_cast<const float4*>(bc + (SCAN_TILE + tt) * NP + n0);
            float y = 0.0f;
            if (MODE == 1) dt_sum += dt;
#pragma unroll
            for (int k = 0; k < MAX_PER_LANE; k += 4) {
                const float4 b4 = Bt[k / 4], c4 = MODE == 1 ? b4 : Ct[k / 4];
                const float bb[4] = {b4.x, b4.y, b4.z, b4.w}, cc4[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    // exp(dt A) S as S + expm1(dt A) S: a decay close to 1 keeps its distance from 1 to full precision, so
                    // that no rounding of the factor itself (always the same way for a given dt A) adds up over a long context
                    S[k + e] = fmaf(du, bb[e], fmaf(decay_minus_one<sizeof(T) == 2>(dt * a[k + e]), S[k + e], S[k + e]));
                    if (MODE != 1) y = fmaf(S[k + e], cc4[e], y);
                }
            }
            if (MODE != 1) {
                for (int o = L >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                if (live && sub == 0)
                    out[(size_t)(first + t0 + tt) * C + c] = from_f32<T>((y + s_skip[tt * per_block + cc]) * s_gate[tt * per_block + cc]);
            }
        }
    }
    if (!live) return;
    if (MODE == 1) {
#pragma unroll
        for (int k = 0; k < MAX_PER_LANE; ++k)
            if (n0 + k < N) seg_state[n0 + k] = S[k];
        if (sub == 0) ws[(size_t)seg_slots * CN + (size_t)(seg_base[r] + seg) * C + c] = dt_sum;
        return;
    }
    if (!last_segment) return;
#pragma unroll
    for (int k = 0; k < MAX_PER_LANE; ++k)
        if (n0 + k < N) Sg[n0 + k] = S[k];
    if (sub == 0 && taps > 1) scan_move_tail(tail + (size_t)slot * (taps - 1) * C + c, xz + (size_t)first_req * ldx + c, ldx, C, n_req, taps);
}

// ---------------------------------------------------------------------------------------- a lane per two states, one pass
//
// With up to 16 states a channel and enough channels, a portion needs no segments: a lane per two states gives 8 C chains, which walk all the tokens
// once where the segments' two launches compute every decay twice.  A block takes 16 channels.  Half of its warps make dt, dt u, the gate and the skip
// of each (token, channel) of the next 32 tokens once, from loads asked for a tile earlier, and store the results of the tile before; the other half
// steps through a tile meanwhile, with packed instructions over its lanes' two states (the same operations as a state each, so the same states bit for
// bit).  dt and dt u lie twice in shared memory, B and C as pairs of states of two tokens, so that every operand comes as the packed instruction
// takes it; S C is left in shared memory, and every 16 tokens a lane sums the values of one channel's two tokens.
// 2,048 tokens, 4,096 channels of 16 states: 146 us; a lane per state, every warp in both roles, 170; in segments 345.  What bounds it: issue slots, of
// which a lane per state took twice as many for the same operands read from shared memory.  Not faster: every warp in both roles (225), tiles of 64
// tokens (144 and 151 where tiles of 32 took 143 and 137 for one portion of 2,048 and three of 682: two blocks on an SM instead of three), registers
// for four blocks (148 and 138), the operands of the next four tokens asked for ahead (152 against 145).
// decay_minus_one of two states at one dt, which comes twice, with packed arithmetic where FAST.
__device__ __forceinline__ unsigned long long ls_pair(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ unsigned long long ls_mul(unsigned long long x, unsigned long long y) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ unsigned long long ls_add(unsigned long long x, unsigned long long y) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ unsigned long long ls_fma(unsigned long long x, unsigned long long y, unsigned long long z) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ float ls_lo(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float ls_hi(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
template <bool FAST>
__device__ __forceinline__ unsigned long long decay_minus_one_pair(unsigned long long dt, unsigned long long a) {
    const unsigned long long x = ls_mul(dt, a);
    if (!FAST) return ls_pair(decay_minus_one<false>(ls_lo(x)), decay_minus_one<false>(ls_hi(x)));
    constexpr float LOG2E = 1.44269504088896341f;
    unsigned long long p = ls_fma(x, ls_pair(1.0f / 120.0f, 1.0f / 120.0f), ls_pair(1.0f / 24.0f, 1.0f / 24.0f));
    p = ls_fma(x, p, ls_pair(1.0f / 6.0f, 1.0f / 6.0f));
    p = ls_fma(x, p, ls_pair(0.5f, 0.5f));
    p = ls_mul(x, ls_fma(x, p, ls_pair(1.0f, 1.0f)));
    const unsigned long long y = ls_mul(x, ls_pair(LOG2E, LOG2E));
    float e0, e1;                            // beyond e^-87 a decay is zero beside the 1 that is taken from it
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(ls_lo(y)));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(ls_hi(y)));
    const unsigned long long far = ls_add(ls_pair(e0, e1), ls_pair(-1.0f, -1.0f));
    return ls_pair(ls_lo(x) > -0.25f ? ls_lo(p) : ls_lo(far), ls_hi(x) > -0.25f ? ls_hi(p) : ls_hi(far));
}
constexpr int LS_N = 16, LS_CH = 16, LS_WALK = LS_N / 2 * LS_CH, LS_THREADS = 2 * LS_WALK, LS_TILE = 32, LS_LD = LS_TILE + 1;
struct LsTile {
    float4 dd[LS_CH][LS_LD];                     // [channel][token]: dt, dt, dt u, dt u
    float2 gs[LS_CH][LS_LD];                     // [channel][token]: gate, skip
    float bc[2][LS_TILE / 2][2 * LS_N];          // B, then C: [two tokens][two states][token of the two][state of the two]
};

// grid (R ceil(C / 16)), a request's blocks of channels side by side, the requests from that end of the list on where the longer one stands (a step lists its
// decoding requests before its prompt portions): a long portion's blocks so start together, on SMs of their own (1,500 tokens beside 8 requests of one,
// 1,536 channels: 151 us with the requests' blocks in turn, 73 so).  256 threads: warps 0-3 walk, warps 4-7 make the next tile's values meanwhile and
// store the last tile's results.
template <typename T>
__global__ void __launch_bounds__(LS_THREADS, 3) scan_lanes_kernel(const T* u, const float* dt_raw, const float* dt_bias, const float* proj, int ldp, int b_col,
                                                                   int c_col, const float* A, const float* Dskip, const float* xz, int ldx, int z_col,
                                                                   float* state, float* tail, const int* q_start, const int* slot_ids, T* out, int C, int N,
                                                                   int taps) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t ls_smem[];
    LsTile* tiles = reinterpret_cast<LsTile*>(ls_smem);
    __shared__ __align__(16) float s_y[LS_WALK / 32][8][80];                 // a warp's S C: [two tokens][channel, 20 apart][lane][token of the two]
    __shared__ T s_out[2][LS_TILE][LS_CH];
    const int of_request = (C + LS_CH - 1) / LS_CH, last = gridDim.x / of_request - 1, place = blockIdx.x / of_request;
    const int r = q_start[1] - q_start[0] > q_start[last + 1] - q_start[last] ? place : last - place;
    const int c0 = blockIdx.x % of_request * LS_CH, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, first = q_start[r], n_tok = q_start[r + 1] - first;
    if (n_tok <= 0) return;
    const int n_tiles = (n_tok + LS_TILE - 1) / LS_TILE, slot = slot_ids[r];
    if (warp >= LS_WALK / 32) {
        constexpr int SHARE = LS_TILE * LS_CH / LS_WALK, SHARE_BC = LS_TILE * 2 * LS_N / LS_WALK;
        const int tid = threadIdx.x - LS_WALK, pc = tid & 15, pt = tid >> 4, bn = tid & 31, bt = tid >> 5;
        const bool p_in = c0 + pc < C, b_in = (bn & 15) < N;
        const float bias = p_in ? dt_bias[c0 + pc] : 0.0f, skip = p_in ? Dskip[c0 + pc] : 0.0f;
        const int col = bn < LS_N ? b_col + bn : c_col + bn - LS_N;
        float f_dt[SHARE], f_z[SHARE], f_bc[SHARE_BC];
        T f_u[SHARE];                            // as stored: a conversion beside the load waits for it (8,192 tokens, 2,048 channels: 490 us so, 398 as it is)
        auto fetch = [&](int t0) {
#pragma unroll
            for (int j = 0; j < SHARE; ++j) {
                const int t = t0 + pt + LS_WALK / LS_CH * j;
                const size_t row = (size_t)(first + t);
                const bool in = p_in && t < n_tok;
                f_dt[j] = in ? dt_raw[row * C + c0 + pc] : 0.0f;
                f_u[j] = in ? u[row * C + c0 + pc] : from_f32<T>(0.0f);
                f_z[j] = in ? xz[row * ldx + z_col + c0 + pc] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < SHARE_BC; ++j) {
                const int t = t0 + bt + LS_WALK / 32 * j;
                f_bc[j] = b_in && t < n_tok ? proj[(size_t)(first + t) * ldp + col] : 0.0f;
            }
        };
        auto make = [&](LsTile& x) {
#pragma unroll
            for (int j = 0; j < SHARE; ++j) {
                const int t = pt + LS_WALK / LS_CH * j;
                const float dt = softplus_f(f_dt[j] + bias), uu = to_f32(f_u[j]), du = dt * uu;
                x.dd[pc][t] = make_float4(dt, dt, du, du);
                x.gs[pc][t] = make_float2(silu_f(f_z[j]), skip * uu);
            }
#pragma unroll
            for (int j = 0; j < SHARE_BC; ++j) {
                const int t = bt + LS_WALK / 32 * j;
                x.bc[bn >> 4][t >> 1][((bn & 15) >> 1) * 4 + (t & 1) * 2 + (bn & 1)] = f_bc[j];
            }
        };
        auto store = [&](int i) {
            const int t0 = i * LS_TILE;
#pragma unroll
            for (int j = 0; j < SHARE; ++j) {
                const int t = pt + LS_WALK / LS_CH * j;
                if (p_in && t0 + t < n_tok) out[(size_t)(first + t0 + t) * C + c0 + pc] = s_out[i & 1][t][pc];
            }
        };
        fetch(0);
        make(tiles[0]);
        fetch(LS_TILE);
        __syncthreads();
        for (int i = 0; i < n_tiles; ++i) {
            if (i + 1 < n_tiles) make(tiles[(i + 1) & 1]);
            fetch((i + 2) * LS_TILE);
            if (i > 0) store(i - 1);
            __syncthreads();
        }
        store(n_tiles - 1);
        return;
    }
    const int tid = threadIdx.x, cc = tid >> 3, n = (tid & 7) * 2, c = c0 + cc;
    const bool has0 = c < C && n < N, has1 = c < C && n + 1 < N;             // a state beyond N has A = B = C = 0 and stays zero
    const float a0 = has0 ? A[(size_t)c * N + n] : 0.0f, a1 = has1 ? A[(size_t)c * N + n + 1] : 0.0f;
    const unsigned long long a = ls_pair(a0, a1);
    float* mine = state + ((size_t)slot * C + (c < C ? c : 0)) * N + n;
    unsigned long long S = ls_pair(has0 ? mine[0] : 0.0f, has1 ? mine[1] : 0.0f);
    __syncthreads();
    for (int i = 0; i < n_tiles; ++i) {
        const LsTile& x = tiles[i & 1];
        const int nt = min(LS_TILE, n_tok - i * LS_TILE);
#pragma unroll 1
        for (int g = 0; g < LS_TILE; g += 16) {
            if (g >= nt) break;
            auto walk = [&](auto whole) {                    // whole: 16 tokens; else the nt - g that there are
#pragma unroll
                for (int q = 0; q < 16; q += 4) {
                    unsigned long long near_one[4], du[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const ulonglong2 dd = *reinterpret_cast<const ulonglong2*>(&x.dd[cc][g + q + e]);
                        near_one[e] = decay_minus_one_pair<sizeof(T) == 2>(dd.x, a), du[e] = dd.y;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const ulonglong2 b2 = *reinterpret_cast<const ulonglong2*>(&x.bc[0][(g + q) / 2 + h][n * 2]), c2 = *reinterpret_cast<const ulonglong2*>(&x.bc[1][(g + q) / 2 + h][n * 2]);
                        float y[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            // exp(dt A) S as S + expm1(dt A) S, as above
                            const unsigned long long next = ls_fma(du[2 * h + e], e ? b2.y : b2.x, ls_fma(near_one[2 * h + e], S, S));
                            if (decltype(whole)::value || g + q + 2 * h + e < nt) S = next;
                            const unsigned long long sc = ls_mul(S, e ? c2.y : c2.x);
                            y[e] = ls_lo(sc) + ls_hi(sc);
                        }
                        *reinterpret_cast<float2*>(&s_y[warp][q / 2 + h][(lane >> 3) * 20 + (lane & 7) * 2]) = make_float2(y[0], y[1]);
                    }
                }
            };
            if (g + 16 <= nt) walk(std::true_type{});
            else walk(std::false_type{});
            __syncwarp();
            // a lane sums the eight lanes' values of one channel's two tokens
            const int pair = lane >> 2, ch = lane & 3, c_at = warp * 4 + ch;
            const ulonglong2* p = reinterpret_cast<const ulonglong2*>(&s_y[warp][pair][ch * 20]);
            const ulonglong2 v0 = p[0], v1 = p[1], v2 = p[2], v3 = p[3];
            const unsigned long long y2 = ls_add(ls_add(ls_add(v0.x, v0.y), ls_add(v1.x, v1.y)), ls_add(ls_add(v2.x, v2.y), ls_add(v3.x, v3.y)));
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tok = g + 2 * pair + e;
                const float2 gs = x.gs[c_at][tok];
                s_out[i & 1][tok][c_at] = from_f32<T>(((e ? ls_hi(y2) : ls_lo(y2)) + gs.y) * gs.x);
            }
            __syncwarp();
        }
        __syncthreads();
    }
    if (has0) mine[0] = ls_lo(S);
    if (has1) mine[1] = ls_hi(S);
    if (c < C && n == 0 && taps > 1) scan_move_tail(tail + (size_t)slot * (taps - 1) * C + c, xz + (size_t)first * ldx + c, ldx, C, n_tok, taps);
}

template <typename T>
__global__ void cast_columns_kernel(const float* src, int ld, int col0, int n, T* out, size_t total) {
    pdl_enter();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    out[i] = from_f32<T>(src[(i / n) * ld + col0 + i % n]);
}

}  // namespace

// out[t, c] = dtype(silu(causal convolution over the request's inputs)).  x: FP32 [T, ldx], channels in its first C columns.
// w: FP32 [C, taps] (last column: the current token's), bias FP32 [C], tail FP32 [slots, taps-1, C] (read only here; the scan
// kernel moves it on).
Q6K_API int q6k_conv_silu(const float* x, int ldx, const float* w, const float* bias, const float* tail, const int* req_of_token,
                          const int* q_start, const int* slot_ids, void* out, int T_, int C, int taps, int dtype, int requests, cudaStream_t st) {
    if (T_ == 0) return 0;
    Q6K_REQUIRE(T_ > 0 && C > 0 && taps >= 1 && taps <= MAX_TAPS, "conv_silu: bad sizes T=%d C=%d taps=%d (at most %d taps)", T_, C, taps, MAX_TAPS);
    dim3 grid(T_, (C + 255) / 256);
    Q6K_REQUIRE(grid.y <= 65535, "conv_silu: %d channels exceed the grid limit", C);
    if (conv_rows_taken(T_, requests, x, ldx, bias, tail, out, C, C, taps)) {
        Q6K_DISPATCH(dtype, (conv_rows<T, true>(x, ldx, w, bias, tail, req_of_token, q_start, slot_ids, (T*)out, C, T_, C, taps, 1, st)););
        return q6k_check_launch("conv_silu");
    }
    Q6K_DISPATCH(dtype, q6k_launch(conv_silu_kernel<T>, grid, 256, 0, st, x, ldx, w, bias, tail, req_of_token, q_start, slot_ids,
                                   (T*)out, C, taps););
    return q6k_check_launch("conv_silu");
}

// How many lanes share a channel for N states: the least power of two that leaves each lane at most eight (independent
// chains of the recurrence in one thread hide each other's latency; segments and channels supply the threads).
Q6K_API int q6k_selective_scan_lanes(int N) {
    int L = 1;
    while (L < 32 && L * MAX_PER_LANE < N) L *= 2;
    return L;
}

// u: dtype [T, C] (the convolution's result); dt_raw: FP32 [T, C]; proj: FP32 [T, ldp] with B in columns b_col.. and C in
// c_col.. (N each); A: FP32 [C, N] (negative); Dskip: FP32 [C]; xz: FP32 [T, ldx] with the convolution's inputs in columns
// 0.. and the gate z in columns z_col..; state: FP32 [slots, C, N]; tail: FP32 [slots, taps-1, C]; out: dtype [T, C].
// Tokens per segment when a portion is walked by several blocks.
Q6K_API int q6k_selective_scan_segment() { return 64; }

// Whether a step of T_ rows whose longest portion has up to `segments` segments goes a lane per two states in one pass.  More than 16 states
// take more lanes; fewer than 9 leave half of them idle.  A chain takes 46 ns a token however few there are, and more from a block an SM on; the segments'
// launches take 70 us and then what their 30 instructions per token and state take, spread over the chip (W million states of tokens: 1.3 us each beside
// the 70, 2.45 once they fill it).  One pass and segments, both measured (us, bfloat16): one portion of 2,048 tokens, 640 channels 94 and 100, 4,096 channels
// 146 and 349; of 4,096, 768 channels 184 and 150, 1,024 185 and 191, 1,536 185 and 255; of 8,192, 640 channels 362 and 230, 1,024 395 and 364, 1,536 401
// and 527.  Below 10,000 chains for each token of the longest portion segments stay.  Without segments (up to 64 tokens) a walk of eight states a lane
// takes 0.58 us a token of the longest portion, a lane per two states 4.4 us for every round of blocks (three are resident on an SM), whatever their
// tokens (4,096 channels: 64 tokens 35 and 9 us, 64 beside 8 of one 41 and 32, 32 portions of 8 28 and 86); from 25 tokens a request on the
// latter has the fewer instructions too (8 portions of 64: 53 and 41).  A step of single tokens keeps the former (nothing to fetch ahead).
static bool lanes_taken(int T_, int R, int C, int N, int segments, int longest) {
    const long long blocks = (C + LS_CH - 1) / LS_CH;
    if (N <= 8 || N > LS_N || T_ < 8 * R || blocks > 65535 || R * blocks > 0x7fffffffLL) return false;
    if (segments > 1) {
        const float most = (float)segments * q6k_selective_scan_segment(), W = (float)T_ * C * LS_N * 1e-6f;       // tokens of the longest portion, rounded up
        const float one_pass = 3.0f + most * fmaxf(0.046f, 0.043f * ((float)T_ / most) * (float)blocks / 148), in_segments = fmaxf(70.0f + 1.3f * W, 30.0f + 2.45f * W);
        return (float)T_ * C * N >= most * 10000.0f && one_pass < in_segments;
    }
    return T_ >= 25 * R || 5.0f + 4.4f * (float)(R * blocks) / (3 * 148) < 3.0f + 0.58f * (float)longest;
}
Q6K_API int q6k_selective_scan_lanes_taken(int T_, int R, int C, int N, int segments) { return lanes_taken(T_, R, C, N, segments, R > 0 ? T_ / R : 0); }

// Floats of scratch for `seg_slots` segments in all and R requests.
Q6K_API long long q6k_selective_scan_workspace(int seg_slots, int R, int C, int N) { return R > 0 ? (long long)seg_slots * C * (N + 1) : 0; }

// segments > 1: portions are walked in segments of q6k_selective_scan_segment() tokens (`segments`: the most of any request;
// seg_base: int32 [R], the first segment slot of each request; seg_slots: their total; ws: the scratch above).  longest: tokens of the
// longest portion (0: not said).
Q6K_API int q6k_selective_scan(const void* u, const float* dt_raw, const float* dt_bias, const float* proj, int ldp, int b_col, int c_col,
                               const float* A, const float* Dskip, const float* xz, int ldx, int z_col, float* state, float* tail,
                               const int* q_start, const int* slot_ids, void* out, int R, int C, int N, int taps, int dtype,
                               int segments, const int* seg_base, int seg_slots, float* ws, int T_, int longest, cudaStream_t st) {
    if (R == 0) return 0;
    const int L = q6k_selective_scan_lanes(N);
    Q6K_REQUIRE(R > 0 && C > 0 && N > 0 && N <= L * MAX_PER_LANE, "selective_scan: bad sizes R=%d C=%d N=%d (at most %d states)", R, C, N,
                32 * MAX_PER_LANE);
    Q6K_REQUIRE(taps >= 1 && taps <= MAX_TAPS, "selective_scan: %d taps (at most %d)", taps, MAX_TAPS);
    const int per_block = 128 / L;
    dim3 grid(R, (C + per_block - 1) / per_block);
    Q6K_REQUIRE(grid.y <= 65535, "selective_scan: %d channels exceed the grid limit", C);
    if (lanes_taken(T_, R, C, N, segments, longest > 0 ? longest : T_ / R)) {
        Q6K_DISPATCH(dtype, {
            if (cudaFuncSetAttribute(scan_lanes_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (int)sizeof(LsTile)) != cudaSuccess)
                return q6k_check_launch("selective_scan: shared memory attribute");
            q6k_launch(scan_lanes_kernel<T>, dim3((unsigned)R * ((C + LS_CH - 1) / LS_CH)), LS_THREADS, 2 * sizeof(LsTile), st, (const T*)u, dt_raw, dt_bias, proj, ldp, b_col, c_col,
                       A, Dskip, xz, ldx, z_col, state, tail, q_start, slot_ids, (T*)out, C, N, taps);
        });
        return q6k_check_launch("selective_scan (lanes)");
    }
    const size_t smem = (size_t)SCAN_TILE * (2 * L * MAX_PER_LANE + 4 * per_block) * sizeof(float);
    const int seg_len = q6k_selective_scan_segment();
#define SCAN_LAUNCH(MODE, GRID)                                                                                                      \
    Q6K_DISPATCH(dtype, if (smem > 48 * 1024) cudaFuncSetAttribute(selective_scan_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
                 q6k_launch(selective_scan_kernel<T, MODE>, GRID, 128, smem, st, (const T*)u, dt_raw, dt_bias, proj, ldp, b_col, c_col, A, \
                                   Dskip, xz, ldx, z_col, state, tail, q_start, slot_ids, (T*)out, C, N, L, taps, ws, seg_base, seg_len, seg_slots););
    if (segments <= 1) {
        SCAN_LAUNCH(0, grid);
        return q6k_check_launch("selective_scan");
    }
    Q6K_REQUIRE(seg_base && ws && seg_slots > 0 && segments <= 65535, "selective_scan: segments need their slots and scratch");
    dim3 grid3(R, grid.y, segments);
    SCAN_LAUNCH(1, grid3);
    if (int rc = q6k_check_launch("selective_scan (segments)")) return rc;
    q6k_launch(scan_fold_kernel, dim3((unsigned)(R * (((size_t)C * N + 255) / 256))), 256, 0, st, ws, A, state, q_start, slot_ids, seg_base, seg_len, seg_slots, C, N);
    if (int rc = q6k_check_launch("selective_scan (fold)")) return rc;
    SCAN_LAUNCH(2, grid3);
#undef SCAN_LAUNCH
    return q6k_check_launch("selective_scan");
}

// out[t, j] = dtype(src[t, col0 + j]), j < n: a few columns of an FP32 product as the next product's operand.
Q6K_API int q6k_cast_columns(const float* src, int ld, int col0, int n, void* out, int rows, int dtype, cudaStream_t st) {
    if (rows == 0 || n == 0) return 0;
    Q6K_REQUIRE(rows > 0 && n > 0 && col0 >= 0 && col0 + n <= ld, "cast_columns: columns %d..%d of %d", col0, col0 + n, ld);
    const size_t total = (size_t)rows * n;
    Q6K_DISPATCH(dtype, q6k_launch(cast_columns_kernel<T>, dim3((unsigned)((total + 255) / 256)), 256, 0, st, src, ld, col0, n, (T*)out, total););
    return q6k_check_launch("cast_columns");
}
