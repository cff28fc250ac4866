// The recurrences of `recurrent.cu` over prompts' portions, a chunk of 32 tokens at a time.
//
// Token by token, a matrix S [D][E] is a chain: every token's pass over S (and, for the delta rules, the
// sum over a column that its write needs) waits for the token before, 390 to 520 cycles each, however
// many SMs are idle.  Over a chunk of tokens the same rules are products of small matrices.  With G_t the
// product of the decays of tokens 1..t of the chunk (a number, or a vector over the key channels), S0 the
// state at the chunk's start and everything in fp32:
//
//   A[t][s] = q_t . (k_s decayed from s to t), s <= t        o_t = (G_t q_t) . S0 + sum_s A[t][s] u_s
//   S' = G_end S0 + sum_s (k_s decayed from s to the end) u_s^T
//   u_s = v_s for the rules whose write needs no sum; for the delta rules, with
//   N[t][s] = beta_t k_t . (k_s decayed from s to t), s < t:
//       (1 + N) u = beta (v - (G k) S0), so  u = U - W S0  with  (1 + N) [U | W] = beta [v | G k],
//       and  o_t = (G_t q_t - (A W)_t) . S0 + (A U)_t.
//
// Products of decays are taken as products (a decay may be 0), never as quotients of running products.
//
// chunk_local_kernel: everything of a chunk that does not need S0, all chunks and heads side by side; the
// two triangular systems are one column a thread, its 32 values in registers.
// chunk_walk_kernel: a block owns 16 (or 8) columns of a head's S and walks the chunks in order: per
// chunk two products on fp32 FMA (rows of Q, and W, over S; k^T over u), the next chunk's operands on
// their way by asynchronous copies.  Bound by the fp32 pipe: its 2 or 3 multiply-adds per entry of S and
// token are what the token-by-token walk does too.
//
// The result differs from the token-by-token walk by rounding, and with the way a prompt is cut: the
// bfloat16 engine's prompts alone take this path; decoded tokens and the float32 engine keep the walk.
#define CB_PDL_BIT 11      // this file's bit in CRUCIBLE_PDL (shared with recurrent.cu)
#include "common.cuh"

namespace {

constexpr int RULE_DELTA = 0, RULE_MLSTM = 1, RULE_WKV = 2, RULE_SSD = 3, RULE_CHANNEL = 4;
template <int RULE> constexpr bool VECTOR_DECAY = RULE == RULE_WKV || RULE == RULE_CHANNEL;
template <int RULE> constexpr bool IS_DELTA = RULE == RULE_DELTA || RULE == RULE_CHANNEL;
// rules whose queries' rows over S0 are rows of their own (else they are the rows of q as they are,
// the decay being a number a token)
template <int RULE> constexpr bool OWN_Q = RULE != RULE_SSD && RULE != RULE_MLSTM;
constexpr int CT = 32;              // tokens of a chunk
constexpr int THREADS = 256;
constexpr int AP = CT + 4;          // pitch of the [CT][CT] matrices: rows of whole 16-byte pieces

struct Args {
    const float* qkv;               // rows of C floats: q heads at q_off, k at k_off, v at v_off, decays at w_off
    int C, q_off, k_off, v_off, w_off;
    const float *sc0, *sc1;         // [rows][H]: (decay, beta), (log keep, log in), (decay, step)
    const int *req_row_start, *req_state_slot;
    unsigned char* state;
    long slot_stride, s_off, n_off, m_off;
    float* out;                     // [rows][H][E]
    int H, G, D, E;
    const float *per_head, *kept;
    // workspaces: rows [rows][H][D] (wq: queries over S0, ww: W, wk: keys decayed to the chunk's end),
    // wu [rows][H][E], ws [rows][H] of four numbers (see chunk_local), wg [chunks][H][D]
    float *wq, *ww, *wk, *wu, *wg;
    float4* ws;
};

__device__ __forceinline__ float* state_at(unsigned char* state, long slot_stride, int slot, long off) {
    return reinterpret_cast<float*>(state + (size_t)slot * slot_stride + off);
}
__device__ __forceinline__ void cp16(float* smem, const float* gmem) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gmem) : "memory");
}
// a chunk's place among the step's chunks: strictly growing over a request's chunks and over requests
__device__ __forceinline__ size_t chunk_place(int row, int r) { return (size_t)(row / CT + r); }

// ---- what a chunk can do without the state before it ------------------------------------------
// ws of a token and head: x = G_t (mLSTM: the sum of its log keeps from the chunk's start), y = what its
// row of k is times when it joins the state (the decay to the chunk's end, the step size), z, w (mLSTM):
// the running maximum of the chunk alone and its row's sum of A.
template <int DP, int RULE>
__global__ void __launch_bounds__(THREADS) chunk_local_kernel(const Args a) {
    cb_pdl_trigger();
    cb_pdl_wait();
    constexpr int P = DP + 4;                       // pitch: 8 neighbouring rows' 16-byte reads hit 32 banks
    constexpr bool VECTOR = VECTOR_DECAY<RULE>, DELTA = IS_DELTA<RULE>;
    const int r = blockIdx.z, head = blockIdx.y;
    const int row0 = a.req_row_start[r] + blockIdx.x * CT;
    const int cnt = min(CT, a.req_row_start[r + 1] - row0);
    if (cnt <= 0) return;
    extern __shared__ __align__(16) float smem[];
    float* sk = smem;                               // [CT][P]
    float* sq = sk + CT * P;
    float* sw = sq + CT * P;                        // vector decays only
    float* sA = sw + (VECTOR ? CT * P : 0);         // [CT][AP]
    float* sN = sA + CT * AP;                       // delta rules; before that (scalar decays) L
    float* sa = sN + CT * AP;                       // [CT] decay of a token, [CT] beta or step
    float* sb = sa + CT;
    float* part = sb + CT;                          // vector decays: [DP / 16][2][CT][CT] shares of the dots
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = a.D, E = a.E, H = a.H;
    const int g = head / (H / a.G);

    for (int i = tid; i < CT * (DP / 4); i += THREADS) {
        const int t = i / (DP / 4), d = (i - t * (DP / 4)) * 4;
        const bool in = t < cnt && d < D;
        const float* src = a.qkv + (size_t)(row0 + t) * a.C;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
        *reinterpret_cast<float4*>(sk + t * P + d) = in ? *reinterpret_cast<const float4*>(src + a.k_off + (size_t)g * D + d) : zero;
        *reinterpret_cast<float4*>(sq + t * P + d) = in ? *reinterpret_cast<const float4*>(src + a.q_off + (size_t)g * D + d) : zero;
        if (VECTOR) *reinterpret_cast<float4*>(sw + t * P + d) = in ? *reinterpret_cast<const float4*>(src + a.w_off + (size_t)head * D + d) : one;
    }
    if (warp == 0) {
        // the chunk's numbers, a token a lane; tokens beyond the portion's end change nothing
        const bool in = lane < cnt;
        const size_t at = (size_t)(row0 + lane) * H + head;
        float dec = 1.f, b = 0.f;
        if (RULE == RULE_MLSTM) {
            float f = in ? a.sc0[at] : 0.f, i = in ? a.sc1[at] : -INFINITY;
            const float f_own = f, i_own = i;
            // over tokens 1..t: f = sum of the log keeps, i = max over s of (i_s + log keeps after s)
#pragma unroll
            for (int x = 1; x < CT; x <<= 1) {
                const float fp = __shfl_up_sync(0xffffffffu, f, x), ip = __shfl_up_sync(0xffffffffu, i, x);
                if (lane >= x) {
                    i = fmaxf(f + ip, i);
                    f = fp + f;
                }
            }
            const float before = __shfl_up_sync(0xffffffffu, i, 1);
            dec = lane == 0 ? 0.f : expf(f_own + before - i);
            b = in ? expf(i_own - i) : 0.f;
            if (in) a.ws[at] = make_float4(f, 0.f, i, 0.f);
        } else {
            if (!VECTOR && in) dec = a.sc0[at];
            if (RULE != RULE_WKV && in) b = a.sc1[at];
        }
        sa[lane] = dec;
        sb[lane] = b;
        if (!VECTOR) {
            // L[t][s] = product of the decays of s + 1 .. t; a column s a lane
            __syncwarp();
            float l = 0.f, G = 1.f;
            for (int t = 0; t < CT; ++t) {
                const float x = sa[t];
                l = t == lane ? 1.f : l * x;
                sN[t * AP + lane] = l;
                if (t <= lane) G *= x;
            }
            if (in) {
                const float to_end = l * (RULE == RULE_DELTA ? 1.f : b);
                if (RULE == RULE_MLSTM) a.ws[at].y = to_end;
                else a.ws[at] = make_float4(G, to_end, 0.f, 0.f);
            }
        }
    }
    __syncthreads();

    // the dots of the chunk's rows: A, and for the delta rules N
    if (!VECTOR) {
        const int tr = tid >> 4, tc = tid & 15;     // rows tr, tr + 16 against columns tc, tc + 16
        float qk[3] = {0.f, 0.f, 0.f}, kk[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
        for (int d = 0; d < DP; d += 4) {
            float4 q[2], k[2], c[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                q[i] = *reinterpret_cast<const float4*>(sq + (tr + 16 * i) * P + d);
                if (DELTA) k[i] = *reinterpret_cast<const float4*>(sk + (tr + 16 * i) * P + d);
                c[i] = *reinterpret_cast<const float4*>(sk + (tc + 16 * i) * P + d);
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) {           // (0, 0), (1, 0), (1, 1): the fourth lies above the diagonal
                const float4 x = q[p > 0], z = c[p > 1];
                qk[p] = fmaf(x.x, z.x, qk[p]); qk[p] = fmaf(x.y, z.y, qk[p]);
                qk[p] = fmaf(x.z, z.z, qk[p]); qk[p] = fmaf(x.w, z.w, qk[p]);
                if (DELTA) {
                    const float4 y = k[p > 0];
                    kk[p] = fmaf(y.x, z.x, kk[p]); kk[p] = fmaf(y.y, z.y, kk[p]);
                    kk[p] = fmaf(y.z, z.z, kk[p]); kk[p] = fmaf(y.w, z.w, kk[p]);
                }
            }
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const int t = tr + (p > 0 ? 16 : 0), s = tc + (p > 1 ? 16 : 0);
            const float l = sN[t * AP + s];         // 0 above the diagonal
            sA[t * AP + s] = qk[p] * l * (DELTA ? 1.f : sb[s]);
            if (DELTA) sN[t * AP + s] = s < t ? sb[t] * kk[p] * l : 0.f;
        }
        sA[tr * AP + tc + 16] = 0.f;
        if (DELTA) sN[tr * AP + tc + 16] = 0.f;
        __syncthreads();
    } else {
        // a column s a lane, 16 channels a warp: the key decays on its way down the rows
        if (warp < DP / 16) {
            const int d0 = warp * 16, s = lane;
            float w[16], first = 0.f;
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 k = *reinterpret_cast<const float4*>(sk + s * P + d0 + i);
                w[i] = k.x; w[i + 1] = k.y; w[i + 2] = k.z; w[i + 3] = k.w;
            }
            if (RULE == RULE_WKV) {                 // a token's own key counts through the bonus
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float u = d0 + i < D ? a.per_head[(size_t)head * D + d0 + i] : 0.f;
                    first = fmaf(u * w[i], sq[s * P + d0 + i], first);
                }
            }
            float* to = part + (size_t)warp * 2 * CT * CT;
            for (int t = 0; t < CT; ++t) {
                float qk[4] = {0.f, 0.f, 0.f, 0.f}, kk[4] = {0.f, 0.f, 0.f, 0.f};
                const float* rq = sq + t * P + d0;
                const float* rk = sk + t * P + d0;
                const float* rw = sw + t * P + d0;
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(rq + i);
                    const float4 y = *reinterpret_cast<const float4*>(rk + i);
                    const float4 z = *reinterpret_cast<const float4*>(rw + i);
                    const float qv[4] = {x.x, x.y, x.z, x.w}, kv[4] = {y.x, y.y, y.z, y.w}, gv[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (RULE == RULE_CHANNEL && t > s) w[i + e] *= gv[e];
                        qk[e] = fmaf(qv[e], w[i + e], qk[e]);
                        if (DELTA) kk[e] = fmaf(kv[e], w[i + e], kk[e]);
                        if (RULE == RULE_WKV && t > s) w[i + e] *= gv[e];
                    }
                }
                float x = (qk[0] + qk[1]) + (qk[2] + qk[3]);
                if (RULE == RULE_WKV && t == s) x = first;
                to[t * CT + s] = t >= s ? x : 0.f;
                if (DELTA) to[CT * CT + t * CT + s] = t > s ? (kk[0] + kk[1]) + (kk[2] + kk[3]) : 0.f;
            }
        }
        __syncthreads();
        for (int i = tid; i < CT * CT; i += THREADS) {
            const int t = i / CT, s = i - t * CT;
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int w = 0; w < DP / 16; ++w) {
                x += part[(size_t)w * 2 * CT * CT + i];
                if (DELTA) y += part[(size_t)(w * 2 + 1) * CT * CT + i];
            }
            sA[t * AP + s] = x;
            if (DELTA) sN[t * AP + s] = sb[t] * y;
        }
        __syncthreads();
    }

    if (RULE == RULE_MLSTM && tid < cnt) {
        float n = 0.f;
        for (int s = 0; s <= tid; ++s) n += sA[tid * AP + s];
        a.ws[(size_t)(row0 + tid) * H + head].w = n;
    }
    // vector decays: keys decayed to the chunk's end, and the whole chunk's decay
    if (VECTOR && tid < D) {
        float to_end = 1.f;
        for (int t = cnt - 1; t >= 0; --t) {
            a.wk[((size_t)(row0 + t) * H + head) * D + tid] = sk[t * P + tid] * to_end;
            to_end *= sw[t * P + tid];
        }
        a.wg[(chunk_place(row0, r) * H + head) * D + tid] = to_end;
    }
    // the columns: E of v, then (delta rules: W; other vector decays: the decayed queries) D of the keys
    const int columns = E + (OWN_Q<RULE> ? D : 0);
    for (int c = tid; c < columns; c += THREADS) {
        float x[CT];
        const bool is_v = c < E;
        const int d = c - E;
        if (is_v) {
            const float* src = a.qkv + (size_t)row0 * a.C + a.v_off + (size_t)head * E + c;
#pragma unroll
            for (int t = 0; t < CT; ++t) x[t] = t < cnt ? src[(size_t)t * a.C] : 0.f;
        } else if (DELTA) {
            float G = 1.f;
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                G *= VECTOR ? sw[t * P + d] : sa[t];
                x[t] = sk[t * P + d] * G;
            }
        }
        if (DELTA) {
            // forward substitution down the column
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                float s0 = 0.f, s1 = 0.f;
#pragma unroll
                for (int s = 0; s < t; s += 4) {
                    const float4 n = *reinterpret_cast<const float4*>(sN + t * AP + s);
                    s0 = fmaf(n.x, x[s], s0);
                    if (s + 1 < t) s1 = fmaf(n.y, x[s + 1], s1);
                    if (s + 2 < t) s0 = fmaf(n.z, x[s + 2], s0);
                    if (s + 3 < t) s1 = fmaf(n.w, x[s + 3], s1);
                }
                x[t] = fmaf(sb[t], x[t], -(s0 + s1));
            }
        }
        const float skip = RULE == RULE_SSD ? a.per_head[head] : 0.f;
        float G = 1.f;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            float s0 = 0.f, s1 = 0.f;
            if (is_v || DELTA) {
#pragma unroll
                for (int s = 0; s <= t; s += 4) {
                    const float4 n = *reinterpret_cast<const float4*>(sA + t * AP + s);
                    s0 = fmaf(n.x, x[s], s0);
                    if (s + 1 <= t) s1 = fmaf(n.y, x[s + 1], s1);
                    if (s + 2 <= t) s0 = fmaf(n.z, x[s + 2], s0);
                    if (s + 3 <= t) s1 = fmaf(n.w, x[s + 3], s1);
                }
            }
            const float o = s0 + s1;
            if (t < cnt) {
                const size_t at = (size_t)(row0 + t) * H + head;
                if (is_v) {
                    a.out[at * E + c] = RULE == RULE_SSD ? fmaf(skip, x[t], o) : o;
                    if (DELTA) a.wu[at * E + c] = x[t];
                } else {
                    // wkv reads the state before its token's decay
                    if (RULE != RULE_WKV) G *= VECTOR ? sw[t * P + d] : sa[t];
                    a.wq[at * a.D + d] = fmaf(sq[t * P + d], G, -o);
                    if (RULE == RULE_WKV) G *= sw[t * P + d];
                    if (DELTA) a.ww[at * a.D + d] = x[t];
                }
            }
        }
    }
}

// ---- the state from chunk to chunk ---------------------------------------------------------------
template <int DP, int RULE, int ET>
__global__ void __launch_bounds__(THREADS) chunk_walk_kernel(const Args a) {
    cb_pdl_trigger();
    cb_pdl_wait();
    constexpr int P = DP + 4, CG = ET / 4;
    constexpr bool VECTOR = VECTOR_DECAY<RULE>, DELTA = IS_DELTA<RULE>;
    constexpr int ROWS = DELTA ? 2 * CT : CT;            // rows over S: the queries', then W
    constexpr int RG = 16;                               // row groups; a thread has ROWS / 16 rows of one
    constexpr int SPLIT = THREADS / (RG * CG);           // shares of the sum over D
    constexpr int DS = DP / SPLIT;
    constexpr int STAGE = (ROWS + CT) * P + CT * ET;     // rows over S, keys, u
    extern __shared__ __align__(16) float smem[];
    float* S = smem;                                     // [DP][ET]
    float* red = S + DP * ET;                            // [SPLIT][ROWS][ET]
    float* su = red + SPLIT * ROWS * ET;                 // [CT][ET]: u as it joins the state
    float* sg = su + CT * ET;                            // [DP]: the chunk's decay; mLSTM: n
    float* sx = sg + DP;                                 // [CT][2]: mLSTM's factors of a row's two shares
    float4* sc = reinterpret_cast<float4*>(sx + 2 * CT); // [2][CT] the tokens' numbers
    float* stage = reinterpret_cast<float*>(sc + 2 * CT);
    const int r = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * ET;
    const int tid = threadIdx.x;
    const int D = a.D, E = a.E, H = a.H;
    const int g = head / (H / a.G);
    const int row0 = a.req_row_start[r], row1 = a.req_row_start[r + 1];
    const int slot = a.req_state_slot[r];
    float* state = state_at(a.state, a.slot_stride, slot, a.s_off) + (size_t)head * D * E;
    const float* n0 = RULE == RULE_MLSTM ? a.kept + (size_t)r * (H * D + H) : nullptr;
    float m0 = RULE == RULE_MLSTM ? n0[(size_t)H * D + head] : 0.f;
    for (int i = tid; i < DP * ET; i += THREADS) {
        const int d = i / ET, c = i - d * ET;
        S[i] = d < D && col0 + c < E ? state[(size_t)d * E + col0 + c] : 0.f;
    }
    if (RULE == RULE_MLSTM)
        for (int d = tid; d < DP; d += THREADS) sg[d] = d < D ? n0[(size_t)head * D + d] : 0.f;
    for (int i = tid; i < 2 * STAGE; i += THREADS) stage[i] = 0.f;      // the rows' and columns' padding
    __syncthreads();

    auto fetch = [&](int base, int buf) {
        float* rows = stage + buf * STAGE;
        float* keys = rows + ROWS * P;
        float* u = keys + CT * P;
        const int cnt = min(CT, row1 - base);
        const int per = D >> 2;
        for (int i = tid; i < CT * per; i += THREADS) {
            const int t = i / per, d = (i - t * per) << 2;
            if (t < cnt) {
                const size_t at = (size_t)(base + t) * H + head;
                const float* src = a.qkv + (size_t)(base + t) * a.C + (size_t)g * D + d;
                cp16(rows + t * P + d, OWN_Q<RULE> ? a.wq + at * D + d : src + a.q_off);
                if (DELTA) cp16(rows + (CT + t) * P + d, a.ww + at * D + d);
                cp16(keys + t * P + d, VECTOR ? a.wk + at * D + d : src + a.k_off);
            } else {                                     // a portion's last chunk: rows of an earlier one are there
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(rows + t * P + d) = zero;
                if (DELTA) *reinterpret_cast<float4*>(rows + (CT + t) * P + d) = zero;
                *reinterpret_cast<float4*>(keys + t * P + d) = zero;
            }
        }
        for (int i = tid; i < CT * CG; i += THREADS) {
            const int t = i / CG, c = (i - t * CG) * 4;
            if (t < cnt && col0 + c < E) {
                const size_t row = (size_t)(base + t);
                cp16(u + t * ET + c, DELTA ? a.wu + (row * H + head) * E + col0 + c
                                           : a.qkv + row * a.C + a.v_off + (size_t)head * E + col0 + c);
            } else {
                *reinterpret_cast<float4*>(u + t * ET + c) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (!VECTOR && tid < CT) {
            if (tid < cnt) cp16(reinterpret_cast<float*>(sc + buf * CT + tid),
                                reinterpret_cast<const float*>(a.ws + (size_t)(base + tid) * H + head));
            else sc[buf * CT + tid] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (row0 < row1) fetch(row0, 0);
    int buf = 0;
    for (int base = row0; base < row1; base += CT, buf ^= 1) {
        const int cnt = min(CT, row1 - base);
        const float* rows = stage + buf * STAGE;
        const float* keys = rows + ROWS * P;
        const float* u = keys + CT * P;
        const float4* nums = sc + buf * CT;
        // where this thread's sums of the first product go
        const int orow = tid / CG, ocol = (tid - orow * CG) * 4;
        const bool has_out = orow < cnt && col0 + ocol < E;
        float* out_at = a.out + ((size_t)(base + orow) * H + head) * E + col0 + ocol;
        float4 local = make_float4(0.f, 0.f, 0.f, 0.f);
        if (has_out) local = *reinterpret_cast<const float4*>(out_at);
        if (base + CT < row1) {
            fetch(base + CT, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        if (VECTOR && tid < D) sg[tid] = a.wg[(chunk_place(base, r) * H + head) * D + tid];
        __syncthreads();
        // the rows over S
        {
            const int share = tid / (RG * CG), in = tid - share * (RG * CG);
            const int rg = in / CG, cg = in - rg * CG;
            float acc[ROWS / RG][4];
#pragma unroll
            for (int i = 0; i < ROWS / RG; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 4
            for (int d = share * DS; d < share * DS + DS; d += 4) {
                float4 x[ROWS / RG], y[4];
#pragma unroll
                for (int i = 0; i < ROWS / RG; ++i)
                    x[i] = *reinterpret_cast<const float4*>(rows + (rg + RG * i) * P + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(S + (d + j) * ET + 4 * cg);
#pragma unroll
                for (int i = 0; i < ROWS / RG; ++i) {
                    const float xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        acc[i][0] = fmaf(xs[j], y[j].x, acc[i][0]);
                        acc[i][1] = fmaf(xs[j], y[j].y, acc[i][1]);
                        acc[i][2] = fmaf(xs[j], y[j].z, acc[i][2]);
                        acc[i][3] = fmaf(xs[j], y[j].w, acc[i][3]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < ROWS / RG; ++i)
                *reinterpret_cast<float4*>(red + ((size_t)share * ROWS + rg + RG * i) * ET + 4 * cg) =
                    make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        float g_end = 1.f, in_end = 1.f;
        if (RULE == RULE_MLSTM) {
            // n . q of a token by eight lanes, then the factors of its row's two shares
            const int t = tid >> 3, p = tid & 7;
            float nq = 0.f;
#pragma unroll 4
            for (int d = p; d < DP; d += 8) nq = fmaf(sg[d], rows[t * P + d], nq);
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) nq += __shfl_xor_sync(0xffffffffu, nq, x);
            const float4 own = nums[t], last = nums[cnt - 1];
            const float m = fmaxf(own.x + m0, own.z);
            const float before = expf(own.x + m0 - m), within = expf(own.z - m);
            const float low = fmaxf(fabsf(fmaf(before, nq, within * own.w)), expf(-m)) + 1e-6f;
            if (p == 0) {
                sx[2 * t] = before / low;
                sx[2 * t + 1] = within / low;
            }
            const float m_end = fmaxf(last.x + m0, last.z);
            g_end = expf(last.x + m0 - m_end);
            in_end = expf(last.z - m_end);
            m0 = m_end;
        } else if (!VECTOR) {
            g_end = nums[cnt - 1].x;
        }
        __syncthreads();
        if (orow < ROWS) {
            float4 sum = *reinterpret_cast<const float4*>(red + (size_t)orow * ET + ocol);
#pragma unroll
            for (int x = 1; x < SPLIT; ++x) {
                const float4 y = *reinterpret_cast<const float4*>(red + ((size_t)x * ROWS + orow) * ET + ocol);
                sum.x += y.x; sum.y += y.y; sum.z += y.z; sum.w += y.w;
            }
            if (orow < CT) {
                float fa = 1.f, fb = 1.f;
                if (RULE == RULE_SSD) fa = nums[orow].x;
                if (RULE == RULE_MLSTM) {
                    fa = sx[2 * orow];
                    fb = sx[2 * orow + 1];
                }
                if (RULE == RULE_MLSTM) {
                    local.x *= fb; local.y *= fb; local.z *= fb; local.w *= fb;
                }
                if (has_out)
                    *reinterpret_cast<float4*>(out_at) = make_float4(fmaf(fa, sum.x, local.x), fmaf(fa, sum.y, local.y),
                                                                     fmaf(fa, sum.z, local.z), fmaf(fa, sum.w, local.w));
            } else {
                const int t = orow - CT;
                const float4 own = *reinterpret_cast<const float4*>(u + t * ET + ocol);
                const float f = VECTOR ? 1.f : nums[t].y;
                *reinterpret_cast<float4*>(su + t * ET + ocol) =
                    make_float4(f * (own.x - sum.x), f * (own.y - sum.y), f * (own.z - sum.z), f * (own.w - sum.w));
            }
        }
        if (!DELTA)
            for (int i = tid; i < CT * CG; i += THREADS) {
                const int t = i / CG, c = (i - t * CG) * 4;
                const float4 own = *reinterpret_cast<const float4*>(u + t * ET + c);
                const float f = VECTOR ? 1.f : nums[t].y * in_end;
                *reinterpret_cast<float4*>(su + t * ET + c) = make_float4(f * own.x, f * own.y, f * own.z, f * own.w);
            }
        __syncthreads();
        // the state: decayed, and the chunk's k^T u
        for (int i = tid; i < (DP / 2) * CG; i += THREADS) {
            const int d = (i / CG) * 2, cg = i % CG;
            float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
            for (int t = 0; t < CT; ++t) {
                const float2 k = *reinterpret_cast<const float2*>(keys + t * P + d);
                const float4 v = *reinterpret_cast<const float4*>(su + t * ET + 4 * cg);
                x[0] = fmaf(k.x, v.x, x[0]); x[1] = fmaf(k.x, v.y, x[1]); x[2] = fmaf(k.x, v.z, x[2]); x[3] = fmaf(k.x, v.w, x[3]);
                y[0] = fmaf(k.y, v.x, y[0]); y[1] = fmaf(k.y, v.y, y[1]); y[2] = fmaf(k.y, v.z, y[2]); y[3] = fmaf(k.y, v.w, y[3]);
            }
            const float ga = VECTOR ? sg[d] : g_end, gb = VECTOR ? sg[d + 1] : g_end;
            float4* a0 = reinterpret_cast<float4*>(S + (size_t)d * ET + 4 * cg);
            float4* a1 = reinterpret_cast<float4*>(S + (size_t)(d + 1) * ET + 4 * cg);
            const float4 p = *a0, q = *a1;
            *a0 = make_float4(fmaf(ga, p.x, x[0]), fmaf(ga, p.y, x[1]), fmaf(ga, p.z, x[2]), fmaf(ga, p.w, x[3]));
            *a1 = make_float4(fmaf(gb, q.x, y[0]), fmaf(gb, q.y, y[1]), fmaf(gb, q.z, y[2]), fmaf(gb, q.w, y[3]));
        }
        if (RULE == RULE_MLSTM)
            for (int d = tid; d < DP; d += THREADS) {
                float n = 0.f;
#pragma unroll 8
                for (int t = 0; t < CT; ++t) n = fmaf(keys[t * P + d], nums[t].y, n);
                sg[d] = fmaf(g_end, sg[d], in_end * n);
            }
        __syncthreads();
    }
    for (int i = tid; i < DP * ET; i += THREADS) {
        const int d = i / ET, c = i - d * ET;
        if (d < D && col0 + c < E) state[(size_t)d * E + col0 + c] = S[i];
    }
    if (RULE == RULE_MLSTM && blockIdx.z == 0) {
        float* N = state_at(a.state, a.slot_stride, slot, a.n_off) + (size_t)head * D;
        for (int d = tid; d < D; d += THREADS) N[d] = sg[d];
        if (tid == 0) state_at(a.state, a.slot_stride, slot, a.m_off)[head] = m0;
    }
}

template <typename K>
int allow_smem(K kernel, size_t smem) {
    return smem > 48 * 1024 ? (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : 0;
}

template <int DP, int RULE, int ET>
int launch_walk(const Args& a, int n_requests, cudaStream_t s) {
    constexpr bool DELTA = IS_DELTA<RULE>;
    constexpr int ROWS = DELTA ? 2 * CT : CT, SPLIT = THREADS / (16 * (ET / 4)), P = DP + 4;
    const size_t floats = DP * ET + SPLIT * ROWS * ET + CT * ET + DP + 2 * CT + 8 * CT + 2 * ((ROWS + CT) * P + CT * ET);
    const int rc = allow_smem(chunk_walk_kernel<DP, RULE, ET>, floats * sizeof(float));
    if (rc) return rc;
    const dim3 grid(n_requests, a.H, (a.E + ET - 1) / ET);
    cb_launch(chunk_walk_kernel<DP, RULE, ET>, grid, dim3(THREADS), floats * sizeof(float), s, a);
    return cb_last_error();
}

template <int DP, int RULE>
int launch_chunks(const Args& a, int n_requests, int max_new, cudaStream_t s) {
    constexpr int P = DP + 4;
    const size_t floats = (VECTOR_DECAY<RULE> ? 3 : 2) * CT * P + 2 * CT * AP + 2 * CT
                          + (VECTOR_DECAY<RULE> ? (DP / 16) * 2 * CT * CT : 0);
    int rc = allow_smem(chunk_local_kernel<DP, RULE>, floats * sizeof(float));
    if (rc) return rc;
    const dim3 grid((max_new + CT - 1) / CT, a.H, n_requests);
    cb_launch(chunk_local_kernel<DP, RULE>, grid, dim3(THREADS), floats * sizeof(float), s, a);
    rc = cb_last_error();
    if (rc) return rc;
    return launch_walk<DP, RULE, 16>(a, n_requests, s);
}

}  // namespace

// The rules and their operands are those of cb_matrix_memory (recurrent.cu); max_new: the most tokens a
// request brings.  Workspaces, fp32: wq, ww, wk [rows][H][D] and wu [rows][H][E] (those the rule needs:
// delta wq ww wu; wkv wq wk; channel all four; others none), ws [rows][H][4], wg [rows / 32 + requests][H][D].
CB_EXPORT int cb_matrix_memory_chunks(int rule, const float* qkv, int C, int q_off, int k_off, int v_off,
                                      const float* sc0, const float* sc1, const int* req_row_start,
                                      const int* req_state_slot, void* state, long slot_stride, long s_off,
                                      long n_off, long m_off, float* out, int n_requests, int max_new, int n_heads,
                                      int n_qk_heads, int key_dim, int value_dim, int w_off, const float* per_head,
                                      const float* kept, float* wq, float* ww, float* wk, float* wu, float* ws,
                                      float* wg, void* stream) {
    if (n_requests <= 0 || max_new <= 0) return 0;
    const bool vector = rule == RULE_WKV || rule == RULE_CHANNEL;
    if (n_heads % n_qk_heads != 0 || key_dim > 128 || n_requests > 65535 || n_heads > 65535
        || ((C | q_off | k_off | v_off | key_dim | value_dim | (vector ? w_off : 0)) & 3) != 0)
        return CB_ERR_UNSUPPORTED;
    if ((rule == RULE_WKV || rule == RULE_SSD) && per_head == nullptr) return CB_ERR_UNSUPPORTED;
    if (rule == RULE_MLSTM && kept == nullptr) return CB_ERR_UNSUPPORTED;
    Args a;
    a.qkv = qkv; a.C = C; a.q_off = q_off; a.k_off = k_off; a.v_off = v_off; a.w_off = w_off;
    a.sc0 = sc0; a.sc1 = sc1; a.req_row_start = req_row_start; a.req_state_slot = req_state_slot;
    a.state = (unsigned char*)state; a.slot_stride = slot_stride; a.s_off = s_off; a.n_off = n_off; a.m_off = m_off;
    a.out = out; a.H = n_heads; a.G = n_qk_heads; a.D = key_dim; a.E = value_dim;
    a.per_head = per_head; a.kept = kept;
    a.wq = wq; a.ww = ww; a.wk = wk; a.wu = wu; a.wg = wg; a.ws = reinterpret_cast<float4*>(ws);
    cudaStream_t s = (cudaStream_t)stream;
#define CB_CHUNKS(RR)                                                                                       \
    if (rule == RR)                                                                                         \
        return key_dim <= 64 ? launch_chunks<64, RR>(a, n_requests, max_new, s)                             \
                             : launch_chunks<128, RR>(a, n_requests, max_new, s)
    CB_CHUNKS(RULE_DELTA);
    CB_CHUNKS(RULE_MLSTM);
    CB_CHUNKS(RULE_WKV);
    CB_CHUNKS(RULE_SSD);
    CB_CHUNKS(RULE_CHANNEL);
#undef CB_CHUNKS
    return CB_ERR_UNSUPPORTED;
}
