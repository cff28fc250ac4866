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
// Products of decays are taken as products (a decay may be 0), never as quotients of running products; no
// sum runs over a later token's values, not even times zero (a later NaN stays later).
//
// chunk_local_kernel: everything of a chunk that does not need S0, all chunks and heads side by side; the
// two triangular systems are one column a thread, its 32 values in registers.
// Rules without a sum: chunk_local also leaves what the chunk adds to S, chunk_scan_kernel turns that into
// S as every chunk begins, and chunk_out_kernel adds the queries over it, again all chunks side by side.
// Delta rules: chunk_walk_kernel; a block owns 16 (or 8) columns of a head's S and walks the chunks in
// order: per chunk two products on fp32 FMA (rows of Q and W over S; k^T over u), the next chunk's
// operands on their way by TMA.
//
// Measured at 2,048 tokens (token by token -> in chunks), 16 heads of 128: delta 503 -> 201 us (the chunks'
// numbers 64, the walk 137), channel delta 551 -> 251, mLSTM 590 -> 172, wkv 467 -> 169, state space 408 -> 168;
// 8 heads: 502 -> 126, 551 -> 152, 589 -> 91, 467 -> 90, 407 -> 79.  16,384 tokens of 16 heads in slices (256 MB of
// workspaces): delta 1,768 us, 1,760 at once; mLSTM 1,340 and 1,292; state space 1,403 and 1,380.
//
// The result differs from the token-by-token walk by rounding, and with the way a prompt is cut: the
// bfloat16 engine's prompts alone take this path; decoded tokens and the float32 engine keep the walk.
#define CB_PDL_BIT 11      // this file's bit in CRUCIBLE_PDL (shared with recurrent.cu)
#include <type_traits>
#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int RULE_DELTA = 0, RULE_MLSTM = 1, RULE_WKV = 2, RULE_SSD = 3, RULE_CHANNEL = 4;
template <int RULE> constexpr bool VECTOR_DECAY = RULE == RULE_WKV || RULE == RULE_CHANNEL;
template <int RULE> constexpr bool IS_DELTA = RULE == RULE_DELTA || RULE == RULE_CHANNEL;
// rules whose queries over S0 are rows of their own (else they are the rows of q as they are, the decay
// being a number a token)
template <int RULE> constexpr bool OWN_Q = RULE != RULE_SSD && RULE != RULE_MLSTM;
constexpr int CT = 32;              // tokens of a chunk
constexpr int THREADS = 256;
constexpr int AP = CT + 4;          // pitch of the [CT][CT] matrices: rows of whole 16-byte pieces
// Padding of chunk_local's rows of keys and queries.  The dots of scalar decays: eight lanes read 64 bytes of two
// neighbouring rows, which lie 16 banks apart (with 4, as the others have it, 12 of 16 banks met twice).  Vector decays: a row a lane,
// 16 bytes of eight rows on 32 banks.
template <int RULE> constexpr int PAD = VECTOR_DECAY<RULE> ? 4 : 16;

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
    float* kept_next;               // mLSTM: n and m as this slice ends, laid out like kept
    int skip, limit;                // the slice: of every request's tokens those from skip on, limit at most
    // workspaces, of the slice (Piece): rows [rows][H][D] (wq: queries over S0, ww: W, wk: keys decayed to the chunk's end),
    // wu [rows][H][E], ws [rows][H] of four numbers (see chunk_local), wg [chunks][H][D] decays; wl
    // [chunks][H][D][E] what a chunk adds to S, then S as it begins; wn [chunks][H][D] likewise of n and wm
    // [chunks][H] of m (mLSTM)
    float *wq, *ww, *wk, *wu, *wg, *wl, *wn, *wm;
    float4* ws;
    int rows, piece_rows;           // of qkv, and of the workspaces
    int* status;                    // a wait that ran out is recorded here
};

// two fp32 numbers in one register pair, multiplied and added by one instruction
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t fma_pair(pair_t a, pair_t b, pair_t c) {
    pair_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ pair_t make_pair_of(float lo, float hi) {
    pair_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 split_pair(pair_t p) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float pair_sum(pair_t p) {
    const float2 v = split_pair(p);
    return v.x + v.y;
}
__device__ __forceinline__ ulonglong2 pairs_at(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

__device__ __forceinline__ float* state_at(unsigned char* state, long slot_stride, int slot, long off) {
    return reinterpret_cast<float*>(state + (size_t)slot * slot_stride + off);
}
// The slice's rows of a request: [row0, row1) of the step; their rows of a workspace are `shift` less.
// (A request's first: the rows of the requests before it, or limit for each of those if that is less.)
struct Piece { int row0, row1, shift; };
__device__ __forceinline__ Piece piece_of(const Args& a, int r) {
    const int start = a.req_row_start[r], before = start - a.req_row_start[0];
    Piece p;
    p.row0 = start + a.skip;
    p.row1 = min(a.req_row_start[r + 1], p.row0 + a.limit);
    p.shift = p.row0 - (int)min((long)before, (long)r * a.limit);
    return p;
}
// a chunk's place among the slice's chunks: strictly growing over a request's chunks and over requests
__device__ __forceinline__ size_t chunk_place(int row, int r) { return (size_t)(row / CT + r); }

// row t of a lower triangular matrix times a column in registers (pairs of neighbouring tokens), entries
// 0 .. COUNT - 1
template <int COUNT, int COLS>
__device__ __forceinline__ void row_times(const float* row, const pair_t (&x)[COLS][CT / 2], float (&sum)[COLS]) {
    pair_t a[COLS], b[COLS];
    float tail[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) a[c] = b[c] = 0, tail[c] = 0.f;
#pragma unroll
    for (int s = 0; s < COUNT; s += 4) {
        const ulonglong2 n = pairs_at(row + s);
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            if (s + 1 < COUNT) a[c] = fma_pair(n.x, x[c][s / 2], a[c]);
            else tail[c] = split_pair(n.x).x * split_pair(x[c][s / 2]).x;
            if (s + 3 < COUNT) b[c] = fma_pair(n.y, x[c][s / 2 + 1], b[c]);
            else if (s + 2 < COUNT) tail[c] = split_pair(n.y).x * split_pair(x[c][s / 2 + 1]).x;
        }
    }
#pragma unroll
    for (int c = 0; c < COLS; ++c) sum[c] = (pair_sum(a[c]) + pair_sum(b[c])) + tail[c];
}
template <int T>
__device__ __forceinline__ void set_token(pair_t (&x)[CT / 2], float v) {
    const float2 p = split_pair(x[T / 2]);
    x[T / 2] = T % 2 ? make_pair_of(p.x, v) : make_pair_of(v, p.y);
}
template <int T>
__device__ __forceinline__ float get_token(const pair_t (&x)[CT / 2]) {
    const float2 p = split_pair(x[T / 2]);
    return T % 2 ? p.y : p.x;
}
// F::template at<T>() for T = 0 .. CT - 1, unrolled
template <int T, typename F>
__device__ __forceinline__ void each_token(F& f) {
    if constexpr (T < CT) {
        f.template at<T>();
        each_token<T + 1>(f);
    }
}

// forward substitution down the columns: (1 + N) x = b x
template <int COLS> struct Substitute {
    pair_t (&x)[COLS][CT / 2];
    const float *N, *b;
    template <int T> __device__ __forceinline__ void at() {
        float sum[COLS];
        row_times<T>(N + T * AP, x, sum);
#pragma unroll
        for (int c = 0; c < COLS; ++c) set_token<T>(x[c], fmaf(b[T], get_token<T>(x[c]), -sum[c]));
    }
};
// columns of v: their tokens' results within the chunk, and u for the delta rules
template <int RULE, int COLS> struct ValueColumn {
    pair_t (&x)[COLS][CT / 2];
    const float* A;
    float *out, *wu, skip;
    size_t stride;
    int cnt, apart, cols;             // columns this thread has, `apart` from one another
    template <int T> __device__ __forceinline__ void at() {
        if (T < cnt) {
            float o[COLS];
            row_times<T + 1>(A + T * AP, x, o);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                if (c >= cols) break;
                const float v = get_token<T>(x[c]);
                out[T * stride + c * apart] = RULE == RULE_SSD ? fmaf(skip, v, o[c]) : o[c];
                if (IS_DELTA<RULE>) wu[T * stride + c * apart] = v;
            }
        }
    }
};
// key channels: the queries' rows over S0, and W for the delta rules
template <int RULE, int P, int COLS> struct KeyColumn {
    pair_t (&x)[COLS][CT / 2];
    const float *A, *q, *decay;            // q, decay: the channels' columns (decay: or one number a token)
    float *wq, *ww, G[COLS];
    size_t stride;
    int cnt, apart, cols;
    template <int T> __device__ __forceinline__ void at() {
        if (T < cnt) {
            float o[COLS];
            if (IS_DELTA<RULE>) row_times<T + 1>(A + T * AP, x, o);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                if (c >= cols) break;
                const float g = VECTOR_DECAY<RULE> ? decay[T * P + c * apart] : decay[T];
                if (RULE != RULE_WKV) G[c] *= g;          // wkv reads the state before its token's decay
                if (IS_DELTA<RULE>) ww[T * stride + c * apart] = get_token<T>(x[c]);
                wq[T * stride + c * apart] = fmaf(q[T * P + c * apart], G[c], IS_DELTA<RULE> ? -o[c] : 0.f);
                if (RULE == RULE_WKV) G[c] *= g;
            }
        }
    }
};

// ---- what a chunk can do without the state before it ------------------------------------------
// ws of a token and head: x = G_t (mLSTM: the sum of its log keeps from the chunk's start), y = what its
// row of k is times when it joins the state (the decay to the chunk's end, the step size), z, w (mLSTM):
// the running maximum of the chunk alone and its row's sum of A.
template <int DP, int RULE>
__global__ void __launch_bounds__(THREADS, 2) chunk_local_kernel(const Args a) {
    cb_pdl_trigger();
    cb_pdl_wait();
    constexpr bool VECTOR = VECTOR_DECAY<RULE>, DELTA = IS_DELTA<RULE>;
    constexpr int P = DP + PAD<RULE>;
    const int r = blockIdx.z, head = blockIdx.y;
    const Piece piece = piece_of(a, r);
    const int row0 = piece.row0 + blockIdx.x * CT, own0 = row0 - piece.shift;
    const int cnt = min(CT, piece.row1 - row0);
    if (cnt <= 0) return;
    extern __shared__ __align__(16) float smem[];
    float* sk = smem;                               // [CT][P]
    float* sq = sk + CT * P;
    float* sw = sq + CT * P;                        // vector decays only
    float* sA = sw + (VECTOR ? CT * P : 0);         // [CT][AP]
    float* sN = sA + CT * AP;                       // delta rules; before that (scalar decays) L
    float* sa = sN + CT * AP;                       // [CT] decay of a token, [CT] beta or step
    float* sb = sa + CT;
    float* sf = sb + CT;                            // [CT] what a row of k is times when it joins the state
    float* part = sf + CT;                          // vector decays: [DP / 16][1 or 2][CT][CT] shares of the dots;
                                                    // then (rules without a sum) [CT][DP + 4] values
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = a.D, E = a.E, H = a.H;
    const int g = head / (H / a.G);

    if (warp == 0) {
        // the chunk's numbers, a token a lane; tokens beyond the portion's end change nothing
        const bool in = lane < cnt;
        const size_t at = (size_t)(row0 + lane) * H + head, own_at = (size_t)(own0 + lane) * H + head;
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
            // (a log gate of -inf lets nothing in; until one does, the maximum is -inf and both are 0)
            const float top = i == -INFINITY ? 0.f : i;
            dec = lane == 0 ? 0.f : expf(f_own + before - top);
            b = in ? expf(i_own - top) : 0.f;
            if (in) a.ws[own_at] = make_float4(f, 0.f, i, 0.f);
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
#pragma unroll 8
            for (int t = 0; t < CT; ++t) {
                const float x = sa[t];
                l = t == lane ? 1.f : l * x;
                sN[t * AP + lane] = t < lane ? 0.f : l;
                if (t <= lane) G *= x;
            }
            if (in) {
                const float to_end = l * (RULE == RULE_DELTA ? 1.f : b);
                sf[lane] = to_end;
                if (RULE == RULE_MLSTM) a.ws[own_at].y = to_end;
                else a.ws[own_at] = make_float4(G, to_end, 0.f, 0.f);
            }
        }
    }
    // (scalar decays: the first warp is at the numbers, a chain of its own, meanwhile)
    if (VECTOR || warp > 0)
    for (int i = VECTOR ? tid : tid - 32; i < CT * (DP / 4); i += VECTOR ? THREADS : THREADS - 32) {
        const int t = i / (DP / 4), d = (i - t * (DP / 4)) * 4;
        const bool in = t < cnt && d < D;
        const float* src = a.qkv + (size_t)(row0 + t) * a.C;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
        *reinterpret_cast<float4*>(sk + t * P + d) = in ? *reinterpret_cast<const float4*>(src + a.k_off + (size_t)g * D + d) : zero;
        *reinterpret_cast<float4*>(sq + t * P + d) = in ? *reinterpret_cast<const float4*>(src + a.q_off + (size_t)g * D + d) : zero;
        if (VECTOR) *reinterpret_cast<float4*>(sw + t * P + d) = in ? *reinterpret_cast<const float4*>(src + a.w_off + (size_t)head * D + d) : one;
    }
    __syncthreads();

    // the dots of the chunk's rows: A, and for the delta rules N
    if (!VECTOR) {
        // rows tr + 8 i against columns tc + 8 j, i >= j (the others lie above the diagonal); four
        // neighbouring lanes share the sum over D, 16 bytes of every 64
        const int share = tid & 3, tr = (tid >> 2) & 7, tc = tid >> 5;
        pair_t qk[10], kk[10];
#pragma unroll
        for (int p = 0; p < 10; ++p) qk[p] = kk[p] = 0;
#pragma unroll 2
        for (int d = 4 * share; d < DP; d += 16) {
            ulonglong2 q[4], k[4], c[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                q[i] = pairs_at(sq + (tr + 8 * i) * P + d);
                if (DELTA) k[i] = pairs_at(sk + (tr + 8 * i) * P + d);
                c[i] = pairs_at(sk + (tc + 8 * i) * P + d);
            }
#pragma unroll
            for (int i = 0, p = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j, ++p) {
                    qk[p] = fma_pair(q[i].x, c[j].x, qk[p]);
                    qk[p] = fma_pair(q[i].y, c[j].y, qk[p]);
                    if (DELTA) {
                        kk[p] = fma_pair(k[i].x, c[j].x, kk[p]);
                        kk[p] = fma_pair(k[i].y, c[j].y, kk[p]);
                    }
                }
        }
#pragma unroll
        for (int i = 0, p = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j, ++p) {     // (what lands above the diagonal is never read)
                float x = pair_sum(qk[p]), y = DELTA ? pair_sum(kk[p]) : 0.f;
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                x += __shfl_xor_sync(0xffffffffu, x, 2);
                if (DELTA) {
                    y += __shfl_xor_sync(0xffffffffu, y, 1);
                    y += __shfl_xor_sync(0xffffffffu, y, 2);
                }
                const int t = tr + 8 * i, at = tc + 8 * j;
                if (share == 0) {
                    const float l = sN[t * AP + at];
                    sA[t * AP + at] = x * l * (DELTA ? 1.f : sb[at]);
                    if (DELTA) sN[t * AP + at] = sb[t] * y * l;
                }
            }
        __syncthreads();
    } else {
        // a column s a lane, 16 channels a warp: the key decays on its way down the rows
        constexpr int SHARE = (DELTA ? 2 : 1) * CT * CT;
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
            float* to = part + (size_t)warp * SHARE;
#pragma unroll 2
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
                to[t * CT + s] = x;
                if (DELTA) to[CT * CT + t * CT + s] = (kk[0] + kk[1]) + (kk[2] + kk[3]);
            }
        }
        __syncthreads();
        for (int i = tid; i < CT * CT; i += THREADS) {
            const int t = i / CT, s = i - t * CT;
            float x = 0.f, y = 0.f;
#pragma unroll
            for (int w = 0; w < DP / 16; ++w) {
                x += part[(size_t)w * SHARE + i];
                if (DELTA) y += part[(size_t)w * SHARE + CT * CT + i];
            }
            sA[t * AP + s] = x;
            if (DELTA) sN[t * AP + s] = sb[t] * y;
        }
        __syncthreads();
    }

    if (RULE == RULE_MLSTM) {
        for (int t = warp; t < cnt; t += THREADS / 32) {
            const float n = cb_warp_sum(lane <= t ? sA[t * AP + lane] : 0.f);
            if (lane == 0) a.ws[(size_t)(own0 + t) * H + head].w = n;
        }
    }
    const size_t first = (size_t)row0 * H + head, own = (size_t)own0 * H + head;      // the chunk's first row: results, workspaces
    // vector decays: keys decayed to the chunk's end, and the whole chunk's decay
    if (VECTOR && tid < D) {
        float to_end = 1.f;
        for (int t = cnt - 1; t >= 0; --t) {
            const float k = sk[t * P + tid] * to_end;
            if (DELTA) a.wk[(own + (size_t)t * H) * D + tid] = k;
            else sk[t * P + tid] = k;               // (its dots have been taken)
            to_end *= sw[t * P + tid];
        }
        a.wg[(chunk_place(own0, r) * H + head) * D + tid] = to_end;
    }
    // the columns: E of v, then (delta rules: W; other vector decays: the decayed queries) D of the keys.
    // Delta rules: two a thread, so that a row of N or A out of shared memory serves both
    constexpr int COLS = DELTA ? 2 : 1;
    auto groups = [](int n) { return (n + COLS - 1) / COLS; };
    const int v_groups = groups(E), k_groups = OWN_Q<RULE> ? groups(D) : 0;
    for (int c = tid; c < v_groups + k_groups; c += THREADS) {
        pair_t x[COLS][CT / 2];
        const bool is_v = c < v_groups;
        const int apart = is_v ? v_groups : k_groups, d = is_v ? c : c - v_groups;
        const int cols = COLS > 1 && d + apart < (is_v ? E : D) ? 2 : 1;
        if (is_v) {
            const float* src = a.qkv + (size_t)row0 * a.C + a.v_off + (size_t)head * E + d;
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                float v[CT];
#pragma unroll
                for (int t = 0; t < CT; ++t) v[t] = t < cnt && i < cols ? src[(size_t)t * a.C + i * apart] : 0.f;
#pragma unroll
                for (int t = 0; t < CT; t += 2) x[i][t / 2] = make_pair_of(v[t], v[t + 1]);
            }
        } else if (DELTA) {
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                const int k = i < cols ? d + i * apart : d;
                float G = 1.f;
#pragma unroll
                for (int t = 0; t < CT; t += 2) {
                    const float ga = G * (VECTOR ? sw[t * P + k] : sa[t]);
                    G = ga * (VECTOR ? sw[(t + 1) * P + k] : sa[t + 1]);
                    x[i][t / 2] = make_pair_of(sk[t * P + k] * ga, sk[(t + 1) * P + k] * G);
                }
            }
        }
        if (DELTA) {
            Substitute<COLS> f{x, sN, sb};
            each_token<0>(f);
        }
        if (is_v) {
            ValueColumn<RULE, COLS> f{x, sA, a.out + first * E + d, DELTA ? a.wu + own * E + d : nullptr,
                                      RULE == RULE_SSD ? a.per_head[head] : 0.f, (size_t)H * E, cnt, apart, cols};
            each_token<0>(f);
        } else {
            KeyColumn<RULE, P, COLS> f{x, sA, sq + d, VECTOR ? sw + d : sa, a.wq + own * D + d,
                                       DELTA ? a.ww + own * D + d : nullptr, {}, (size_t)H * D, cnt, apart, cols};
#pragma unroll
            for (int i = 0; i < COLS; ++i) f.G[i] = 1.f;
            each_token<0>(f);
        }
    }
    if (!DELTA) {
        // what the chunk adds to the state: k^T u, 8 x 8 (4 x 4) sums a thread; 16 operands out of shared
        // memory for 64 multiply-adds
        constexpr int Q = DP / 64;
        const int tx = tid & 15, ty = tid >> 4;
        float* sv = part;
        for (int e0 = 0; e0 < E; e0 += DP) {
            __syncthreads();
            for (int i = tid; i < CT * (DP / 4); i += THREADS) {
                const int t = i / (DP / 4), e = (i % (DP / 4)) * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t < cnt && e0 + e < E) {
                    v = *reinterpret_cast<const float4*>(a.qkv + (size_t)(row0 + t) * a.C + a.v_off + (size_t)head * E + e0 + e);
                    if (!VECTOR) {
                        const float f = sf[t];
                        v = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
                    }
                }
                *reinterpret_cast<float4*>(sv + t * P + e) = v;
            }
            __syncthreads();
            pair_t acc[4 * Q][2 * Q];
#pragma unroll
            for (int i = 0; i < 4 * Q; ++i)
#pragma unroll
                for (int c = 0; c < 2 * Q; ++c) acc[i][c] = 0;
#pragma unroll 2
            for (int t = 0; t < cnt; ++t) {
                float4 k[Q];
                ulonglong2 v[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    k[q] = *reinterpret_cast<const float4*>(sk + t * P + 64 * q + 4 * ty);
                    v[q] = pairs_at(sv + t * P + 64 * q + 4 * tx);
                }
#pragma unroll
                for (int i = 0; i < 4 * Q; ++i) {
                    const float4 kq = k[i / 4];
                    const float x = i % 4 == 0 ? kq.x : i % 4 == 1 ? kq.y : i % 4 == 2 ? kq.z : kq.w;
                    const pair_t f = make_pair_of(x, x);
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        acc[i][2 * q] = fma_pair(f, v[q].x, acc[i][2 * q]);
                        acc[i][2 * q + 1] = fma_pair(f, v[q].y, acc[i][2 * q + 1]);
                    }
                }
            }
            float* to = a.wl + (chunk_place(own0, r) * H + head) * (size_t)D * E;
#pragma unroll
            for (int i = 0; i < 4 * Q; ++i) {
                const int d = 64 * (i / 4) + 4 * ty + i % 4;
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int e = e0 + 64 * q + 4 * tx;
                    if (d < D && e < E)
                        *reinterpret_cast<ulonglong2*>(to + (size_t)d * E + e) = make_ulonglong2(acc[i][2 * q], acc[i][2 * q + 1]);
                }
            }
        }
        if (RULE == RULE_MLSTM && tid < D) {
            float n = 0.f;
            for (int t = 0; t < cnt; ++t) n = fmaf(sk[t * P + tid], sf[t], n);
            a.wn[(chunk_place(own0, r) * H + head) * D + tid] = n;
        }
    }
}

// ---- rules whose write needs no sum over a column: the states, then their part of the results --------
// S as each chunk begins, in the place of what the chunk before left there to add: a thread has four
// entries of S and goes from chunk to chunk, the next chunks' additions asked for ahead.  Bound by the
// bytes of wl both ways.  The last block of a head (mLSTM) takes n and m.
template <int RULE>
__global__ void __launch_bounds__(THREADS) chunk_scan_kernel(const Args a) {
    cb_pdl_trigger();
    cb_pdl_wait();
    const int r = blockIdx.z, head = blockIdx.y;
    const int D = a.D, E = a.E, H = a.H;
    const Piece piece = piece_of(a, r);
    const int own0 = piece.row0 - piece.shift, n = piece.row1 - piece.row0;
    if (n <= 0) return;
    const int chunks = (n + CT - 1) / CT;
    const int slot = a.req_state_slot[r];
    const float* n0 = RULE == RULE_MLSTM ? a.kept + (size_t)r * (H * D + H) : nullptr;
    float m = RULE == RULE_MLSTM ? n0[(size_t)H * D + head] : 0.f;
    // the chunks' numbers, 64 at a time: the decay of the state before a chunk (wkv: a vector, read
    // below), the factor of what it adds, m as it begins
    constexpr int BATCH = 64, AHEAD = 8;
    __shared__ float4 sx[BATCH];
    __shared__ float sg[BATCH], si[BATCH], sm[BATCH];
    auto numbers = [&](int c0) {
        if (RULE == RULE_WKV) return;
        __syncthreads();
        if (threadIdx.x < BATCH && c0 + (int)threadIdx.x < chunks)
            sx[threadIdx.x] = a.ws[(size_t)(own0 + min(n, (c0 + (int)threadIdx.x + 1) * CT) - 1) * H + head];
        __syncthreads();
        if (RULE == RULE_SSD) {
            if (threadIdx.x < BATCH) sg[threadIdx.x] = sx[threadIdx.x].x, si[threadIdx.x] = 1.f;
        } else if (threadIdx.x == 0) {
            for (int k = 0; k < min(BATCH, chunks - c0); ++k) {
                sm[k] = m;
                m = fmaxf(sx[k].x + m, sx[k].z);
            }
        }
        __syncthreads();
        if (RULE == RULE_MLSTM && threadIdx.x < BATCH && c0 + (int)threadIdx.x < chunks) {
            const float4 own = sx[threadIdx.x];
            const float before = sm[threadIdx.x], after = fmaxf(own.x + before, own.z);
            sg[threadIdx.x] = expf(own.x + before - after);
            si[threadIdx.x] = expf(own.z - after);
        }
        __syncthreads();
    };
    const size_t step = (size_t)H * D * E;          // neighbouring chunks of a request are neighbours in wl
    const int i = (blockIdx.x * THREADS + threadIdx.x) * 4, d = i / E;
    const bool mine = i < D * E;
    const bool with_n = RULE == RULE_MLSTM && blockIdx.x == gridDim.x - 1;
    const int dn = threadIdx.x;
    float* S = state_at(a.state, a.slot_stride, slot, a.s_off) + (size_t)head * D * E + i;
    const size_t first = chunk_place(own0, r) * H + head;
    float* at = a.wl + first * (size_t)D * E + i;
    float4 s = mine ? *reinterpret_cast<const float4*>(S) : make_float4(0.f, 0.f, 0.f, 0.f);
    float v = with_n && dn < D ? n0[(size_t)head * D + dn] : 0.f;
    for (int b0 = 0; b0 < chunks; b0 += BATCH) {
        numbers(b0);
        const int b1 = min(chunks, b0 + BATCH);
        for (int c0 = b0; c0 < b1; c0 += AHEAD) {
            float4 x[AHEAD];
            float gw[AHEAD], xn[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
                if (c0 + k < b1) {
                    if (mine) x[k] = *reinterpret_cast<const float4*>(at + (c0 + k) * step);
                    if (RULE == RULE_WKV && mine) gw[k] = a.wg[(first + (size_t)(c0 + k) * H) * D + d];
                    if (with_n && dn < D) xn[k] = a.wn[(first + (size_t)(c0 + k) * H) * D + dn];
                }
#pragma unroll
            for (int k = 0; k < AHEAD; ++k) {
                if (c0 + k >= b1) break;
                const float g = RULE == RULE_WKV ? gw[k] : sg[c0 + k - b0], in = RULE == RULE_MLSTM ? si[c0 + k - b0] : 1.f;
                if (mine) {
                    *reinterpret_cast<float4*>(at + (c0 + k) * step) = s;
                    s = make_float4(fmaf(g, s.x, in * x[k].x), fmaf(g, s.y, in * x[k].y), fmaf(g, s.z, in * x[k].z),
                                    fmaf(g, s.w, in * x[k].w));
                }
                if (with_n) {
                    const size_t place = first + (size_t)(c0 + k) * H;
                    if (dn == 0) a.wm[place] = sm[c0 + k - b0];
                    if (dn < D) {
                        a.wn[place * D + dn] = v;
                        v = fmaf(g, v, in * xn[k]);
                    }
                }
            }
        }
    }
    if (mine) *reinterpret_cast<float4*>(S) = s;
    if (with_n) {
        float* next = a.kept_next != nullptr ? a.kept_next + (size_t)r * (H * D + H) : nullptr;
        if (dn < D) {
            state_at(a.state, a.slot_stride, slot, a.n_off)[(size_t)head * D + dn] = v;
            if (next != nullptr) next[(size_t)head * D + dn] = v;
        }
        if (dn == 0) {
            state_at(a.state, a.slot_stride, slot, a.m_off)[head] = m;
            if (next != nullptr) next[(size_t)H * D + head] = m;
        }
    }
}

// A chunk's queries over the state at its beginning: a warp has 16 tokens, 128 columns, four
// neighbouring ones a lane, and half of the channels; sums of two neighbouring tokens are one
// instruction.  Per channel a lane reads 16 bytes of S, eight channels at once, and 64 of queries for 64
// multiply-adds.
constexpr int OUT_THREADS = 128;
template <int DP, int RULE>
__global__ void __launch_bounds__(OUT_THREADS, 4) chunk_out_kernel(const Args a) {
    cb_pdl_trigger();
    cb_pdl_wait();
    __shared__ __align__(16) float sq[DP * AP];      // [D][CT]: queries, a channel's tokens side by side
    __shared__ __align__(16) float half[2][16][128 + 4];
    const int r = blockIdx.z, head = blockIdx.y;
    const Piece piece = piece_of(a, r);
    const int row0 = piece.row0 + blockIdx.x * CT, own0 = row0 - piece.shift;
    const int cnt = min(CT, piece.row1 - row0);
    if (cnt <= 0) return;
    const int D = a.D, E = a.E, H = a.H, g = head / (H / a.G);
    const int lane = threadIdx.x & 31, group = (threadIdx.x >> 5) & 1, upper = threadIdx.x >> 6, t0 = group * 16;
    for (int i = threadIdx.x; i < CT * (D / 4); i += OUT_THREADS) {
        const int t = i % CT, d = (i / CT) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < cnt)
            q = *reinterpret_cast<const float4*>(OWN_Q<RULE> ? a.wq + ((size_t)(own0 + t) * H + head) * D + d
                                                             : a.qkv + (size_t)(row0 + t) * a.C + a.q_off + (size_t)g * D + d);
        sq[d * AP + t] = q.x; sq[(d + 1) * AP + t] = q.y; sq[(d + 2) * AP + t] = q.z; sq[(d + 3) * AP + t] = q.w;
    }
    __syncthreads();
    const size_t place = chunk_place(own0, r) * H + head;
    // the factors of a token's two shares (what it has within the chunk, what comes from the state), in
    // the lane of the token
    float within = 1.f, before = 1.f;
    {
        const int t = t0 + (lane & 15);
        float4 own = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!VECTOR_DECAY<RULE> && t < cnt) own = a.ws[(size_t)(own0 + t) * H + head];
        if (RULE == RULE_SSD) before = own.x;
        if (RULE == RULE_MLSTM) {
            const float* n = a.wn + place * D;
            float nq = 0.f;
            for (int d = lane >> 4; d < D; d += 2) nq = fmaf(n[d], sq[d * AP + t], nq);
            nq += __shfl_xor_sync(0xffffffffu, nq, 16);
            const float m0 = a.wm[place];
            const float m = fmaxf(own.x + m0, own.z);
            before = expf(own.x + m0 - m);
            within = expf(own.z - m);
            const float low = fmaxf(fabsf(fmaf(before, nq, within * own.w)), expf(-m)) + 1e-6f;
            before /= low;
            within /= low;
        }
    }
    for (int e = lane * 4; e - lane * 4 < E; e += 128) {
        const bool in = e < E;
        const float* S = a.wl + place * (size_t)D * E + e;
        pair_t acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0;
        const int d0 = upper ? D / 8 * 4 : 0, d1 = upper ? D : D / 8 * 4;       // (D: a multiple of 4)
        constexpr int AHEAD = 8;
        for (int db = d0; db < d1; db += AHEAD) {
            float4 s[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
                s[k] = in && db + k < d1 ? *reinterpret_cast<const float4*>(S + (size_t)(db + k) * E) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < AHEAD; ++j) {
                if (db + j >= d1) break;
                const pair_t c[4] = {make_pair_of(s[j].x, s[j].x), make_pair_of(s[j].y, s[j].y), make_pair_of(s[j].z, s[j].z),
                                     make_pair_of(s[j].w, s[j].w)};
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const ulonglong2 q = pairs_at(sq + (db + j) * AP + t0 + 2 * i);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        acc[i][k] = fma_pair(q.x, c[k], acc[i][k]);
                        acc[i + 1][k] = fma_pair(q.y, c[k], acc[i + 1][k]);
                    }
                }
            }
        }
        // The two halves' sums: each warp closes eight of its tokens, and leaves the other eight's shares to the
        // other half's.  What they have within the chunk is asked for first: a load behind each
        // store, which may be to the same place, took the memory's latency 16 times (a quarter of the kernel).
        float4 l[8];
        const int mine0 = upper * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = t0 + mine0 + i;
            l[i] = in && t < cnt ? *reinterpret_cast<const float4*>(a.out + ((size_t)(row0 + t) * H + head) * E + e)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if ((i >= 8) != (upper != 0)) {
                float x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 v = split_pair(acc[i / 2][k]);
                    x[k] = i % 2 ? v.y : v.x;
                }
                *reinterpret_cast<float4*>(&half[group][i][lane * 4]) = make_float4(x[0], x[1], x[2], x[3]);
            }
        __syncthreads();
        auto close = [&](auto first) {
            constexpr int FIRST = decltype(first)::value;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float fw = __shfl_sync(0xffffffffu, within, FIRST + i), fb = __shfl_sync(0xffffffffu, before, FIRST + i);
                float x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 v = split_pair(acc[(FIRST + i) / 2][k]);
                    x[k] = i % 2 ? v.y : v.x;
                }
                const float4 other = *reinterpret_cast<const float4*>(&half[group][FIRST + i][lane * 4]);
                x[0] += other.x; x[1] += other.y; x[2] += other.z; x[3] += other.w;
                const int t = t0 + FIRST + i;
                if (in && t < cnt)
                    *reinterpret_cast<float4*>(a.out + ((size_t)(row0 + t) * H + head) * E + e) =
                        make_float4(fmaf(fb, x[0], fw * l[i].x), fmaf(fb, x[1], fw * l[i].y),
                                    fmaf(fb, x[2], fw * l[i].z), fmaf(fb, x[3], fw * l[i].w));
            }
        };
        if (upper) close(std::integral_constant<int, 8>{});
        else close(std::integral_constant<int, 0>{});
    }
}

// ---- the delta rules: the state from chunk to chunk ---------------------------------------------
// The chain from chunk to chunk is W's rows over S, u, and k^T over u; the queries' rows over S are beside it.
// All of them are bound by the bytes that shared memory hands to registers (56 % of the cycles; fp32 FMA 31 %) and by
// the chain's latencies.  So a thread's piece of a product is up to 8 x 4 numbers (12 reads of 16 bytes for 128
// products), what is left of a sum lies in neighbouring lanes, which halve it among themselves by exchanges (no shares
// in shared memory), S lies there twice, as the chunk begins and as it ends, and a chunk has two barriers: u is
// there; the state is there.  2,048 tokens of 16 heads of 128 with the chunks' numbers, against pieces of 4 x 4, shares
// in shared memory and four barriers: delta 240 -> 233 us, channel delta 328 -> 280; 8 heads 166 -> 143, 214 -> 170.
// The queries' rows beside the chain with 8 columns a block, too: 34.3 -> 35.1 (333 tokens of 8 heads of 128) and
// 25.7 -> 28.3 (300 of 64), where W's rows alone leave a thread a piece of 2 x 4.  What a token has within the chunk, asked
// for before the chunk's barrier: 196 -> 202.
// S's columns lie in shared memory as rows [ET][PS], so that sums over D run over neighbouring pairs; column
// 4 j + i is row i * (ET / 4) + j, and the pitch puts the rows that neighbouring lanes write 128 / ET banks apart.

// SHARES lanes, `apart` from each other, each with its share of the same COUNT sums: share i is left with the
// i-th of SHARES pieces of them, in the first places
template <int COUNT, int SHARES>
__device__ __forceinline__ void shares_summed(float* sum, int share, int apart) {
    if constexpr (SHARES > 1) {
        constexpr int N = COUNT / 2, STEP = SHARES / 2;
        const bool upper = (share & STEP) != 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, upper ? sum[i] : sum[i + N], STEP * apart);
            sum[i] = (upper ? sum[i + N] : sum[i]) + other;
        }
        shares_summed<N, STEP>(sum, share, apart);
    }
}

// COUNT rows [COUNT][DP] over the columns of S, by N threads: a thread's piece is ROWS rows, RG apart, and 4 columns,
// CG apart (in their order in shared memory); eight neighbouring lanes share the sum over D, 128 bytes of a row at a time
template <int DP, int ET, int COUNT, int N>
struct RowsOverState {
    static constexpr int SHARES = 8, CG = ET / 4, PS = DP + 32 / CG, RG = N / (SHARES * CG), ROWS = COUNT / RG;
    static constexpr int SUMS = ROWS * 4, LEFT = SUMS / SHARES;     // left to a lane: 4 or 2 columns of a row
    static_assert(DP % (4 * SHARES) == 0 && (LEFT == 4 || LEFT == 2), "");
    int row, col, x_at, y_at;
    __device__ __forceinline__ explicit RowsOverState(int t) : share(t % SHARES) {
        const int cg = t / SHARES % CG, rg = t / (SHARES * CG);
        row = rg + RG * (share * LEFT / 4);
        col = cg * 4 + share * LEFT % 4;
        x_at = rg * DP + share * 4;
        y_at = cg * PS + share * 4;
    }
    __device__ __forceinline__ void take(const float* rows, const float* S, float (&sum)[SUMS]) const {
        pair_t acc[ROWS][4];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0;
#pragma unroll
        for (int d = 0; d < DP; d += 4 * SHARES) {
            ulonglong2 x[ROWS], y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = pairs_at(S + y_at + CG * j * PS + d);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) x[i] = pairs_at(rows + x_at + RG * i * DP + d);
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fma_pair(x[i].x, y[j].x, acc[i][j]);
                    acc[i][j] = fma_pair(x[i].y, y[j].y, acc[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < SUMS; ++i) sum[i] = pair_sum(acc[i / 4][i % 4]);
        shares_summed<SUMS, SHARES>(sum, share, 1);
    }
private:
    int share;
};

// The operands come by TMA, a box of 32 rows each, that a warp of its own asks for: as asynchronous copies of 16 bytes by
// the threads that compute they were 1,000 to 1,600 of a chunk's 4,650 cycles; by two more warps the pipe that
// serves shared memory was still theirs (237 -> 251 us), and a bulk copy a row costs that warp 60 cycles (401 us).
struct WalkMaps { CUtensorMap q, w, k, u, s; };          // wq, ww, the keys, wu, ws
// 16 columns: the queries' rows over S by four warps of their own, beside both products of the chain, the second of
// which has all eight warps (against four that left the second product for them: 32 x 64 heads, 700 tokens 72.5 ->
// 67.3 us, 16 x 128 heads, 2,048 tokens 200 -> 196, per channel 251 -> 247.7).  8: with W's rows, before them.
// CROWDED: more blocks of heads of 64 than SMs, two to an SM: they hide one another's latencies, and four warps leave the
// second product for the queries' rows.  (The nine warps of a block are three on one of the SM's four quarters, so
// two blocks need at most 96 registers a thread.)  32 heads, 20 portions of 100: the walk 182 us with 104 registers, 168
// with the queries' warps apart, 145 with three blocks and spills, 120 so; 8 portions of 130 75.5, 71.3, 77.7 and 56.0.
template <int ET, bool CROWDED> constexpr int QUERY_THREADS = ET == 16 && !CROWDED ? 128 : 0;
template <int DP, int RULE, int ET, bool CROWDED>
__global__ void __launch_bounds__(THREADS + QUERY_THREADS<ET, CROWDED> + 32, CROWDED ? 2 : 1)
chunk_walk_kernel(const __grid_constant__ WalkMaps maps, const Args a) {
    cb_pdl_trigger();
    cb_pdl_wait();
    constexpr int CG = ET / 4, PS = DP + 32 / CG;
    constexpr bool VECTOR = VECTOR_DECAY<RULE>;
    constexpr bool BESIDE = ET == 16, APART = QUERY_THREADS<ET, CROWDED> > 0;
    // the queries' rows and W's over S, keys, u, the chunk's decays per channel, the tokens' numbers
    constexpr int STAGE = 3 * CT * DP + CT * ET + DP + 4 * CT;
    static_assert(STAGE % 32 == 0 && (2 * ET * PS + CT * ET) % 32 == 0, "boxes begin on 128-byte boundaries");
    // the second product: shares of the chunk's tokens, in lanes MS * CG apart; a thread has four columns and a piece of four
    // channels, of eight warps, or two pieces, DP / 2 apart, of four
    constexpr int PIECES = APART ? 1 : 2;
    constexpr int TS = 4096 / (DP * ET), MS = 32 / (TS * CG), TOKENS = CT / TS;
    static_assert(TS >= 2 && TS <= 8 && DP / 8 == 4 * MS, "the warps cover the state");
    // (no shared variable beside this one: it would come first, and a box's place is a 128-byte boundary)
    extern __shared__ __align__(1024) float walk_smem[];
    float* states = walk_smem;                           // [2][ET][PS]: as the chunk begins, and as it ends
    float* su = states + 2 * ET * PS;                    // [CT][ET]: u as it joins the state
    float* stage = su + CT * ET;                         // [2][STAGE]
    uint64_t* full = reinterpret_cast<uint64_t*>(stage + 2 * STAGE);      // [2]: a stage's copies have landed
    volatile int* abort_flag = reinterpret_cast<volatile int*>(full + 2);
    const int r = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * ET;
    const int tid = threadIdx.x;
    const int D = a.D, E = a.E, H = a.H;
    const int g = head / (H / a.G);
    const Piece piece = piece_of(a, r);
    const int row0 = piece.row0, row1 = piece.row1, shift = piece.shift;
    if (row0 >= row1) return;
    const int slot = a.req_state_slot[r];
    float* state = state_at(a.state, a.slot_stride, slot, a.s_off) + (size_t)head * D * E;
    auto place_of = [](int c) { return (c & 3) * CG + (c >> 2); };
    for (int i = tid; i < DP * ET; i += blockDim.x) {
        const int d = i / ET, c = i - d * ET;
        states[place_of(c) * PS + d] = d < D && col0 + c < E ? state[(size_t)d * E + col0 + c] : 0.f;
    }
    for (int d = D + tid; d < DP; d += blockDim.x) {     // (the boxes bring zeros beyond the sizes; these decays are no box)
        float* sg = stage + 3 * CT * DP + CT * ET;
        sg[d] = sg[STAGE + d] = 0.f;
    }
    if (tid == 0) {
        tc::mbar_init(&full[0], 1);
        tc::mbar_init(&full[1], 1);
        *abort_flag = 0;
        tc::fence_barrier_init();
    }
    __syncthreads();

    if (tid >= THREADS + QUERY_THREADS<ET, CROWDED>) {
        // ---- the loader --------------------------------------------------------------------------------
        const int lane = tid & 31;
        auto landed = [&](int i) {                       // the copies of chunk i
            bool got = false;
            for (uint32_t n = 0; n < tc::WAIT_LIMIT && !got; ++n) got = tc::mbar_try_wait(&full[i & 1], (i >> 1) & 1);
            return got;
        };
        auto fetch = [&](int base, int i) {
            float* rows = stage + (i & 1) * STAGE;
            float* keys = rows + 2 * CT * DP;
            float* u = keys + CT * DP;
            float* gs = u + CT * ET;
            const int cnt = min(CT, row1 - base);
            uint64_t* bar = &full[i & 1];
            if (tc::elect_one()) {
                tc::mbar_expect_tx(bar, 4 * (3 * CT * DP + CT * ET + (VECTOR ? D : 4 * CT)));
                tc::tma_load_3d(rows + CT * DP, &maps.w, bar, 0, head, base - shift);
                tc::tma_load_3d(u, &maps.u, bar, col0, head, base - shift);
                tc::tma_load_3d(keys, &maps.k, bar, 0, VECTOR ? head : g, VECTOR ? base - shift : base);
                tc::tma_load_3d(rows, &maps.q, bar, 0, head, base - shift);
                if (!VECTOR) tc::tma_load_3d(gs + DP, &maps.s, bar, 0, head, base - shift);
                else asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                  ::"r"(tc::smem_u32(gs)), "l"(a.wg + (chunk_place(base - shift, r) * H + head) * D), "r"(4 * D),
                                  "r"(tc::smem_u32(bar)) : "memory");
            }
            __syncwarp();
            if (cnt < CT) {
                // a portion's last chunk: what lies behind its rows is another's, or nothing, and must not count
                landed(i);
                for (int x = cnt * DP + lane; x < CT * DP; x += 32) rows[x] = rows[CT * DP + x] = keys[x] = 0.f;
                for (int x = cnt * ET + lane; x < CT * ET; x += 32) u[x] = 0.f;
                if (!VECTOR && lane >= cnt) *reinterpret_cast<float4*>(gs + DP + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        fetch(row0, 0);
        int sent = 1;
        for (int base = row0; base < row1; base += CT) {
            __syncthreads();                             // the chunk's first barrier: the other stage is free
            if (base + CT < row1) fetch(base + CT, sent), ++sent;
        }
        if (*abort_flag)                                 // no copy is left in flight
            for (int i = max(0, sent - 2); i < sent; ++i) landed(i);
        __syncthreads();
        return;
    }
    RowsOverState<DP, ET, BESIDE ? CT : 2 * CT, THREADS> first(tid);
    RowsOverState<DP, ET, CT, THREADS / 2> queries(tid % (THREADS / 2));
    // the state's part: a share of the tokens, channels ud + DP / 2 i, columns 4 uc + c
    const int lane = tid & 31, uc = lane % CG, part = lane / (CG * MS);
    const int ud = (tid / 32 % (APART ? 8 : 4) * MS + lane / CG % MS) * 4;
    int buf = 0;
    uint32_t phase = 0;
    for (int base = row0; base < row1; base += CT, phase ^= buf, buf ^= 1) {
        const int cnt = min(CT, row1 - base);
        const float* rows = stage + buf * STAGE;
        const float* keys = rows + 2 * CT * DP;
        const float* u = keys + CT * DP;
        const float* sg = u + CT * ET;
        const float* S = states + buf * ET * PS;
        const float4* nums = reinterpret_cast<const float4*>(sg + DP);
        // what a token has within the chunk, and with the state's share added
        auto out_at = [&](int t, int c) { return a.out + ((size_t)(base + t) * H + head) * E + col0 + c; };
        auto within = [&](bool has, int t, int c, float* to, int n) {
#pragma unroll
            for (int k = 0; k < n; k += 2) {
                const float2 l = has ? *reinterpret_cast<const float2*>(out_at(t, c + k)) : make_float2(0.f, 0.f);
                to[k] = l.x; to[k + 1] = l.y;
            }
        };
        auto put = [&](int t, int c, const float* l, const float* sum, int n) {
#pragma unroll
            for (int k = 0; k < n; k += 2)
                *reinterpret_cast<float2*>(out_at(t, c + k)) = make_float2(l[k] + sum[k], l[k + 1] + sum[k + 1]);
        };
        float local[4];
        const bool first_out = !BESIDE && first.row < cnt && col0 + first.col < E;
        if (!BESIDE) within(first_out, first.row, first.col, local, first.LEFT);
        // the state is there, and the other stage is free; the chunk's operands are there
        __syncthreads();
        if (!tc::mbar_wait(&full[buf], phase, abort_flag) && !*abort_flag)
            tc::give_up(abort_flag, a.status, tc::ST_EPILOGUE_TIMEOUT);      // (the rest is computed from what there is)
        if (APART && tid >= THREADS) {
            const bool has = queries.row < cnt && col0 + queries.col < E;
            within(has, queries.row, queries.col, local, queries.LEFT);
            float sum[queries.SUMS];
            queries.take(rows, S, sum);
            if (has) put(queries.row, queries.col, local, sum, queries.LEFT);
            continue;
        }
        {
            float sum[first.SUMS];
            first.take(rows + (BESIDE ? CT * DP : 0), S, sum);
            const int t = first.row - (BESIDE ? 0 : CT);
            if (t >= 0) {
                const float f = VECTOR ? 1.f : nums[t].y;
#pragma unroll
                for (int k = 0; k < first.LEFT; k += 2) {
                    const float2 own = *reinterpret_cast<const float2*>(u + t * ET + first.col + k);
                    *reinterpret_cast<float2*>(su + t * ET + first.col + k) =
                        make_float2(f * (own.x - sum[k]), f * (own.y - sum[k + 1]));
                }
            } else if (first_out) {
                put(first.row, first.col, local, sum, first.LEFT);
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");      // (the loader is at its copies)
        if (!APART && tid >= THREADS / 2) {
            if (BESIDE) {
                const bool has = queries.row < cnt && col0 + queries.col < E;
                within(has, queries.row, queries.col, local, queries.LEFT);
                float sum[queries.SUMS];
                queries.take(rows, S, sum);
                if (has) put(queries.row, queries.col, local, sum, queries.LEFT);
            }
        } else {
            pair_t x[PIECES][4][2];
#pragma unroll
            for (int c = 0; c < 4 * PIECES; ++c) x[c / 4][c % 4][0] = x[c / 4][c % 4][1] = 0;
#pragma unroll
            for (int i = 0; i < TOKENS; ++i) {
                const int t = part * TOKENS + i;
                const ulonglong2 k0 = pairs_at(keys + t * DP + ud), k1 = pairs_at(keys + t * DP + (PIECES - 1) * (DP / 2) + ud);
                const float4 v = *reinterpret_cast<const float4*>(su + t * ET + uc * 4);
                const pair_t f[4] = {make_pair_of(v.x, v.x), make_pair_of(v.y, v.y), make_pair_of(v.z, v.z), make_pair_of(v.w, v.w)};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    x[0][c][0] = fma_pair(k0.x, f[c], x[0][c][0]);
                    x[0][c][1] = fma_pair(k0.y, f[c], x[0][c][1]);
                    if constexpr (!APART) {
                        x[1][c][0] = fma_pair(k1.x, f[c], x[1][c][0]);
                        x[1][c][1] = fma_pair(k1.y, f[c], x[1][c][1]);
                    }
                }
            }
            // the tokens' shares: a piece of the channels to each half of the lanes (two pieces), then half of its columns
            float sum[16 * PIECES];
#pragma unroll
            for (int i = 0; i < 8 * PIECES; ++i) {
                const float2 v = split_pair(x[i / 8][i / 2 % 4][i % 2]);
                sum[2 * i] = v.x; sum[2 * i + 1] = v.y;
            }
            shares_summed<16 * PIECES, TS>(sum, part, CG * MS);
            constexpr int COLS = 4 * PIECES / TS, SPLIT = TS / PIECES;          // lanes that share a piece's columns
            const int d = ud + (part / SPLIT) * (DP / 2), c0 = uc * 4 + part % SPLIT * COLS;
            const float g_end = VECTOR ? 1.f : nums[cnt - 1].x;
            const float4 own = *reinterpret_cast<const float4*>(sg + d);
            float* next = states + (buf ^ 1) * ET * PS;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const int at = place_of(c0 + c) * PS + d;
                float4 p = *reinterpret_cast<const float4*>(S + at);
                p.x = fmaf(VECTOR ? own.x : g_end, p.x, sum[4 * c]);
                p.y = fmaf(VECTOR ? own.y : g_end, p.y, sum[4 * c + 1]);
                p.z = fmaf(VECTOR ? own.z : g_end, p.z, sum[4 * c + 2]);
                p.w = fmaf(VECTOR ? own.w : g_end, p.w, sum[4 * c + 3]);
                *reinterpret_cast<float4*>(next + at) = p;
            }
        }
    }
    __syncthreads();
    if (APART && tid >= THREADS) return;
    for (int i = tid; i < DP * ET; i += THREADS) {
        const int d = i / ET, c = i - d * ET;
        if (d < D && col0 + c < E) state[(size_t)d * E + col0 + c] = states[buf * ET * PS + place_of(c) * PS + d];
    }
}

// (`configured`: a kernel's own, so that only its first launch asks)
template <typename K>
int allow_smem(K kernel, size_t smem, bool& configured) {
    if (configured || smem <= 48 * 1024) return 0;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    configured = e == cudaSuccess;
    return (int)e;
}

template <int DP, int RULE, int ET, bool CROWDED = false>
int launch_walk(const Args& a, int n_requests, cudaStream_t s) {
    constexpr size_t bytes = sizeof(float) * (2 * ET * (DP + 128 / ET) + CT * ET + 2 * (3 * CT * DP + CT * ET + DP + 4 * CT)) + 32;
    static_assert(bytes <= 226 * 1024, "a block's shared memory");
    static bool configured = false;
    const int rc = allow_smem(chunk_walk_kernel<DP, RULE, ET, CROWDED>, bytes, configured);
    if (rc) return rc;
    WalkMaps maps;
    const uint64_t width = (uint64_t)a.H * a.D;
    if (!tc::make_map_heads_f32(&maps.q, a.wq, a.piece_rows, a.H, a.D, width, DP, CT) ||
        !tc::make_map_heads_f32(&maps.w, a.ww, a.piece_rows, a.H, a.D, width, DP, CT) ||
        !(VECTOR_DECAY<RULE> ? tc::make_map_heads_f32(&maps.k, a.wk, a.piece_rows, a.H, a.D, width, DP, CT)
                             : tc::make_map_heads_f32(&maps.k, a.qkv + a.k_off, a.rows, a.G, a.D, a.C, DP, CT)) ||
        !tc::make_map_heads_f32(&maps.u, a.wu, a.piece_rows, a.H, a.E, (uint64_t)a.H * a.E, ET, CT) ||
        !tc::make_map_heads_f32(&maps.s, a.ws, a.piece_rows, a.H, 4, (uint64_t)a.H * 4, 4, CT))
        return CB_ERR_UNSUPPORTED;
    const dim3 grid(n_requests, a.H, (a.E + ET - 1) / ET);
    cb_launch(chunk_walk_kernel<DP, RULE, ET, CROWDED>, grid, dim3(THREADS + QUERY_THREADS<ET, CROWDED> + 32), bytes, s, maps, a);
    return cb_last_error();
}

constexpr long CROWD = 148;          // blocks of the walk's 16 columns: beyond one an SM two share it

template <int DP, int RULE>
int launch_chunks(const Args& a, int n_requests, int max_new, cudaStream_t s) {
    constexpr int P = DP + PAD<RULE>;
    // the shares of the dots, then the values (rules without a sum)
    constexpr int part = VECTOR_DECAY<RULE> ? (DP / 16) * (IS_DELTA<RULE> ? 2 : 1) * CT * CT : 0;
    constexpr int values = IS_DELTA<RULE> ? 0 : CT * P;
    constexpr size_t bytes = sizeof(float) * ((VECTOR_DECAY<RULE> ? 3 : 2) * CT * P + 2 * CT * AP + 3 * CT
                                              + (part > values ? part : values));
    static_assert(bytes <= 227 * 1024, "a block's shared memory");
    static bool configured = false;
    int rc = allow_smem(chunk_local_kernel<DP, RULE>, bytes, configured);
    if (rc) return rc;
    const dim3 grid((max_new + CT - 1) / CT, a.H, n_requests);
    cb_launch(chunk_local_kernel<DP, RULE>, grid, dim3(THREADS), bytes, s, a);
    rc = cb_last_error();
    if (rc) return rc;
    if constexpr (IS_DELTA<RULE>) {
        // few heads: half the columns a block, so that twice as many SMs have one (8 heads of 128 x 128)
        const long blocks = (long)n_requests * a.H * ((a.E + 15) / 16);
        if (blocks <= 74) return launch_walk<DP, RULE, 8>(a, n_requests, s);
        if constexpr (DP == 64)
            if (blocks > CROWD) return launch_walk<DP, RULE, 16, true>(a, n_requests, s);
        return launch_walk<DP, RULE, 16>(a, n_requests, s);
    } else {
        cb_launch(chunk_scan_kernel<RULE>, dim3((a.D * a.E / 4 + THREADS - 1) / THREADS, a.H, n_requests), dim3(THREADS), 0,
                  s, a);
        rc = cb_last_error();
        if (rc) return rc;
        cb_launch(chunk_out_kernel<DP, RULE>, grid, dim3(OUT_THREADS), 0, s, a);
        return cb_last_error();
    }
}

}  // namespace

// The rules and their operands are those of cb_matrix_memory (recurrent.cu); max_new: the most tokens a
// request brings.  The portions are taken in slices of `limit` tokens of every request (a multiple of 32, or
// at least max_new: one slice), one after the other through the state, with the same bits whatever limit
// is.  Workspaces, fp32, those the rule needs, rows being the slice's (no more than the step's, nor than
// requests * limit): wq (delta, channel, wkv), ww (delta, channel), wk (channel) [rows][H][D], wu (delta, channel)
// [rows][H][E], ws [rows][H][4]; with chunks = rows / 32 + requests: wg (wkv, channel) and wn (mLSTM)
// [chunks][H][D], wm (mLSTM) [chunks][H], wl (mLSTM, wkv, state space) [chunks][H][D][E]; kept_room (mLSTM in
// several slices) [2][requests][H*D + H].
CB_EXPORT int cb_matrix_memory_chunks(int rule, const float* qkv, int C, int q_off, int k_off, int v_off,
                                      const float* sc0, const float* sc1, const int* req_row_start,
                                      const int* req_state_slot, void* state, long slot_stride, long s_off,
                                      long n_off, long m_off, float* out, int n_requests, int max_new, int n_heads,
                                      int n_qk_heads, int key_dim, int value_dim, int w_off, const float* per_head,
                                      const float* kept, int limit, float* kept_room, float* wq, float* ww, float* wk, float* wu, float* ws,
                                      float* wg, float* wl, float* wn, float* wm, int rows, int piece_rows, int* status,
                                      void* stream) {
    if (n_requests <= 0 || max_new <= 0) return 0;
    const bool vector = rule == RULE_WKV || rule == RULE_CHANNEL;
    if (n_heads % n_qk_heads != 0 || key_dim > 128 || n_requests > 65535 || n_heads > 65535
        || ((C | q_off | k_off | v_off | key_dim | value_dim | (vector ? w_off : 0)) & 3) != 0
        || ((s_off | slot_stride) & 15) != 0 || (((uintptr_t)state | (uintptr_t)qkv | (uintptr_t)out) & 15) != 0)
        return CB_ERR_UNSUPPORTED;
    if ((rule == RULE_WKV || rule == RULE_SSD) && per_head == nullptr) return CB_ERR_UNSUPPORTED;
    if (rule == RULE_MLSTM && (kept == nullptr || (limit < max_new && kept_room == nullptr))) return CB_ERR_UNSUPPORTED;
    if (limit <= 0 || (limit < max_new && limit % CT != 0)) return CB_ERR_UNSUPPORTED;
    Args a;
    a.qkv = qkv; a.C = C; a.q_off = q_off; a.k_off = k_off; a.v_off = v_off; a.w_off = w_off;
    a.sc0 = sc0; a.sc1 = sc1; a.req_row_start = req_row_start; a.req_state_slot = req_state_slot;
    a.state = (unsigned char*)state; a.slot_stride = slot_stride; a.s_off = s_off; a.n_off = n_off; a.m_off = m_off;
    a.out = out; a.H = n_heads; a.G = n_qk_heads; a.D = key_dim; a.E = value_dim;
    a.per_head = per_head; a.kept = kept;
    a.wq = wq; a.ww = ww; a.wk = wk; a.wu = wu; a.wg = wg; a.wl = wl; a.wn = wn; a.wm = wm; a.ws = reinterpret_cast<float4*>(ws);
    cudaStream_t s = (cudaStream_t)stream;
    a.limit = limit;
    a.rows = rows; a.piece_rows = piece_rows;
    a.status = status;
    const size_t kept_size = (size_t)n_requests * n_heads * (key_dim + 1);
    for (int skip = 0, slice = 0; skip < max_new; skip += limit, ++slice) {
        a.skip = skip;
        const int most = max_new - skip < limit ? max_new - skip : limit;
        a.kept_next = rule == RULE_MLSTM && skip + most < max_new ? kept_room + (slice & 1) * kept_size : nullptr;
        int rc = CB_ERR_UNSUPPORTED;
#define CB_CHUNKS(RR)                                                                                       \
        if (rule == RR)                                                                                     \
            rc = key_dim <= 64 ? launch_chunks<64, RR>(a, n_requests, most, s)                              \
                               : launch_chunks<128, RR>(a, n_requests, most, s)
        CB_CHUNKS(RULE_DELTA);
        CB_CHUNKS(RULE_MLSTM);
        CB_CHUNKS(RULE_WKV);
        CB_CHUNKS(RULE_SSD);
        CB_CHUNKS(RULE_CHANNEL);
#undef CB_CHUNKS
        if (rc) return rc;
        a.kept = a.kept_next;
    }
    return 0;
}
