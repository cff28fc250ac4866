// Paged attention of the 32-bit path over tiles of keys, all in fp32 on CUDA cores.
//
// A block takes 32 (or 16) packed rows of one request and one key/value head, rows being (position, head
// of the group) pairs, and walks the keys in tiles: scores as a product of row and key tiles, a running
// maximum and sum a row, probabilities through shared memory, then the product with the values.  A key
// read from memory serves all the block's rows; the one-warp-a-row kernels (attention_generic.cu,
// sink_attention.cu) read it once a row and reduce every score over a warp, which bounds them: 700 tokens
// of 12 heads of 64: 909 us there, 71 here; a token each of 24 requests behind 3,800 keys, 8 heads of 128:
// 7.7 ms a layer there, 0.63 here.
//
// A row's result is a function of its own query and keys: tiles begin at multiples of the tile's size
// from position 0, a score is one sum over the features in a fixed order, a tile's probabilities are
// added in one order, values in ascending position; a tile in which a row sees nothing leaves its
// numbers as they are.  So a row has the same bits however a prompt was cut and whatever the block's
// other rows are, and decoded tokens run the same arithmetic.  Keys a row does not see count for nothing
// whatever their values hold (they are not multiplied by zero).
//
// Sizes: key and value sizes up to 256 that are multiples of 4, rows of whole 16-byte pieces, any page
// size; window, chunks, kept first tokens, a sink, a gate, an output scale as in sink_attention.cu.
#define CB_PDL_BIT 8      // this file's bit in CRUCIBLE_PDL (shared with attention_generic.cu)
#include <type_traits>
#include "common.cuh"

namespace {

struct Params {
    const float* q;
    int q_stride;
    const float* gate;
    int gate_stride;
    float* out;
    int out_stride;
    const float *k_cache, *v_cache, *sinks;
    const int *req_row_start, *req_first_pos, *block_table;
    int table_stride, n_heads, n_kv_heads, n_rep, key_dim, value_dim, page_tokens;
    float scale;
    int window, chunked, keep_first;
    float out_scale;
    int gate_per_head;
};

typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t fma_pair(pair_t a, pair_t b, pair_t c) {
    pair_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ pair_t both(float x) {
    pair_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ float2 split_pair(pair_t p) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ ulonglong2 pairs_at(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ void cp16(float* smem, const float* gmem) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// keys of a tile: a function of the row sizes alone (see above)
template <int DP> constexpr int TILE = DP <= 128 ? 64 : 32;
template <int DP, int QR> constexpr size_t SMEM_FLOATS =
    (size_t)QR * (DP + 4) + 2 * (size_t)TILE<DP> * (DP + 4) + (size_t)QR * (TILE<DP> + 4) + 2 * (size_t)TILE<DP>;

// DP: both sizes padded; QR: packed rows of a block, 16 or 32.  Thread (ty, tx) of TY x 16 has the rows
// ty + TY i; of the scores the keys tx + 16 j, of the output the features 4 tx + 64 c ...
template <int DP, int QR, int THREADS>
__global__ void __launch_bounds__(THREADS, (DP <= 64 ? 512 : 256) / THREADS) attention_f32_kernel(const Params p) {
    cb_pdl_trigger();
    cb_pdl_wait();
    constexpr int P = DP + 4, KT = TILE<DP>, PP = KT + 4, TY = THREADS / 16, NR = QR / TY, NK = KT / 16, NC = DP / 64;
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                  // [QR][P]
    float* sk = sq + QR * P;           // [KT][P]
    float* sv = sk + KT * P;           // [KT][P]
    float* sp = sv + KT * P;           // [QR][PP] probabilities, -1 for a key the row does not see
    int* srow = reinterpret_cast<int*>(sp + QR * PP);      // [2][KT] where a tile's keys lie
    const int req = blockIdx.z, kvh = blockIdx.y;
    const int row_base = p.req_row_start[req];
    const int n_rows = (p.req_row_start[req + 1] - row_base) * p.n_rep;
    const int tiles = (n_rows + QR - 1) / QR;
    if ((int)blockIdx.x >= tiles) return;
    const int r0 = (tiles - 1 - (int)blockIdx.x) * QR;          // the longest rows first
    const int first_pos = p.req_first_pos[req];
    const int* table = p.block_table + (size_t)req * p.table_stride;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int D = p.key_dim, E = p.value_dim;

    for (int i = tid; i < QR * (DP / 4); i += THREADS) {
        const int r = i / (DP / 4), d = (i % (DP / 4)) * 4, row = r0 + r;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n_rows && d < D)
            x = *reinterpret_cast<const float4*>(p.q + (size_t)(row_base + row / p.n_rep) * p.q_stride +
                                                 (size_t)(kvh * p.n_rep + row % p.n_rep) * D + d);
        *reinterpret_cast<float4*>(sq + r * P + d) = x;
    }
    auto low = [&](int pos) {
        return p.window <= 0 ? 0 : p.chunked ? pos - pos % p.window : max(0, pos - p.window + 1);
    };
    int pos[NR], lo[NR], kept[NR];
    bool real[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int row = r0 + ty + TY * i;
        real[i] = row < n_rows;
        pos[i] = first_pos + min(row, n_rows - 1) / p.n_rep;
        lo[i] = low(pos[i]);
        kept[i] = min(p.keep_first, lo[i]);
    }
    // the block's keys: tiles of the kept first tokens, then from the first row's first key on
    const int last_pos = first_pos + min(n_rows - 1, r0 + QR - 1) / p.n_rep;
    const int first_key = low(first_pos + r0 / p.n_rep), key_lo = first_key / KT * KT;
    const int kept_tiles = p.window > 0 ? min((p.keep_first + KT - 1) / KT, key_lo / KT) : 0;
    const int n_tiles = kept_tiles + (last_pos - key_lo) / KT + 1;
    auto tile_key0 = [&](int j) { return j < kept_tiles ? j * KT : key_lo + (j - kept_tiles) * KT; };
    // Where a tile's keys lie: the row of the pool's rows of this head, a key a thread, looked up a tile ahead (by every
    // piece of 16 bytes for itself, behind a division and a dependent load each, the two fetches of a tile took
    // a third of its time).  Keys that none of the block's rows sees (behind its last position, ahead of its windows)
    // have none: they are zeros and not read, their page may have been given back.
    auto place = [&](int j) {
        const int key = tile_key0(j) + tid;
        if (key > last_pos || (key < first_key && key >= p.keep_first)) return -1;
        const int page = table[key / p.page_tokens];
        return (page * p.n_kv_heads + kvh) * p.page_tokens + key % p.page_tokens;
    };
    auto fetch = [&](int j, const float* cache, int n, float* to) {
        const int* rows = srow + (j & 1) * KT;
#pragma unroll 4
        for (int i = tid; i < KT * (DP / 4); i += THREADS) {
            const int t = i / (DP / 4), d = (i % (DP / 4)) * 4, row = rows[t];
            if (row >= 0 && d < n) cp16(to + t * P + d, cache + (size_t)row * n + d);
            else *reinterpret_cast<float4*>(to + t * P + d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        cp_commit();
    };
    if (tid < KT) srow[tid] = place(0);
    __syncthreads();
    float m[NR], l[NR];
    pair_t acc[NR][2 * NC];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * NC; ++c) acc[i][c] = 0;
    }
    fetch(0, p.k_cache, D, sk);
    fetch(0, p.v_cache, E, sv);
    for (int j = 0; j < n_tiles; ++j) {
        const int key0 = tile_key0(j);
        const int ahead = tid < KT && j + 1 < n_tiles ? place(j + 1) : -1;
        cp_wait<1>();                  // the tile's keys
        __syncthreads();
        pair_t s[NR][NK];
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
            for (int k = 0; k < NK; ++k) s[i][k] = 0;
#pragma unroll 4
        for (int d = 0; d < DP; d += 4) {
            ulonglong2 x[NR], y[NK];
#pragma unroll
            for (int i = 0; i < NR; ++i) x[i] = pairs_at(sq + (ty + TY * i) * P + d);
#pragma unroll
            for (int k = 0; k < NK; ++k) y[k] = pairs_at(sk + (tx + 16 * k) * P + d);
#pragma unroll
            for (int i = 0; i < NR; ++i)
#pragma unroll
                for (int k = 0; k < NK; ++k) {
                    s[i][k] = fma_pair(x[i].x, y[k].x, s[i][k]);
                    s[i][k] = fma_pair(x[i].y, y[k].y, s[i][k]);
                }
        }
        bool whole = true;             // every row sees every key of the tile
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            float v[NK], top = -INFINITY;
            bool seen[NK];
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                const int key = key0 + tx + 16 * k;
                seen[k] = key <= pos[i] && (key >= lo[i] || key < kept[i]);
                const float2 h = split_pair(s[i][k]);
                v[k] = (h.x + h.y) * p.scale;
                if (seen[k]) top = fmaxf(top, v[k]);
                whole = whole && seen[k];
            }
#pragma unroll
            for (int x = 1; x < 16; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[i], top);
            const float corr = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                const float e = seen[k] ? expf(v[k] - m_new) : 0.f;
                sum += e;
                sp[(ty + TY * i) * PP + tx + 16 * k] = seen[k] ? e : -1.f;
            }
#pragma unroll
            for (int x = 1; x < 16; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[i] = fmaf(l[i], corr, sum);
            m[i] = m_new;
            const pair_t f = both(corr);
#pragma unroll
            for (int c = 0; c < 2 * NC; ++c) acc[i][c] = fma_pair(acc[i][c], f, 0);
        }
        if (tid < KT) srow[((j + 1) & 1) * KT + tid] = ahead;
        whole = __syncthreads_and(whole);        // the keys have been read, the probabilities are written
        if (j + 1 < n_tiles) fetch(j + 1, p.k_cache, D, sk);
        else cp_commit();
        cp_wait<1>();                  // the tile's values
        __syncthreads();
        if (whole) {
#pragma unroll 2
            for (int k = 0; k < KT; k += 4) {
                float4 w[NR];
#pragma unroll
                for (int i = 0; i < NR; ++i) w[i] = *reinterpret_cast<const float4*>(sp + (ty + TY * i) * PP + k);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    ulonglong2 v[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c) v[c] = pairs_at(sv + (k + e) * P + 4 * tx + 64 * c);
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        const pair_t f = both(e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w);
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            acc[i][2 * c] = fma_pair(f, v[c].x, acc[i][2 * c]);
                            acc[i][2 * c + 1] = fma_pair(f, v[c].y, acc[i][2 * c + 1]);
                        }
                    }
                }
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < KT; ++k) {
                ulonglong2 v[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) v[c] = pairs_at(sv + k * P + 4 * tx + 64 * c);
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const float w = sp[(ty + TY * i) * PP + k];
                    if (w < 0.f) continue;                      // not seen (a NaN is)
                    const pair_t f = both(w);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        acc[i][2 * c] = fma_pair(f, v[c].x, acc[i][2 * c]);
                        acc[i][2 * c + 1] = fma_pair(f, v[c].y, acc[i][2 * c + 1]);
                    }
                }
            }
        }
        __syncthreads();               // the values and the probabilities have been read
        if (j + 1 < n_tiles) fetch(j + 1, p.v_cache, E, sv);
        else cp_commit();
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        if (!real[i]) continue;
        const int row = r0 + ty + TY * i;
        const int t = row_base + row / p.n_rep, h = kvh * p.n_rep + row % p.n_rep;
        float corr = 1.f, sum = l[i];
        if (p.sinks != nullptr) {
            const float sk_ = p.sinks[h], m_new = fmaxf(m[i], sk_);
            corr = expf(m[i] - m_new);
            sum = fmaf(sum, corr, expf(sk_ - m_new));
        }
        const float inv = corr / sum;
        const float* gate = p.gate != nullptr
            ? p.gate + (size_t)t * p.gate_stride + (p.gate_per_head ? (size_t)h : (size_t)h * E) : nullptr;
        float* out = p.out + (size_t)t * p.out_stride + (size_t)h * E;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = 4 * tx + 64 * c;
            if (d >= E) continue;
            const float2 a = split_pair(acc[i][2 * c]), b = split_pair(acc[i][2 * c + 1]);
            float o[4] = {a.x * inv, a.y * inv, b.x * inv, b.y * inv};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (gate != nullptr) o[e] *= 1.0f / (1.0f + expf(-gate[p.gate_per_head ? 0 : d + e]));
                o[e] *= p.out_scale;
            }
            *reinterpret_cast<float4*>(out + d) = make_float4(o[0], o[1], o[2], o[3]);
        }
    }
}

template <int DP, int QR, int THREADS>
int launch(const Params& p, int n_requests, int max_new, cudaStream_t s) {
    constexpr size_t bytes = SMEM_FLOATS<DP, QR> * sizeof(float);
    static_assert(bytes <= 227 * 1024, "a block's shared memory");
    static bool configured = false;
    if (!configured && bytes > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<DP, QR, THREADS>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const dim3 grid((max_new * p.n_rep + QR - 1) / QR, p.n_kv_heads, n_requests);
    cb_launch(attention_f32_kernel<DP, QR, THREADS>, grid, dim3(THREADS), bytes, s, p);
    return cb_last_error();
}

}  // namespace

// warps: of a block of 32 rows, 8 or 4; the same bits either way.
CB_EXPORT int cb_attention_f32(const float* q, int q_stride, const float* gate, int gate_stride, float* out,
                               int out_stride, const float* k_cache, const float* v_cache, const float* sinks,
                               const int* req_row_start, const int* req_first_pos, const int* block_table,
                               int table_stride, int n_requests, int max_new, int n_heads, int n_kv_heads,
                               int key_dim, int value_dim, int page_tokens, float scale, int window, int chunked,
                               int keep_first, float out_scale, int gate_per_head, int warps, void* stream) {
    if (n_requests <= 0 || max_new <= 0) return 0;
    const int most = key_dim > value_dim ? key_dim : value_dim;
    if (n_heads % n_kv_heads != 0 || most > 256 || ((key_dim | value_dim | q_stride | out_stride) & 3) != 0 ||
        ((((uintptr_t)q) | ((uintptr_t)out) | ((uintptr_t)k_cache) | ((uintptr_t)v_cache)) & 15) != 0 ||
        n_requests > 65535 || n_kv_heads > 65535)
        return CB_ERR_UNSUPPORTED;
    Params p;
    p.q = q; p.q_stride = q_stride; p.gate = gate; p.gate_stride = gate_stride; p.out = out; p.out_stride = out_stride;
    p.k_cache = k_cache; p.v_cache = v_cache; p.sinks = sinks;
    p.req_row_start = req_row_start; p.req_first_pos = req_first_pos; p.block_table = block_table;
    p.table_stride = table_stride; p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.n_rep = n_heads / n_kv_heads;
    p.key_dim = key_dim; p.value_dim = value_dim; p.page_tokens = page_tokens; p.scale = scale;
    p.window = window; p.chunked = window > 0 ? chunked : 0; p.keep_first = window > 0 ? keep_first : 0;
    p.out_scale = out_scale; p.gate_per_head = gate_per_head;
    cudaStream_t s = (cudaStream_t)stream;
    const bool few = max_new * p.n_rep <= 16;
    // Blocks of 32 rows: two or more to an SM, so that one's barriers and exponentials run beside another's products,
    // and twice as many to deal out where the longest walks eleven tiles and the average six.  us with 64 rows and eight
    // warps / 32 and four / 32 and eight: 700 tokens of 12 heads of 64 (264 blocks of 32) 76 / 71 / 78, 2,000 of 8 heads of 64
    // (504) 293 / 242 / 277, of 128 on 2 (500) 314 / 310 / 443; 300 of 8 heads of 128 on 2 (76) 58 / 45 / 44.
#define CB_F32_ATTENTION(DD)                                           \
    return few ? launch<DD, 16, 256>(p, n_requests, max_new, s)        \
           : warps == 8 ? launch<DD, 32, 256>(p, n_requests, max_new, s) \
                           : launch<DD, 32, 128>(p, n_requests, max_new, s)
    if (most <= 64) CB_F32_ATTENTION(64);
    if (most <= 128) CB_F32_ATTENTION(128);
    CB_F32_ATTENTION(256);
#undef CB_F32_ATTENTION
}
