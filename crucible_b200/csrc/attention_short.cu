// Attention of single decoded tokens over a short paged context, bfloat16: a block per request and
// key/value head, its warps side by side over the keys, 32 a warp and pass, and one barrier.
//
// What decides such a launch is its chain of round trips, not its bytes (256 keys of 64 features are 64 KB):
// the split kernels (attention_decode_tcgen05.cu, attention_mma.cu) set up barriers, tensor memory and copies, and
// merge the shares of several blocks, 2 us and more of 6 to 9.  Here the chain is table -> keys and
// values (asked for together, straight into registers) -> scores -> values' sums -> one merge in shared
// memory.
//   scores   mma.sync m16n8k16, 16 keys by up to 8 query heads of the group.  Within 32 features a thread of a
//            quad takes [8t, 8t + 8) of its two keys and of its head as the slots of two products: the same
//            permutation of the features on both sides, so every load is 16 bytes.
//   softmax  a warp's own running maximum and sum, in fp32; the exponentials stay in fp32
//   values   on CUDA cores: a lane has 8 features of every KP-th key; the weights of a key come out of shared
//            memory, 16 bytes for four heads
//   merge    the warps' and lanes' shares, with the sink if there is one; then the gate, and one rounding
//
// us a layer with its two products, split kernels -> here, 8 tokens behind 250 keys, 16 heads: of 64 14.0 -> 12.4, of 128 17.3
// -> 14.9; with sink and gate 28.9 -> 20.2, 48 tokens in a window of 1,024 102 -> 60.  A chain of about 4.5 us from the
// wait to the rows for one pass of keys; every 256 keys more are 1.7 us with heads of 64 and 2.9 of 128, 2.6 and 4.8 with more
// than four heads a group, and a block walks them alone (`short_attention_pays` has the lines).
//
// Keys and values of a pass are in registers together, which takes all there are: 250 to 255 of a thread's with heads of 128
// (8 heads a group: 112 bytes spilled), and with heads of 64 and up to four a group the 128 (four: 80 bytes spilled) with
// which sixteen warps, or two blocks of eight, fit an SM.
//
// Reference counterpart: `attention_decode` (engine/kernels/kernels.cu:1740), one block per head over all keys.
#define CB_PDL_BIT 2      // this file's bit in CRUCIBLE_PDL (shared with attention_decode_tcgen05.cu)
#include "common.cuh"
#include <cfloat>

namespace {

struct Args {
    const __nv_bfloat16* q;
    int q_stride;
    __nv_bfloat16* out;
    int out_stride;
    const __nv_bfloat16* gate;        // null, rows laid out like out, or (gate_per_head) one logit a head
    int gate_stride, gate_per_head;
    const __nv_bfloat16 *k_cache, *v_cache;      // [page][kv_head][slot][HD]
    const float* sinks;               // null, or one a query head
    const int *row_start, *first_pos, *table;
    int table_stride, n_rep, n_kv_heads, page_tokens, window;
    float scale_log2, out_scale;      // scale * log2(e)
};

constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float exp2_of(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load16(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }

// HD: features of a head; R: query heads of a group at most (the weights of a key in shared memory are R
// floats); W: warps
template <int HD, int R, int W>
__global__ void __launch_bounds__(32 * W, HD == 64 && R <= 4 && W == 8 ? 2 : 1) attention_short_kernel(const Args a) {
    constexpr int PIECES = HD / 8, KP = 32 / PIECES, U = 32 / KP, I = HD / 32, RP = R < 4 ? 4 : R;
    __shared__ __align__(16) float weights[W][32][RP];
    __shared__ float top[W][8], sum[W][8], rescale[W][8];
    extern __shared__ __align__(16) float parts[];        // [W][KP][R][HD]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int kvh = blockIdx.x, r = blockIdx.y;
    // (the step's metadata is no kernel's output)
    const int row = a.row_start[r], pos = a.first_pos[r];
    const int first = a.window > 0 ? max(0, pos - a.window + 1) : 0, n_keys = pos - first + 1;
    const int* table = a.table + (size_t)r * a.table_stride;
    // a lane's key of a pass: where its row begins in the pages, in rows of HD
    auto place_of = [&](int key) {
        const int at = first + key;
        return key < n_keys ? (long)(table[at / a.page_tokens] * a.n_kv_heads + kvh) * a.page_tokens + at % a.page_tokens : 0l;
    };
    long place = place_of(warp * 32 + lane);
    cb_pdl_wait();
    const __nv_bfloat16* q_row = a.q + (size_t)row * a.q_stride + ((size_t)kvh * a.n_rep + g) * HD + t * 8;
    uint4 q[I];
#pragma unroll
    for (int i = 0; i < I; ++i) q[i] = g < a.n_rep ? load16(q_row + 32 * i) : make_uint4(0, 0, 0, 0);
    // The maximum begins at the lowest finite number, not at -inf: then a score of -inf weighs 0 and a NaN stays one (fmaxf
    // passes over it) whatever else there is, without a test, and 0 times it in what follows is one too.
    float m_run[2] = {-FLT_MAX, -FLT_MAX}, l_run[2] = {0.f, 0.f};
    float o[R][8];
#pragma unroll
    for (int h = 0; h < R; ++h)
#pragma unroll
        for (int e = 0; e < 8; ++e) o[h][e] = 0.f;
    const int piece = lane % PIECES, sub = lane / PIECES;
    for (int base = warp * 32; base < n_keys; base += 32 * W) {
        uint4 k[2][2][I], v[U];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int j = 16 * m + 8 * half + g;
                const __nv_bfloat16* from = a.k_cache + __shfl_sync(0xffffffffu, place, j) * HD + t * 8;
#pragma unroll
                for (int i = 0; i < I; ++i) k[m][half][i] = base + j < n_keys ? load16(from + 32 * i) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = u * KP + sub;
            const __nv_bfloat16* from = a.v_cache + __shfl_sync(0xffffffffu, place, j) * HD + piece * 8;
            v[u] = base + j < n_keys ? load16(from) : make_uint4(0, 0, 0, 0);
        }
        if (base + 32 * W < n_keys) place = place_of(base + 32 * W + lane);
        float c[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            c[m][0] = c[m][1] = c[m][2] = c[m][3] = 0.f;
#pragma unroll
            for (int i = 0; i < I; ++i) {
                mma(c[m], k[m][0][i].x, k[m][1][i].x, k[m][0][i].y, k[m][1][i].y, q[i].x, q[i].y);
                mma(c[m], k[m][0][i].z, k[m][1][i].z, k[m][0][i].w, k[m][1][i].w, q[i].z, q[i].w);
            }
        }
        // c[m][2 half + e]: key 16 m + 8 half + g, head 2 t + e
        float m_new[2] = {m_run[0], m_run[1]}, total[2] = {0.f, 0.f};
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                c[m][x] = base + 16 * m + 8 * (x >> 1) + g < n_keys ? c[m][x] * a.scale_log2 : -INFINITY;
                m_new[x & 1] = fmaxf(m_new[x & 1], c[m][x]);
            }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) m_new[e] = fmaxf(m_new[e], __shfl_xor_sync(0xffffffffu, m_new[e], x));
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                // (0 without the test too; with it heads of 128 behind 1,000 keys take 20.3 us, not 20.65)
                const float p = c[m][x] == -INFINITY ? 0.f : exp2_of(c[m][x] - m_new[x & 1]);
                total[x & 1] += p;
                c[m][x] = p;
            }
        __syncwarp();                                     // the pass before is done with the weights
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                if (2 * t < RP)
                    *reinterpret_cast<float2*>(&weights[warp][16 * m + 8 * half + g][2 * t]) = make_float2(c[m][2 * half], c[m][2 * half + 1]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) total[e] += __shfl_xor_sync(0xffffffffu, total[e], x);
            const float keep = exp2_of(m_run[e] - m_new[e]);
            l_run[e] = fmaf(l_run[e], keep, total[e]);
            m_run[e] = m_new[e];
            if (g == 0) rescale[warp][2 * t + e] = keep;
        }
        __syncwarp();
        if (base >= 32 * W) {
#pragma unroll
            for (int h = 0; h < R; ++h) {
                const float keep = rescale[warp][h];
#pragma unroll
                for (int e = 0; e < 8; ++e) o[h][e] *= keep;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float p[RP], x[8];
#pragma unroll
            for (int h = 0; h < RP; h += 4) {
                const float4 w4 = *reinterpret_cast<const float4*>(&weights[warp][u * KP + sub][h]);
                p[h] = w4.x; p[h + 1] = w4.y; p[h + 2] = w4.z; p[h + 3] = w4.w;
            }
            const __nv_bfloat162* pair = reinterpret_cast<const __nv_bfloat162*>(&v[u]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(pair[e]);
                x[2 * e] = f.x;
                x[2 * e + 1] = f.y;
            }
#pragma unroll
            for (int h = 0; h < R; ++h)
#pragma unroll
                for (int e = 0; e < 8; ++e) o[h][e] = fmaf(p[h], x[e], o[h][e]);
        }
    }
    cb_pdl_trigger();
    if (g == 0) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            top[warp][2 * t + e] = m_run[e];
            sum[warp][2 * t + e] = l_run[e];
        }
    }
    if (warp * 32 < n_keys) {                             // (warps without a key have nothing to leave)
#pragma unroll
        for (int h = 0; h < R; ++h) {
            float* to = parts + (((size_t)warp * KP + sub) * R + h) * HD + piece * 8;
            *reinterpret_cast<float4*>(to) = make_float4(o[h][0], o[h][1], o[h][2], o[h][3]);
            *reinterpret_cast<float4*>(to + 4) = make_float4(o[h][4], o[h][5], o[h][6], o[h][7]);
        }
    }
    __syncthreads();
    const int warps = min(W, (n_keys + 31) / 32);
    for (int i = threadIdx.x; i < a.n_rep * HD; i += 32 * W) {
        const int h = i / HD, d = i - h * HD, head = kvh * a.n_rep + h;
        const float sink = a.sinks != nullptr ? a.sinks[head] * LOG2E : -INFINITY;
        float m = sink;
#pragma unroll
        for (int w = 0; w < W; ++w) m = fmaxf(m, w < warps ? top[w][h] : -INFINITY);
        float l = sink == -INFINITY ? 0.f : exp2_of(sink - m), y = 0.f;
        for (int w = 0; w < warps; ++w) {
            const float f = exp2_of(top[w][h] - m);
            float x = 0.f;
#pragma unroll
            for (int s = 0; s < KP; ++s) x += parts[(((size_t)w * KP + s) * R + h) * HD + d];
            l = fmaf(f, sum[w][h], l);
            y = fmaf(f, x, y);
        }
        y = l > 0.f ? y / l * a.out_scale : y * 0.f;         // (no weight at all, or a NaN)
        if (a.gate != nullptr) {
            const float z = __bfloat162float(a.gate[(size_t)row * a.gate_stride + (a.gate_per_head ? head : head * HD + d)]);
            y *= 1.0f / (1.0f + expf(-z));
        }
        a.out[(size_t)row * a.out_stride + (size_t)head * HD + d] = __float2bfloat16_rn(y);
    }
}

template <int HD, int R, int W>
int launch(const Args& a, int n_requests, cudaStream_t s) {
    constexpr int KP = 32 / (HD / 8), bytes = W * KP * R * HD * 4;
    auto kernel = attention_short_kernel<HD, R, W>;
    if (bytes > 32 * 1024) {
        static thread_local int ready = -1;            // the device whose limit was raised last
        int dev = 0;
        cudaGetDevice(&dev);
        if (ready != dev) {
            const cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (rc != cudaSuccess) return (int)rc;
            ready = dev;
        }
    }
    cb_launch(kernel, dim3(a.n_kv_heads, n_requests), dim3(32 * W), bytes, s, a);
    return cb_last_error();
}

}  // namespace

// Requests that bring one token each: row row_start[r] at position first_pos[r], over its keys from the page table (the token's
// own among them).  q, out, gate: bfloat16 rows; window 0: all keys.  head_dim 64 or 128, at most 8 query heads a
// key/value head, rows on 16 bytes.
CB_EXPORT int cb_attention_short(const void* q, int q_stride, void* out, int out_stride, const void* gate, int gate_stride,
                                 int gate_per_head, const void* k_cache, const void* v_cache, const float* sinks,
                                 const int* row_start, const int* first_pos, const int* table, int table_stride,
                                 int n_requests, int n_heads, int n_kv_heads, int head_dim, int page_tokens, float scale,
                                 int window, float out_scale, void* stream) {
    if (n_requests <= 0) return 0;
    if ((head_dim != 64 && head_dim != 128) || n_kv_heads <= 0 || n_heads % n_kv_heads || n_heads / n_kv_heads > 8 ||
        n_requests > 65535 || page_tokens <= 0 || window < 0 || (q_stride & 7) || ((uintptr_t)q & 15) ||
        ((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15))
        return CB_ERR_UNSUPPORTED;
    Args a;
    a.q = (const __nv_bfloat16*)q; a.q_stride = q_stride; a.out = (__nv_bfloat16*)out; a.out_stride = out_stride;
    a.gate = (const __nv_bfloat16*)gate; a.gate_stride = gate_stride; a.gate_per_head = gate_per_head;
    a.k_cache = (const __nv_bfloat16*)k_cache; a.v_cache = (const __nv_bfloat16*)v_cache; a.sinks = sinks;
    a.row_start = row_start; a.first_pos = first_pos; a.table = table; a.table_stride = table_stride;
    a.n_rep = n_heads / n_kv_heads; a.n_kv_heads = n_kv_heads; a.page_tokens = page_tokens; a.window = window;
    a.scale_log2 = scale * LOG2E; a.out_scale = out_scale;
    cudaStream_t s = (cudaStream_t)stream;
    if (head_dim == 64) {
        // (sixteen warps take an SM's registers: a block to an SM)
        const bool many = (long)n_requests * n_kv_heads > 148;
        if (a.n_rep <= 2) return many ? launch<64, 2, 8>(a, n_requests, s) : launch<64, 2, 16>(a, n_requests, s);
        if (a.n_rep <= 4) return many ? launch<64, 4, 8>(a, n_requests, s) : launch<64, 4, 16>(a, n_requests, s);
        return launch<64, 8, 8>(a, n_requests, s);
    }
    if (a.n_rep <= 2) return launch<128, 2, 8>(a, n_requests, s);
    return a.n_rep <= 4 ? launch<128, 4, 8>(a, n_requests, s) : launch<128, 8, 8>(a, n_requests, s);
}
