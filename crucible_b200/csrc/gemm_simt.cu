// C[M,N] (+)= A[M,K] . W[N,K]^T on CUDA cores with fp32 multiply-add: the
// matrix product of the true 32-bit path, and the refuge of the bfloat16 path
// for shapes its tensor-core kernel refuses.  No tensor cores, no reduced-
// precision mode.  Every output element is one sum over k in ascending order,
// whatever M and N are and wherever its tile lies, so a row's result does not
// depend on what else is in the batch.
//
// gemm_f32_kernel, fp32 rows of whole 16-byte pieces: a block owns TM x TN of C and walks K in stages of
// TK that asynchronous copies bring ahead; both operands lie row by row in shared memory (pitch TK + 4
// floats: 8 neighbouring rows' 16-byte reads hit all banks), and a thread takes four of k of each of its
// RM + RN rows at a time, the next four on their way.  Two things bound it: the bytes that come out of
// shared memory (RM + RN operands for RM x RN multiply-adds; a read costs by the bytes that reach
// registers, broadcast or not), and, where there are few outputs, every output's chain of additions.
// Hence four forms, from 2 x 2 sums a thread, so that few rows still spread over the SMs, to 8 x 4
// (`pick_form` has the rule and the measured costs).
// us before (gemm_rows_kernel for all) -> now, W in L2, K = N = 1,024: 5 rows 21.0 -> 12.0, 28 rows 46.6 ->
// 12.6, 116 rows 48.3 -> 17.2, 301 rows 48.7 -> 32.4, 700 rows 63.3 -> 49.7; 700 x 768 x 768 37.5 -> 27.3
// (0.41 of the SMs' multiply-adds; the copies out of shared memory alone would be 20); 2,048 x 2,304 x 768
// 172 -> 165.  Stages are whole, so a K just past one costs up to a stage more, where gemm_rows_kernel is taken instead.  (A
// tail of half a stage in a second copy of the loop's body: 5 to 12 % slower at whole stages.)
//
// gemm_rows_kernel, everything else (bfloat16 rows, rows off 16 bytes) and where `pick_form` says so: tiles of 64 x 64 with 8 x 4 sums a
// thread, or 16 x 32 with 4 x 1 for up to 16 rows; the next 16 of k are on their way through registers,
// which convert them.  (The forms above fed through registers: 15 % slower from 700 rows on.)
//
// Reference counterpart: `gemm_f32` (engine/kernels/kernels.cu:922), 16x16 scalar tiles.
#define CB_PDL_BIT 9      // this file's bit in CRUCIBLE_PDL
#include "common.cuh"

namespace {

// A head a z of the grid: its rows of A and its results lie a_head and c_head elements further, its matrix w_head
struct Product {
    int M, N, K, lda, ldw, ldc;
    long a_head, w_head, c_head;
};

// 16 bytes of a row, zeros (and no access) where `in` is false
__device__ __forceinline__ void copy16(float* smem, const float* gmem, bool in) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(in ? 16 : 0) : "memory");
}

template <bool ACCUMULATE, int TM, int TN, int RM, int RN, int TK, int STAGES>
__global__ void __launch_bounds__(TM * TN / (RM * RN))
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, const Product p) {
    cb_pdl_trigger();
    cb_pdl_wait();
    constexpr int RY = TM / RM, CX = TN / RN, THREADS = RY * CX, P = TK + 4, ROWS = TM + TN;
    constexpr int PASS = THREADS / (TK / 4);
    static_assert(CX % 8 == 0 && RY % 4 == 0 && TM % PASS == 0 && TN % PASS == 0, "whole warps of 8 x 4 threads");
    extern __shared__ __align__(16) float smem[];       // [STAGES][TM rows of A, TN rows of W][P]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % (CX / 8)) * 8 + (lane & 7), ty = (warp / (CX / 8)) * 4 + (lane >> 3);
    const int M = p.M, N = p.N, K = p.K;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    A += (size_t)blockIdx.z * p.a_head;
    W += (size_t)blockIdx.z * p.w_head;
    C += (size_t)blockIdx.z * p.c_head;
    // a thread's share of a stage: the same four of k of every PASS-th row
    const int r0 = tid / (TK / 4), k_own = tid % (TK / 4) * 4;
    const float* a_own = A + (size_t)(m0 + r0) * p.lda + k_own;
    const float* w_own = W + (size_t)(n0 + r0) * p.ldw + k_own;
    auto load = [&](int stage) {
        float* to = smem + (stage % STAGES) * (ROWS * P) + r0 * P + k_own;
        const int at = stage * TK;
#pragma unroll
        for (int e = 0; e < ROWS; e += PASS) {
            const int r = e < TM ? e : e - TM;
            const bool in = (e < TM ? m0 + r0 + r < M : n0 + r0 + r < N) && at + k_own < K;
            const float* src = e < TM ? a_own + (size_t)r * p.lda + at : w_own + (size_t)r * p.ldw + at;
            copy16(to + e * P, in ? src : A, in);
        }
    };
    float acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.f;
    const int stages = (K + TK - 1) / TK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < stages) load(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = 0; s < stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();               // stage s is there, and all are done with the one that the next load replaces
        if (s + STAGES - 1 < stages) load(s + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* a_rows = smem + (s % STAGES) * (ROWS * P) + ty * P;
        const float* w_rows = smem + (s % STAGES) * (ROWS * P) + (TM + tx) * P;
        float a[2][RM][4], w[2][RN][4];                // four of k being multiplied, and the next four
        auto take = [&](int b, int k) {
#pragma unroll
            for (int i = 0; i < RM; ++i) *reinterpret_cast<float4*>(a[b][i]) = *reinterpret_cast<const float4*>(a_rows + i * RY * P + k);
#pragma unroll
            for (int j = 0; j < RN; ++j) *reinterpret_cast<float4*>(w[b][j]) = *reinterpret_cast<const float4*>(w_rows + j * CX * P + k);
        };
        take(0, 0);
#pragma unroll
        for (int k = 0; k < TK; k += 4) {              // (zeros beyond K)
            const int b = k / 4 & 1;
            if (k + 4 < TK) take(b ^ 1, k + 4);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(a[b][i][e], w[b][j][e], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int m = m0 + ty + i * RY;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
            const int n = n0 + tx + j * CX;
            if (n >= N) continue;
            float* to = C + (size_t)m * p.ldc + n;
            *to = ACCUMULATE ? *to + acc[i][j] : acc[i][j];
        }
    }
}

template <bool ACCUMULATE, int TM, int TN, int RM, int RN, int TK, int STAGES>
int launch_form(const float* A, const float* W, float* C, const Product& p, int heads, cudaStream_t s) {
    auto kernel = gemm_f32_kernel<ACCUMULATE, TM, TN, RM, RN, TK, STAGES>;
    constexpr int bytes = STAGES * (TM + TN) * (TK + 4) * 4;
    if (bytes > 48 * 1024) {
        static thread_local int ready = -1;        // the device whose limit was raised last
        int dev = 0;
        cudaGetDevice(&dev);
        if (ready != dev) {
            const cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (rc != cudaSuccess) return (int)rc;
            ready = dev;
        }
    }
    cb_launch(kernel, dim3((p.N + TN - 1) / TN, (p.M + TM - 1) / TM, heads), dim3(TM * TN / (RM * RN)), bytes, s, A, W, C, p);
    return cb_last_error();
}

// The form by what an SM with the most tiles takes for one k, in tenths of a cycle: a part for the chain
// and one a tile, as measured at K = 768 and 1,024 over 8 to 3,255 rows and 16 to 4,608 columns (the choice
// is within 9 % of the best form at all of them).  The smallest form fits an SM six times, the third four.
// -1: gemm_rows_kernel, whose stages are of 16 of k and whose blocks start sooner and fit an SM five times.  All forms
// and it were measured at 15 numbers of rows, 9 of columns and 14 of K from 16 to 2,048; it is ahead
// - at K up to 16 (16 rows of 2,050 2.0 against 2.95 us, 2,050 of 2,050 7.9 against 12.2; few rows of few columns are not);
// - where a K ends in the first half of a stage, so that half a stage is multiplied for nothing, and the tiles are
//   more than the SMs: at 64 x 64 up to K = 512 (700 x 2,050 x 136 15.9 against 17.2, x 264 within 1 %; a tile an SM, 700 x 768 x 136, 9.1
//   against 8.0), at 64 x 32 to 144;
// - at K below 640 where an SM gets 4 and a part of the 64 x 64 tiles: four fit it, so the rest wait (1,300 x 2,050 x 128 22.4
//   against 25.6, x 520 79 against 86, x 768 110 against 106).
// Five to sixteen rows of many columns at a K of one or two stages: the second form before the first (16 x 2,050 x 72 1.14 times
// as fast), and gemm_rows_kernel before both from 288 tiles on (16 x 9,216 x 72 3.7, 4.6 and 4.9 us).  With this choice no size is slower than gemm_rows_kernel's by more than 5 %, but
// 1,000 rows of 16 columns at K = 16 (2.5 against 2.3 us).
constexpr int ROWS_KERNEL = -1;
int pick_form(const Product& p, int heads) {
    auto all = [&](int tm, int tn) { return (long)((p.M + tm - 1) / tm) * ((p.N + tn - 1) / tn) * heads; };
    auto tiles = [&](int tm, int tn) {
        return (p.M + tm - 1) / tm > 65535 ? 1l << 40 : (all(tm, tn) + 147) / 148;     // (a grid has so many rows at the most)
    };
    const long e[4] = {tiles(16, 16), tiles(32, 32), tiles(64, 32), tiles(64, 64)};
    const long cost[4] = {170 * ((e[0] + 5) / 6) + 46 * e[0], 140 + 175 * e[1], 180 * ((e[2] + 3) / 4) + 275 * e[2],
                          170 + 510 * e[3]};
    int form = 0;
    for (int i = 1; i < 4; ++i)
        if (cost[i] < cost[form]) form = i;
    const bool few = p.M <= 16;
    if (p.K <= 16 && (few || all(64, 64) >= 10)) return ROWS_KERNEL;
    if (few && form == 0 && p.M > 4 && p.K <= 80 && all(16, 16) >= (p.K > 64 ? 80 : 149)) return all(16, 16) >= 288 ? ROWS_KERNEL : 1;
    if (few) return form;
    const bool half = p.K % 32 >= 1 && p.K % 32 <= 16;
    if (form == 3 && half && (p.K <= 48 || (e[3] >= 2 && p.K < (e[3] == 2 ? 544 : 512)))) return ROWS_KERNEL;
    if (form == 3 && e[3] == 5 && p.K < 640) return ROWS_KERNEL;
    if (form == 2 && half && e[3] >= 2 && p.K <= 144) return ROWS_KERNEL;
    return form;
}

template <bool ACCUMULATE>
int launch_f32(int form, const float* A, const float* W, float* C, const Product& p, int heads, cudaStream_t s) {
    switch (form) {
        case 0: return launch_form<ACCUMULATE, 16, 16, 2, 2, 64, 4>(A, W, C, p, heads, s);
        case 1: return launch_form<ACCUMULATE, 32, 32, 4, 2, 32, 4>(A, W, C, p, heads, s);
        case 2: return launch_form<ACCUMULATE, 64, 32, 4, 4, 32, 4>(A, W, C, p, heads, s);
        default: return launch_form<ACCUMULATE, 64, 64, 8, 4, 32, 3>(A, W, C, p, heads, s);
    }
}

// ---- rows that are converted or gathered element by element on their way --------------------------

constexpr int TK = 16, THREADS = 128;

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

// four neighbouring elements of a row, zeros beyond its end
template <typename T, bool VEC>
__device__ __forceinline__ float4 four(const T* row, bool in, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!in) return v;
    if (VEC) {
        if (k >= K) return v;
        if (sizeof(T) == 4) return *reinterpret_cast<const float4*>(row + k);
        const uint2 raw = *reinterpret_cast<const uint2*>(row + k);
        const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&raw);
        return make_float4(__bfloat162float(h[0]), __bfloat162float(h[1]), __bfloat162float(h[2]), __bfloat162float(h[3]));
    }
    if (k < K) v.x = cb_to_float(row[k]);
    if (k + 1 < K) v.y = cb_to_float(row[k + 1]);
    if (k + 2 < K) v.z = cb_to_float(row[k + 2]);
    if (k + 3 < K) v.w = cb_to_float(row[k + 3]);
    return v;
}

// TM x TN of C a block, RM x RN sums a thread (RN 4, or 1 for the few-row form)
template <typename TA, typename TC, bool ACCUMULATE, bool VEC, int TM, int TN, int RM, int RN>
__global__ void __launch_bounds__(THREADS)
gemm_rows_kernel(const TA* __restrict__ A, const TA* __restrict__ W, TC* __restrict__ C,
                 int M, int N, int K, int lda, int ldw, int ldc) {
    cb_pdl_trigger();
    cb_pdl_wait();
    static_assert((TM / RM) * (TN / RN) == THREADS, "a thread for every tile of sums");
    constexpr int PM = TM + 4, PN = TN + 4, CX = TN / RN;
    constexpr int LA = (TM * TK / 4 + THREADS - 1) / THREADS, LW = (TN * TK / 4 + THREADS - 1) / THREADS;
    __shared__ __align__(16) float As[2][TK][PM];
    __shared__ __align__(16) float Ws[2][TK][PN];
    const int tid = threadIdx.x;
    const int tx = tid % CX, ty = tid / CX;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    float4 a_next[LA], w_next[LW];
    auto load = [&](int k0) {
#pragma unroll
        for (int e = 0; e < LA; ++e) {
            const int i = tid + e * THREADS, r = i >> 2;
            if (i < TM * 4) a_next[e] = four<TA, VEC>(A + (size_t)(m0 + r) * lda, m0 + r < M, k0 + (i & 3) * 4, K);
        }
#pragma unroll
        for (int e = 0; e < LW; ++e) {
            const int i = tid + e * THREADS, r = i >> 2;
            if (i < TN * 4) w_next[e] = four<TA, VEC>(W + (size_t)(n0 + r) * ldw, n0 + r < N, k0 + (i & 3) * 4, K);
        }
    };
    auto store = [&](int b) {
#pragma unroll
        for (int e = 0; e < LA; ++e) {
            const int i = tid + e * THREADS, r = i >> 2, k = (i & 3) * 4;
            if (i < TM * 4) {
                As[b][k][r] = a_next[e].x; As[b][k + 1][r] = a_next[e].y;
                As[b][k + 2][r] = a_next[e].z; As[b][k + 3][r] = a_next[e].w;
            }
        }
#pragma unroll
        for (int e = 0; e < LW; ++e) {
            const int i = tid + e * THREADS, r = i >> 2, k = (i & 3) * 4;
            if (i < TN * 4) {
                Ws[b][k][r] = w_next[e].x; Ws[b][k + 1][r] = w_next[e].y;
                Ws[b][k + 2][r] = w_next[e].z; Ws[b][k + 3][r] = w_next[e].w;
            }
        }
    };
    float acc[RM][RN];
    pair_t acc2[RM][RN / 2 > 0 ? RN / 2 : 1];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.f;
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) acc2[i][j] = 0;
    }
    load(0);
    store(0);
    __syncthreads();
    int b = 0;
    for (int k0 = 0; k0 < K; k0 += TK, b ^= 1) {
        const bool more = k0 + TK < K;
        if (more) load(k0 + TK);
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            float a[RM];
#pragma unroll
            for (int i = 0; i < RM; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&As[b][kk][ty * RM + i]);
                a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
            }
            if (RN == 4) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][tx * RN]);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const pair_t f = both(a[i]);
                    acc2[i][0] = fma_pair(f, w.x, acc2[i][0]);
                    acc2[i][RN / 2 > 1 ? 1 : 0] = fma_pair(f, w.y, acc2[i][RN / 2 > 1 ? 1 : 0]);
                }
            } else {
                const float w = Ws[b][kk][tx];
#pragma unroll
                for (int i = 0; i < RM; ++i) acc[i][0] = fmaf(a[i], w, acc[i][0]);
            }
        }
        if (more) store(b ^ 1);        // last read before the barrier of the round before
        __syncthreads();
    }
    if (RN == 4)
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN / 2; ++j)
                asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i][2 * j]), "=f"(acc[i][2 * j + 1 < RN ? 2 * j + 1 : 0]) : "l"(acc2[i][j]));
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int m = m0 + ty * RM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
            const int n = n0 + tx * RN + j;
            if (n >= N) continue;
            TC* p = C + (size_t)m * ldc + n;
            if (ACCUMULATE) *p = cb_from_float<TC>(cb_to_float(*p) + acc[i][j]);
            else *p = cb_from_float<TC>(acc[i][j]);
        }
    }
}

template <typename TA, typename TC, bool ACCUMULATE, bool VEC>
int launch_as(const TA* A, const TA* W, TC* C, const Product& p, int heads, cudaStream_t s) {
    if constexpr (VEC && sizeof(TA) == 4 && sizeof(TC) == 4) {
        const int form = pick_form(p, heads);
        if (form != ROWS_KERNEL) return launch_f32<ACCUMULATE>(form, A, W, C, p, heads, s);
    }
    for (int h = 0; h < heads; ++h, A += p.a_head, W += p.w_head, C += p.c_head) {
        if (p.M <= 16)
            cb_launch(gemm_rows_kernel<TA, TC, ACCUMULATE, VEC, 16, 32, 4, 1>, dim3((p.N + 31) / 32, (p.M + 15) / 16),
                      dim3(THREADS), 0, s, A, W, C, p.M, p.N, p.K, p.lda, p.ldw, p.ldc);
        else
            cb_launch(gemm_rows_kernel<TA, TC, ACCUMULATE, VEC, 64, 64, 8, 4>, dim3((p.N + 63) / 64, (p.M + 63) / 64),
                      dim3(THREADS), 0, s, A, W, C, p.M, p.N, p.K, p.lda, p.ldw, p.ldc);
    }
    return cb_last_error();
}

template <typename TA, typename TC>
int launch(const void* A, const void* W, void* C, const Product& p, int heads, int accumulate, cudaStream_t s) {
    // rows of whole groups of four elements, every group on a boundary of its size
    const size_t group = 4 * sizeof(TA);
    const bool vec = ((p.K | p.lda | p.ldw) & 3) == 0 && ((p.a_head | p.w_head) & 3) == 0 && (uintptr_t)A % group == 0
                     && (uintptr_t)W % group == 0;
#define CB_SIMT(ACC, VV) return launch_as<TA, TC, ACC, VV>((const TA*)A, (const TA*)W, (TC*)C, p, heads, s)
    if (accumulate) {
        if (vec) CB_SIMT(true, true);
        CB_SIMT(true, false);
    }
    if (vec) CB_SIMT(false, true);
    CB_SIMT(false, false);
#undef CB_SIMT
}

int dispatch(const void* A, const void* W, void* C, int in_dtype, int out_dtype, const Product& p, int heads, int accumulate, void* stream) {
    if (p.M <= 0 || p.N <= 0 || heads <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    if (in_dtype == CB_F32 && out_dtype == CB_F32) return launch<float, float>(A, W, C, p, heads, accumulate, s);
    if (in_dtype == CB_BF16 && out_dtype == CB_BF16)
        return launch<__nv_bfloat16, __nv_bfloat16>(A, W, C, p, heads, accumulate, s);
    if (in_dtype == CB_BF16 && out_dtype == CB_F32) return launch<__nv_bfloat16, float>(A, W, C, p, heads, accumulate, s);
    return CB_ERR_UNSUPPORTED;
}

}  // namespace

// in_dtype: dtype of A and W; out_dtype: dtype of C.  accumulate: C += A.W^T.
CB_EXPORT int cb_gemm_simt(const void* A, const void* W, void* C, int in_dtype, int out_dtype,
                           int M, int N, int K, int lda, int ldw, int ldc, int accumulate,
                           void* stream) {
    return dispatch(A, W, C, in_dtype, out_dtype, Product{M, N, K, lda, ldw, ldc, 0, 0, 0}, 1, accumulate, stream);
}

// `heads` products (in one launch where the rows are fp32 of whole 16-byte pieces): head h's rows of A and results start a_head and c_head elements further along
// their rows, its matrix w_head elements further.
CB_EXPORT int cb_gemm_simt_heads(const void* A, const void* W, void* C, int in_dtype, int out_dtype,
                                 int M, int N, int K, int lda, int ldw, int ldc, int heads, int a_head, long w_head,
                                 int c_head, void* stream) {
    return dispatch(A, W, C, in_dtype, out_dtype, Product{M, N, K, lda, ldw, ldc, a_head, w_head, c_head}, heads, 0, stream);
}

// The form that an fp32 product of rows of whole 16-byte pieces takes (`pick_form`), for tests.
CB_EXPORT int cb_gemm_simt_form(int M, int N, int K, int heads) {
    return pick_form(Product{M, N, K, K, K, N, 0, 0, 0}, heads);
}
