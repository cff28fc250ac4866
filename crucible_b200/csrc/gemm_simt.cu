// C[M,N] (+)= A[M,K] . W[N,K]^T on CUDA cores with fp32 multiply-add: the
// matrix product of the true 32-bit path, and the refuge of the bfloat16 path
// for shapes its tensor-core kernel refuses.  No tensor cores, no reduced-
// precision mode.  Every output element is one sum over k in ascending order,
// whatever M and N are and wherever its tile lies, so a row's result does not
// depend on what else is in the batch.
//
// Tiles of 64 x 64 with 8 x 4 sums a thread, or 16 x 32 with 4 x 1 for up to 16 rows (more blocks); the
// next 16 of k are on their way from memory while these are multiplied.  The sums of two neighbouring
// columns are one instruction; 12 operands come out of shared memory for 32 multiply-adds, and that
// path is the bound.  Rows of whole 16-byte pieces are read 16 bytes a thread, others element by
// element.  700 x 768 by 1,280 x 768 in fp32: 55 us (25 TFLOP/s), 120 with 4 x 4 sums a
// thread and no load ahead.
//
// Reference counterpart: `gemm_f32` (engine/kernels/kernels.cu:922), 16x16 scalar tiles.
#define CB_PDL_BIT 9      // this file's bit in CRUCIBLE_PDL
#include "common.cuh"

namespace {

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
gemm_simt_kernel(const TA* __restrict__ A, const TA* __restrict__ W, TC* __restrict__ C,
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
int launch_as(const TA* A, const TA* W, TC* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
    if (M <= 16)
        cb_launch(gemm_simt_kernel<TA, TC, ACCUMULATE, VEC, 16, 32, 4, 1>, dim3((N + 31) / 32, (M + 15) / 16),
                  dim3(THREADS), 0, s, A, W, C, M, N, K, lda, ldw, ldc);
    else
        cb_launch(gemm_simt_kernel<TA, TC, ACCUMULATE, VEC, 64, 64, 8, 4>, dim3((N + 63) / 64, (M + 63) / 64),
                  dim3(THREADS), 0, s, A, W, C, M, N, K, lda, ldw, ldc);
    return cb_last_error();
}

template <typename TA, typename TC>
int launch(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw,
           int ldc, int accumulate, cudaStream_t s) {
    // rows of whole groups of four elements, every group on a boundary of its size
    const size_t group = 4 * sizeof(TA);
    const bool vec = ((K | lda | ldw) & 3) == 0 && (uintptr_t)A % group == 0 && (uintptr_t)W % group == 0;
#define CB_SIMT(ACC, VV) return launch_as<TA, TC, ACC, VV>((const TA*)A, (const TA*)W, (TC*)C, M, N, K, lda, ldw, ldc, s)
    if (accumulate) {
        if (vec) CB_SIMT(true, true);
        CB_SIMT(true, false);
    }
    if (vec) CB_SIMT(false, true);
    CB_SIMT(false, false);
#undef CB_SIMT
}

}  // namespace

// in_dtype: dtype of A and W; out_dtype: dtype of C.  accumulate: C += A.W^T.
CB_EXPORT int cb_gemm_simt(const void* A, const void* W, void* C, int in_dtype, int out_dtype,
                           int M, int N, int K, int lda, int ldw, int ldc, int accumulate,
                           void* stream) {
    if (M <= 0 || N <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    if (in_dtype == CB_F32 && out_dtype == CB_F32)
        return launch<float, float>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, s);
    if (in_dtype == CB_BF16 && out_dtype == CB_BF16)
        return launch<__nv_bfloat16, __nv_bfloat16>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, s);
    if (in_dtype == CB_BF16 && out_dtype == CB_F32)
        return launch<__nv_bfloat16, float>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, s);
    return CB_ERR_UNSUPPORTED;
}
