// C[M,N] = A[M,K] . W[N,K]^T in bfloat16 on the 5th-generation tensor cores, for products of more tiles than
// SMs: one block an SM walks its tiles, and a tile's way out runs beside the next tile's products.
//
// A block of `gemm_tcgen05.cu` does one tile: 3 to 4 us of a wave go into its start, the first loads and its
// epilogue, while a 128 x 256 tile's products over K = 2,048 take 9.6 (278 ns a block of 64 of K alone on the
// chip, 300 with all SMs: the tensor cores' rate, so nothing is to be had there).  Here the ring of stages
// runs on from tile to tile, tensor memory holds two accumulators, and eight warps in two groups, one for
// each half of a tile's columns, take the finished one out through buffers of their own.
//
// Roles: warp 0 loads (TMA, 128-byte swizzle), warp 1 owns tensor memory and issues the MMAs, warps 2-9
// are the epilogue: a group takes 64 bytes of its columns of all 128 rows at a time from tensor memory into
// one of its two buffers (64-byte swizzle) and sends it by TMA: a store, or an fp32 add at the memory side.
//
// Epilogues and forms as in `gemm_tcgen05.cu`: STORE_BF16 (with an activation), STORE_F32, SWIGLU_BF16; rows ahead of their
// norm (NormArgs::sumsq_in) with SWIGLU_BF16; a grouped product (NormArgs::plan), of 256 columns a tile.  The rules
// (`_waves_width`, `grouped_waves`) choose 192 or 256 columns; 128, and ACCUM_F32 (a TMA add instead of the store), no rule
// chooses yet: the tests of the tile walk run them, for its edges at three widths.  In a grouped product a tile that ends
// before its 128 rows leaves its buffers row by row, 64 bytes a row, since the rows behind it are another expert's.
//
// us at 2,048 rows, a block a tile (or tall) -> here: gated pair of 2 x 2,816 by K = 2,048 43.2 -> 35.3 (1,338 TFLOP/s),
// of 2 x 2,048 by 768 15.8 -> 13.3; fp32 results of 4,096 by 128 10.2 -> 8.6; 4,096 rows of 8 experts, gate/up of
// 2,816 by 2,048 99.8 -> 90.6, down 53.8 -> 49.2.  Where a wave or less is all there is, a block a tile is ahead
// (5 to 30 %: its successor starts under its end), and so are tall tiles for bf16 results (`_waves_width` has
// the line).  Pairs of blocks (cta_group::2, half of W's bytes) were within 5 % either way: the operands' way
// is not what bounds this.
//
// Sizes: K, lda, ldw multiples of 8, bases on 16 bytes, rows of C of whole 16-byte pieces; tails in M, N and K are
// zero-filled by TMA and masked at the store.  Anything else is refused.
#define CB_PDL_BIT 0      // this file's bit in CRUCIBLE_PDL (shared with gemm_tcgen05.cu)
#include "common.cuh"
#include "tc_common.cuh"
#include "gemm_args.cuh"

namespace {

constexpr int BM = 128;
constexpr int BK = 64;                 // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int THREADS = 320;
constexpr int BUF = BM * 64;           // bytes of a staging buffer: 64 of every row

enum Form { PLAIN = 0, NORM_PRE = 1, GROUPED = 2 };

template <int BN, int STAGES>
struct SharedStorage {
    alignas(1024) uint8_t a[STAGES][BM * BK * 2];
    alignas(1024) uint8_t b[STAGES][BN * BK * 2];
    alignas(1024) uint8_t out[2][2][BUF];       // [group][buffer]
    alignas(8) uint64_t full_bar[STAGES];
    uint64_t empty_bar[STAGES];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

// where a tile lies: rows [m0, m_end), W's first row, and the tile's number along N
struct Tile { int m0, m_end, w_row0, n_tile; };

template <int BN, int STAGES, int EPI, int FORM>
__global__ void __launch_bounds__(THREADS, 1)
gemm_waves_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                  const __grid_constant__ CUtensorMap map_c, void* c_ptr, int M, int N, int K, int ldc, int inter,
                  int m_tiles, int n_tiles, int* __restrict__ status, const NormArgs na) {
    extern __shared__ uint8_t smem_raw[];
    using Storage = SharedStorage<BN, STAGES>;
    Storage& s = *reinterpret_cast<Storage*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_blocks = (K + BK - 1) / BK;
    volatile int* abort_flag = &s.abort_flag;
    constexpr uint32_t TMEM_COLS = BN <= 64 ? 128 : BN <= 128 ? 256 : 512;       // two accumulators
    constexpr uint32_t ACC = TMEM_COLS / 2;
    constexpr uint32_t STAGE_BYTES = (BM + BN) * BK * 2;
    constexpr bool F32 = EPI == STORE_F32 || EPI == ACCUM_F32, PRE = FORM == NORM_PRE;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            tc::mbar_init(&s.full_bar[i], 1);
            tc::mbar_init(&s.empty_bar[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&s.acc_full[i], 1);
            tc::mbar_init(&s.acc_empty[i], 8);
        }
        s.abort_flag = 0;
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_a);
        tc::prefetch_tensormap(&map_w);
        tc::prefetch_tensormap(&map_c);
    }
    if (warp == 1) {
        tc::tmem_alloc(&s.tmem_base, TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem = s.tmem_base;

    // (a plan was written by a kernel before this one: read behind the wait below.)  Neighbouring blocks share a
    // tile of W; in a grouped product they share a tile of rows, since an expert has few of those.
    int tiles = m_tiles * n_tiles;
    auto tile_at = [&](int t) {
        Tile x;
        if (FORM == GROUPED) {
            const int y = t / n_tiles;
            const int* entry = na.plan + 2 + na.n_experts + y;
            x.n_tile = t - y * n_tiles;
            x.m0 = __ldg(entry + na.max_tiles);
            x.m_end = x.m0 + __ldg(entry + 2 * na.max_tiles);
            x.w_row0 = __ldg(entry) * na.w_rows;
        } else {
            x.n_tile = t / m_tiles;
            x.m0 = (t - x.n_tile * m_tiles) * BM;
            x.m_end = M;
            x.w_row0 = 0;
        }
        return x;
    };
    auto load_w = [&](const Tile& x, int kb, int st) {
        if (EPI == SWIGLU_BF16) {
            constexpr int half = BN / 2;
            tc::tma_load_2d(s.b[st], &map_w, &s.full_bar[st], kb * BK, x.w_row0 + x.n_tile * half);
            tc::tma_load_2d(s.b[st] + half * BK * 2, &map_w, &s.full_bar[st], kb * BK, x.w_row0 + inter + x.n_tile * half);
        } else {
            tc::tma_load_2d(s.b[st], &map_w, &s.full_bar[st], kb * BK, x.w_row0 + x.n_tile * BN);
        }
    };
    // the first stages' W go out before the kernels ahead of this one are done: no kernel writes a weight
    const int w_ahead = FORM == GROUPED ? 0 : min(k_blocks, STAGES);
    if (warp == 0 && w_ahead > 0 && tc::elect_one()) {
        const Tile x = tile_at(blockIdx.x);
        for (int kb = 0; kb < w_ahead; ++kb) {
            tc::mbar_expect_tx(&s.full_bar[kb], STAGE_BYTES);
            load_w(x, kb, kb);
        }
    }
    cb_pdl_wait();
    cb_pdl_trigger();
    if (FORM == GROUPED) tiles = min(__ldg(na.plan), na.max_tiles) * n_tiles;

    if (warp == 0) {
        if (tc::elect_one()) {
            int st = 0, ahead = w_ahead, sent = 0;
            uint32_t parity = 1;                         // of a stage's last round, once there was one
            bool ok = true, first_round = true;
            Tile next = tile_at(min((int)blockIdx.x, max(tiles - 1, 0)));
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                const Tile x = next;
                if (t + (int)gridDim.x < tiles) next = tile_at(t + gridDim.x);      // (the plan's answer is on its way meanwhile)
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!first_round && !tc::mbar_wait(&s.empty_bar[st], parity, abort_flag)) {
                        tc::give_up(abort_flag, status, tc::ST_PRODUCER_TIMEOUT);
                        ok = false;
                        break;
                    }
                    if (ahead > 0) {
                        --ahead;
                    } else {
                        tc::mbar_expect_tx(&s.full_bar[st], STAGE_BYTES);
                        load_w(x, kb, st);
                    }
                    tc::tma_load_2d(s.a[st], &map_a, &s.full_bar[st], kb * BK, x.m0);
                    ++sent;
                    if (++st == STAGES) st = 0, parity ^= 1, first_round = false;
                }
            }
            if (*abort_flag) {
                // let our own copies land before the block's shared memory goes away
                for (int i = max(0, sent - STAGES); i < max(sent, w_ahead); ++i)
                    for (uint32_t n = 0; n < tc::WAIT_LIMIT; ++n)
                        if (tc::mbar_try_wait(&s.full_bar[i % STAGES], (i / STAGES) & 1)) break;
            }
        }
    } else if (warp == 1) {
        if (tc::elect_one()) {
            constexpr uint32_t idesc = tc::instr_desc_bf16(BM, BN);
            constexpr uint32_t A_STEP = sizeof(s.a[0]) >> 4, B_STEP = sizeof(s.b[0]) >> 4;
            const uint64_t desc0 = tc::smem_desc_sw128(tc::smem_u32(s.a[0]));
            const uint32_t desc_hi = (uint32_t)(desc0 >> 32), a_lo = (uint32_t)desc0;
            const uint32_t b_lo = (uint32_t)tc::smem_desc_sw128(tc::smem_u32(s.b[0]));
            const uint32_t full0 = tc::smem_u32(&s.full_bar[0]), empty0 = tc::smem_u32(&s.empty_bar[0]);
            int st = 0, n = 0;                           // n: tiles of this block so far
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++n) {
                const uint32_t acc = tmem + (n & 1) * ACC;
                // the accumulator's last tile (two tiles ago) has left it
                if (n >= 2 && !tc::mbar_wait(&s.acc_empty[n & 1], (uint32_t)((n >> 1) - 1) & 1u, abort_flag)) {
                    tc::give_up(abort_flag, status, tc::ST_MMA_TIMEOUT);
                    break;
                }
                tc::tc_fence_after_sync();
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!tc::mbar_wait_at(full0 + 8 * st, phase, abort_flag)) {
                        tc::give_up(abort_flag, status, tc::ST_MMA_TIMEOUT);
                        ok = false;
                        break;
                    }
                    tc::tc_fence_after_sync();
                    const uint32_t a_st = a_lo + st * A_STEP, b_st = b_lo + st * B_STEP;
                    tc::umma_bf16(acc, tc::desc_of(a_st, desc_hi), tc::desc_of(b_st, desc_hi), idesc, kb > 0 ? 1u : 0u);
#pragma unroll
                    for (int k = 1; k < BK / UMMA_K; ++k)
                        tc::umma_bf16_add(acc, tc::desc_of(a_st + 2 * k, desc_hi), tc::desc_of(b_st + 2 * k, desc_hi), idesc);
                    tc::umma_commit_at(empty0 + 8 * st);
                    if (++st == STAGES) st = 0, phase ^= 1;
                }
                if (ok) tc::umma_commit(&s.acc_full[n & 1]);
            }
        }
    } else {
        // ---- epilogue: a group of four warps a half of the tile's columns; lane quarter = warp % 4 ----
        const int group = (warp - 2) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        constexpr int OUT_COLS = EPI == SWIGLU_BF16 ? BN / 2 : BN;     // columns of C per tile
        constexpr int CHUNK = F32 ? 16 : 32;                            // columns of a buffer
        constexpr int CHUNKS = OUT_COLS / 2 / CHUNK;                    // of a group
        static_assert(OUT_COLS % (2 * CHUNK) == 0, "whole buffers in either half");
        const int n_out = EPI == SWIGLU_BF16 ? inter : N;
        const bool sender = lane == 0 && (warp == 2 || warp == 6);
        const int bar = 1 + group;
        int n = 0, used = 0;                             // buffers filled so far
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++n) {
            const Tile x = tile_at(t);
            const int row = x.m0 + r;
            float f = 1.f;
            if (PRE && row < M) {
                float ss = 0.f;
#pragma unroll 4
                for (int i = 0; i < na.parts; ++i) ss += __ldcg(na.sumsq_in + (size_t)i * M + row);
                f = 1.0f / sqrtf(ss / na.width + na.eps);
            }
            int ok = tc::mbar_wait(&s.acc_full[n & 1], (uint32_t)(n >> 1) & 1u, abort_flag);
            if (!ok && !*abort_flag) tc::give_up(abort_flag, status, tc::ST_EPILOGUE_TIMEOUT);
            // the whole group goes on, or none of it
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, %1, 128, p;\n\t"
                         "selp.s32 %0, 1, 0, q;\n\t}" : "+r"(ok) : "r"(bar) : "memory");
            if (!ok) break;
            tc::tc_fence_after_sync();
            const uint32_t lane_addr = tmem + (n & 1) * ACC + ((uint32_t)(quarter * 32) << 16);
            const bool whole = FORM != GROUPED || x.m0 + BM <= x.m_end;
#pragma unroll 1
            for (int c = 0; c < CHUNKS; ++c, ++used) {
                const int col = group * (OUT_COLS / 2) + c * CHUNK;
                uint8_t* buf = s.out[group][used & 1];
                uint8_t* mine = buf + r * 64;
                uint4 pieces[4];
                if (F32) {
                    uint32_t v[16];
                    tc::tmem_ld_32x16(lane_addr + col, v);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 4; ++q) pieces[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                } else {
                    uint32_t v[32];
                    tc::tmem_ld_32x32(lane_addr + col, v);
                    if (EPI == SWIGLU_BF16) {
                        uint32_t u[32];
                        tc::tmem_ld_32x32(lane_addr + BN / 2 + col, u);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            v[j] = __float_as_uint(tc::gated_pair(__uint_as_float(v[j]) * f, __uint_as_float(u[j]) * f,
                                                                  na.glu_limit, na.glu_alpha, na.glu_offset));
                    } else {
                        tc::tmem_ld_wait();
                        if (na.act == 1) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                const float z = fmaxf(__uint_as_float(v[j]), 0.f);
                                v[j] = __float_as_uint(z * z);
                            }
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t pk[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(v[q * 8 + 2 * j]),
                                                                      __uint_as_float(v[q * 8 + 2 * j + 1]));
                            pk[j] = *reinterpret_cast<uint32_t*>(&b2);
                        }
                        pieces[q] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    }
                }
                if (c + 1 == CHUNKS) {                   // the accumulator may take the next tile but one
                    tc::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&s.acc_empty[n & 1]);
                }
                // the buffer's last store has read it (the other one's may still run)
                if (sender) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
#pragma unroll
                for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(mine + ((q ^ ((r >> 1) & 3)) << 4)) = pieces[q];
                tc::fence_proxy_async();
                asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
                const int at = x.n_tile * OUT_COLS + col;
                if (whole) {
                    if (sender) {
                        if (at < n_out) {
                            if (EPI == ACCUM_F32) tc::tma_reduce_add_2d(&map_c, buf, at, x.m0);
                            else tc::tma_store_2d(&map_c, buf, at, x.m0);
                        }
                        tc::tma_store_commit();
                    }
                } else {
                    // four lanes a row; the buffer is written again behind two barriers at least
                    constexpr int ESIZE = F32 ? 4 : 2;
                    const int piece = threadIdx.x & 3;
                    for (int i = ((threadIdx.x - 64) & 127) >> 2; i < x.m_end - x.m0; i += 32) {
                        const uint4 v = *reinterpret_cast<const uint4*>(buf + i * 64 + ((piece ^ ((i >> 1) & 3)) << 4));
                        const int first = at + piece * (16 / ESIZE);
                        if (first < n_out)       // (rows of C are whole 16-byte pieces: n_out is a multiple of one)
                            *reinterpret_cast<uint4*>(static_cast<uint8_t*>(c_ptr) +
                                                      ((size_t)(x.m0 + i) * ldc + first) * ESIZE) = v;
                    }
                    if (sender) tc::tma_store_commit();          // an empty group, so that the count above holds
                }
            }
        }
        if (sender) tc::tma_store_wait_all();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc(tmem, TMEM_COLS);
    }
}

// An output matrix [rows, cols] (bf16 or fp32) written in boxes of [128 rows, 64 bytes] with the 64-byte swizzle.
bool out_map(CUtensorMap* out, const void* base, bool f32, uint64_t rows, uint64_t cols, uint64_t ld) {
    tc::EncodeTiledFn fn = tc::encode_fn();
    if (!fn) return false;
    const uint64_t esize = f32 ? 4 : 2;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * esize};
    cuuint32_t box[2] = {(cuuint32_t)(64 / esize), BM};
    cuuint32_t estr[2] = {1, 1};
    return fn(out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int STAGES, int EPI, int FORM>
int launch_form(const CUtensorMap& ma, const CUtensorMap& mw, void* C, int M, int N, int K, int ldc, int* status,
                cudaStream_t stream, const NormArgs& na) {
    constexpr bool F32 = EPI == STORE_F32 || EPI == ACCUM_F32;
    const int inter = EPI == SWIGLU_BF16 ? N : 0;
    const int m_tiles = FORM == GROUPED ? na.max_tiles : (M + BM - 1) / BM;
    const int n_tiles = ((EPI == SWIGLU_BF16 ? 2 * N : N) + BN - 1) / BN;
    const size_t esize = F32 ? 4 : 2;
    if (((uintptr_t)C & 15) || (size_t)ldc * esize % 16 || (size_t)N * esize % 16) return CB_ERR_UNSUPPORTED;
    CUtensorMap mc;
    if (!out_map(&mc, C, F32, (uint64_t)M, (uint64_t)N, (uint64_t)ldc)) return CB_ERR_UNSUPPORTED;
    constexpr int smem = (int)sizeof(SharedStorage<BN, STAGES>) + 1024;
    static_assert(smem <= 227 * 1024, "a block's shared memory");
    auto kernel = gemm_waves_kernel<BN, STAGES, EPI, FORM>;
    static thread_local int ready = -1;            // the device whose limit was raised last
    int dev = 0;
    cudaGetDevice(&dev);
    if (ready != dev) {
        const cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (rc != cudaSuccess) return (int)rc;
        ready = dev;
    }
    const long tiles = (long)m_tiles * n_tiles;
    if (tiles > 0x3fffffff) return CB_ERR_UNSUPPORTED;
    cb_launch(kernel, dim3((unsigned)(tiles < 148 ? tiles : 148)), dim3(THREADS), smem, stream, ma, mw, mc, C, M, N, K, ldc,
              inter, m_tiles, n_tiles, status, na);
    return cb_last_error();
}

template <int BN, int STAGES>
int launch(int epi, const CUtensorMap& ma, const CUtensorMap& mw, void* C, int M, int N, int K, int ldc, int* status,
           cudaStream_t s, const NormArgs& na) {
    if (na.plan != nullptr) {
        if constexpr (BN == 256) {
            switch (epi) {
                case STORE_BF16: return launch_form<BN, STAGES, STORE_BF16, GROUPED>(ma, mw, C, M, N, K, ldc, status, s, na);
                case STORE_F32: return launch_form<BN, STAGES, STORE_F32, GROUPED>(ma, mw, C, M, N, K, ldc, status, s, na);
                case SWIGLU_BF16: return launch_form<BN, STAGES, SWIGLU_BF16, GROUPED>(ma, mw, C, M, N, K, ldc, status, s, na);
            }
        }
        return CB_ERR_UNSUPPORTED;
    }
    if (na.sumsq_in != nullptr) {
        if constexpr (BN % 128 == 0)
            if (epi == SWIGLU_BF16) return launch_form<BN, STAGES, SWIGLU_BF16, NORM_PRE>(ma, mw, C, M, N, K, ldc, status, s, na);
        return CB_ERR_UNSUPPORTED;
    }
    switch (epi) {
        case STORE_BF16: return launch_form<BN, STAGES, STORE_BF16, PLAIN>(ma, mw, C, M, N, K, ldc, status, s, na);
        case STORE_F32: return launch_form<BN, STAGES, STORE_F32, PLAIN>(ma, mw, C, M, N, K, ldc, status, s, na);
        case ACCUM_F32: return launch_form<BN, STAGES, ACCUM_F32, PLAIN>(ma, mw, C, M, N, K, ldc, status, s, na);
        case SWIGLU_BF16:
            if constexpr (BN % 128 == 0) return launch_form<BN, STAGES, SWIGLU_BF16, PLAIN>(ma, mw, C, M, N, K, ldc, status, s, na);
    }
    return CB_ERR_UNSUPPORTED;
}

}  // namespace

// As `cb_gemm_tcgen05` and, with a plan in `norm`, `cb_gemm_tcgen05_grouped` (whose plan's tiles have 128 rows).
// bn: tile width: 128, 192 (not SWIGLU_BF16) or 256; 256 alone with a plan.
CB_EXPORT int cb_gemm_waves(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int epi,
                            int bn, int* status, void* stream, const void* norm) {
    if (M <= 0 || N <= 0) return 0;
    const NormArgs na = norm ? *static_cast<const NormArgs*>(norm) : NormArgs{};
    if (K <= 0 || (K & 7) || (lda & 7) || (ldw & 7) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) || na.gain != nullptr ||
        na.heads > 0 || na.n_main > 0 || (na.sumsq_in != nullptr && (na.parts < 1 || !(na.width > 0.f))) ||
        (na.plan != nullptr && (na.n_experts <= 0 || na.max_tiles <= 0 || na.w_rows <= 0)))
        return CB_ERR_UNSUPPORTED;
    const uint64_t w_rows = na.plan != nullptr ? (uint64_t)na.n_experts * na.w_rows : epi == SWIGLU_BF16 ? 2 * (uint64_t)N : N;
    CUtensorMap ma, mw;
    if (!tc::make_map_2d(&ma, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, BM) ||
        !tc::make_map_2d(&mw, W, w_rows, (uint64_t)K, (uint64_t)ldw, epi == SWIGLU_BF16 ? bn / 2 : bn))
        return CB_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    switch (bn) {
        case 128: return launch<128, 6>(epi, ma, mw, C, M, N, K, ldc, status, s, na);
        case 192: return launch<192, 4>(epi, ma, mw, C, M, N, K, ldc, status, s, na);
        case 256: return launch<256, 4>(epi, ma, mw, C, M, N, K, ldc, status, s, na);
    }
    return CB_ERR_UNSUPPORTED;
}
