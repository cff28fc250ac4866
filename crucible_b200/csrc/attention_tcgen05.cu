// Paged causal attention for portions of prompts on the 5th-generation tensor
// cores (head size 64, 128 or, keys and values at once, 256; bfloat16): S = Q K^T and O += P V are tcgen05.mma with
// the scores and the output accumulator in tensor memory; K and V pages come in
// by TMA; the softmax has one thread per query row, which reads S from tensor memory and writes P (bf16)
// back to it for the second MMA.
//
// A block takes up to 128 query rows of one request and one KV head; rows are
// (position, head within the group) pairs, so every query head that shares the
// KV head uses the same K and V tiles; a tile holds whole tokens, so that its rows come in by one TMA box
// per 64 features, as the gate's logits do (fetched by the threads, 16 bytes each, a block of 128 rows of 256
// features waited 11 us for its queries).  It walks the keys in tiles of 128.
// Roles: warp 0 loads (a lane a page: table lookups and, where the tile's pages do not follow one another
// in the pool, one TMA box a page side by side; else one box for the tile), warp 1 owns tensor memory
// and issues the MMAs, the others are the softmax.
// P goes back into tensor memory, over the scores that it was made from, and is the first operand of the
// second product there: shared memory carries queries, keys and values alone (a 128 x 128 x 128 tile: 1,280
// cycles of its 128 bytes a cycle; with P written to and read from it 1,790, more than the products' 1,024).
// Two groups of four softmax warps take the tiles in turn (tile j: group j % 2).  Head size 64: each has its
// own reference maximum, sum and accumulator, merged when the keys are through.  128 and 256: one
// accumulator and a reference that goes from tile to tile, so that three (256: two) buffers of scores find room and
// a group's next scores need not wait for its last second product (16 heads of 128, 2,048 tokens 28.2 -> 26.8 us,
// of 256 31.9 -> 31.0; with 64 features there is room for all of it).
// A tile's code is kept short (64 scores at a time, loops not unrolled): a block lives 10 to 20 us,
// and code that is met for the first time comes from memory (the masks of 128 scores, unrolled: 7,500 cycles).
// What bounds it: a pair of tiles takes the two groups some 3,000 cycles (head size 64), of which the
// special-function unit's 8 a warp and exponential make 2,048; the rest is what a tile takes besides (the
// maxima 400, the way to and from the barriers 400), at which the other group is not always busy with its
// exponentials: set half a tile apart the groups were no faster (17.9 and 17.9), in turns slower (18.5), and a quarter
// of the exponentials on the FMA pipe gave 2 %, 7 % less where most blocks are short.
// Measured on one B200, a captured chain of this launch by itself, a 2,048-token prompt: 12 heads of 64 on 4 17.7 us a
// layer (27 with P in shared memory and the rows fetched by hand), 16 heads of 128 on 4, a window of 1,024 and a
// gate 26.5 (58), 16 heads of 256 on 1 30.8 (76), of which 192 features are values 28.5.  (A launch that begins cold, with
// nothing ahead of it, takes 21 of the first.)
//
// Running maximum: a row keeps a reference maximum that is only raised when the
// tile's maximum exceeds it by more than 2^8 (in the base-2 exponent), so P
// stays <= 256 and the accumulator in tensor memory is rescaled rarely; the row
// sum uses the same reference, and the final division makes the result the
// exact softmax-weighted mean whatever the reference was.
//
// Rows of 256 features that are keys and values at once (a latent with its rotated part: one
// key head for all query heads): a stage holds the tile once; the first product reads it
// with the features contracted, the second with the keys contracted.  A tile's 2 x 128 x 128 x 256
// multiply-adds are 2,048 cycles of the tensor pipe, 1,792 where only 192 features are asked for (31.0 -> 29.0 us
// a layer): there a group's softmax, its second product and its next scores stand in a row, 4,500 cycles for
// two tiles, since 512 columns hold no third buffer of scores.
//
// Sizes: head size 64 or 128, or 256 if the pages' rows are keys and values at once; page size a power of two from 8 to 128; any head
// counts and group sizes; window.  Anything else is refused and the mma.sync
// kernel runs.  Every wait is bounded (tc_common.cuh).
// Reference counterpart: `attention_prefill_exact_*`
// (engine/kernels/kernels.cu:2257-2275).
#define CB_PDL_BIT 1      // this file's bit in CRUCIBLE_PDL
#include <type_traits>
#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int ROWS = 128;            // query rows per block = tensor-memory lanes
constexpr int KEYS = 128;            // keys per tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RAISE = 8.0f;        // raise the reference maximum when exceeded by 2^8

struct TcAttnParams {
    const __nv_bfloat16* qkv;
    int qkv_stride;
    __nv_bfloat16* out;
    int out_stride;
    const int* req_row_start;
    const int* req_first_pos;
    const int* block_table;
    int table_stride;
    int n_heads, n_kv_heads, n_rep, n_requests, page_tokens, page_shift;
    int lead, lead_ranks;    // requests at the head of a single token each, and the tile ranks they take
    float scale_log2;
    int window;
    int keep_first;          // with a window: keys before this position stay visible to every later row
    int chunked;             // 1: `window` is the size of chunks counted from position 0: a row reads
                             // the keys of its own chunk up to itself
    float out_scale;         // every result times this
    const float* sinks;      // [n_heads] or null: exp(sink) joins a row's denominator, with no value
    const __nv_bfloat16* gate;   // logits: every result times sigmoid(logit); rows laid out like `out`, or
    int gate_stride;             // (GATE_HEAD) one logit a head
    int tile_rows;           // query rows of a tile: whole tokens' groups of heads
    int q_boxes;             // 1: the queries (and the gate's logits) come in by TMA; tile_rows is 128 else
    int n_pages;             // of the pool
    int runs;                // 1: the 4-D maps may be used for tiles whose pages are consecutive
    int* status;
};

// GATE: the results' gate, fixed when it is compiled: the epilogue runs once per block and its instructions
// come from memory (12 heads of 64 without a gate, a 2,048-token prompt: 32 us; with the code of the gate of a
// logit a result beside it 0.3 us more, of both gates 1.4).
enum Gate { GATE_NONE = 0, GATE_RESULT = 1, GATE_HEAD = 2 };

// HD: the head size, 64, 128 or (keys and values at once) 256.  A tile's operand of 64 features a row
// is one swizzle atom wide: [rows][128 bytes].
// The ring holds what the loader brings, in the order in which the MMA thread takes it.  Head sizes 64
// and 128: the keys of the first S_BUFS tiles, then V_t and K_(t + S_BUFS) in turn, one operand tile a slot; two
// neighbouring slots are one release, of which there are PAIRS.  256:
// a tile's features 0-127, then 128-255; a slot is free once the second product has read it.  Five
// slots are what 227 KB hold beside the queries: the upper half of tile t + 2 travels while the
// second product of tile t reads its own upper half.
// NARROW (256): only the first 192 features are values (a latent; the rotated part is key alone).  Three tiles'
// 192 features and one tile's last 64 then: the last 64 are free again when the tile's scores are there, so all of
// tile t + 2 is there when its scores' turn comes, and a second product is a quarter shorter.
template <int HD, bool NARROW>
struct Storage {
    static constexpr bool BOTH = HD == 256;                 // a cached row is key and value
    static constexpr int VALUES = NARROW ? 192 : HD;        // features of a result
    static constexpr int PART = NARROW ? 64 : BOTH ? 128 : HD;      // features of a slot
    static constexpr int PARTS = HD / PART;
    static constexpr int HALVES = PART / 64;
    static constexpr int PAIRS = HD == 64 ? 4 : 3;
    static constexpr int SLOTS = NARROW ? 10 : BOTH ? 5 : 2 * PAIRS;
    static constexpr int FULLS = NARROW ? 4 : SLOTS;        // narrow: three tiles' 192 features, then the last 64
    static constexpr int RELEASES = NARROW ? 4 : BOTH ? SLOTS : PAIRS;
    // buffers of scores: what 512 columns of tensor memory hold beside the accumulators.  With three the
    // next scores of a group are there when it asks for them; with two they follow its tile's second product.
    static constexpr int S_BUFS = BOTH ? 2 : 3;
    // two softmax groups of four warps take the tiles in turn (tile j: group j % 2).  Head size 64: each with its
    // own reference maximum, sum and accumulator, merged at the end.  Else (SHARED) one accumulator, for
    // which a row's reference goes from tile to tile through shared memory: two of 128 columns would leave
    // room for two buffers of scores, and the next scores would wait for the second product of two tiles back.
    static constexpr int GROUPS = 2;
    static constexpr bool SHARED = HD > 64;
    static constexpr int THREADS = 64 + 128 * GROUPS;       // loader, MMA thread, the softmax groups
    alignas(1024) uint8_t q[HD / 64][ROWS * 128];
    alignas(1024) uint8_t ring[SLOTS][HALVES][KEYS * 128];
    alignas(8) uint64_t full[FULLS];
    uint64_t empty[RELEASES];
    uint64_t q_full, gate_full, o_done;
    uint64_t s_full[S_BUFS], p_half[S_BUFS], p_full[S_BUFS], pv_done[2], m_full[2];
    float m_row[2][ROWS];                                   // shared: a row's reference as of a tile (tile j: j & 1)
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// The first key that a row at position `pos` reads behind the kept first tokens.
__device__ __forceinline__ int first_key(const TcAttnParams& p, int pos) {
    if (p.window <= 0) return 0;
    return p.chunked ? pos - pos % p.window : max(0, pos - p.window + 1);
}

// 2^x by the special-function unit, flushing denormals: the argument is a score
// minus a maximum, so a result below 2^-126 counts as nothing in the row's sum.
__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Two floats in one 64-bit register pair, and the instructions on the pair.
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void pair_to(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// 1 / (1 + e^-x), by t = e^-|x|: 1 / (1 + t), or t / (1 + t) for x < 0.  So the denominator is 1 to 2, where
// the approximate division has its two units in the last place (its IEEE form, inlined 32 times, is what a block would wait
// for at its end: 16 heads of 128, a window of 1,024, 2,048 tokens 32.9 us a layer with it, 26.5 so), and a logit
// far below zero keeps its digits: all 65,536 logits give the bf16 nearest to the true value.  A factor of its own, so
// that a logit a head and the same logit at each of its features give the same bits.
__device__ __forceinline__ float sigmoid(float x) {
    const float t = expf(-fabsf(x));
    return __fdividef(x < 0.f ? t : 1.f, 1.f + t);
}

// the low n bits
__device__ __forceinline__ uint32_t bits_below(int n) {
    return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u;
}

template <int HD, int GATE, bool NARROW>
__global__ void __launch_bounds__(Storage<HD, NARROW>::THREADS, 1)
attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                         const __grid_constant__ CUtensorMap run_k, const __grid_constant__ CUtensorMap run_v,
                         const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_gate,
                         const TcAttnParams p) {
    // 1024-byte alignment (the swizzled tiles need it) is asked of the declaration
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    using Store = Storage<HD, NARROW>;
    constexpr int NH = HD / 64, SLOTS = Store::SLOTS, GROUPS = Store::GROUPS, HALVES = Store::HALVES;
    constexpr int S_BUFS = Store::S_BUFS;
    constexpr bool BOTH = Store::BOTH, SHARED = Store::SHARED;
    constexpr uint32_t SLOT_BYTES = KEYS * Store::PART * 2;
    constexpr uint32_t TMEM_COLS = 512;                  // scores: 128 columns a buffer, then O
    Store& s = *reinterpret_cast<Store*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // grid (heads, requests, tile ranks), the tile rank slowest: blocks start in order of
    // weight over the whole launch, the longest rows first (and no thread divides by a run-time
    // value to find its place: that costs about a hundred cycles each time).  Single tokens at the
    // head of the step have a tile each and lie in ranks of their own ahead of the portions': a
    // block without work is not free, it waits for the SM's shared memory like another (48 tokens
    // beside a portion of 2,048, 16 heads of 64 on 4, a window of 512, with a rank of the
    // portion's 64 for each of them: 12,288 blocks without work, the layer 270 us, 125 now).
    const int kv_head = blockIdx.x;
    int req = blockIdx.y, rank = blockIdx.z;
    if (p.lead > 0) {
        if (rank < p.lead_ranks) {
            req += rank * (int)gridDim.y;
            rank = 0;
            if (req >= p.lead) return;
        } else {
            req += p.lead;
            rank -= p.lead_ranks;
        }
    }
    volatile int* abort_flag = &s.abort_flag;

    if (threadIdx.x == 0) {
        for (int i = 0; i < Store::FULLS; ++i) tc::mbar_init(&s.full[i], 1);
        for (int i = 0; i < Store::RELEASES; ++i) tc::mbar_init(&s.empty[i], 1);
        tc::mbar_init(&s.q_full, p.q_boxes ? 1 : 4 * GROUPS);
        tc::mbar_init(&s.gate_full, 1);
        tc::mbar_init(&s.o_done, 1);
        for (int b = 0; b < S_BUFS; ++b) {
            tc::mbar_init(&s.s_full[b], 1);
            tc::mbar_init(&s.p_half[b], 4);               // one arrival per softmax warp
            tc::mbar_init(&s.p_full[b], 4);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&s.pv_done[b], 1);
            tc::mbar_init(&s.m_full[b], 4);
        }
        s.abort_flag = 0;
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&map_k);
        tc::prefetch_tensormap(&map_v);
        tc::prefetch_tensormap(&map_q);
        if (p.runs) {
            tc::prefetch_tensormap(&run_k);
            tc::prefetch_tensormap(&run_v);
        }
    }
    if (warp == 1) {
        tc::tmem_alloc(&s.tmem_base, TMEM_COLS);
        tc::tmem_relinquish();
    }
    // What follows reads the step's metadata, which was uploaded before the step began: the
    // kernels ahead in the stream write none of it, so it is read, and the first tiles'
    // table entries looked up, before the wait for them.
    const int n_rep = p.n_rep, tile_rows = p.tile_rows;
    const int row_base = p.req_row_start[req];
    const int n_new = p.req_row_start[req + 1] - row_base;
    const int n_rows = n_new * n_rep;
    const int q_tiles = (n_rows + tile_rows - 1) / tile_rows;
    const bool active = rank < q_tiles;
    const int qt = active ? q_tiles - 1 - rank : 0;               // heaviest tiles first
    const int first_pos = p.req_first_pos[req];
    const int* table = p.block_table + (size_t)req * p.table_stride;

    // the block's keys: from the first key any of its rows may read to its last position
    const int first_row = qt * tile_rows;
    const int last_row = min(n_rows, first_row + tile_rows) - 1;
    const int first_tok = first_row / n_rep;
    const int max_pos = first_pos + last_row / n_rep;
    const int min_pos = first_pos + first_tok;
    int key_lo = first_key(p, min_pos);
    key_lo = key_lo / KEYS * KEYS;
    const int key_end = max_pos + 1;
    // kept first tokens: their tiles that lie wholly before the window's first tile come first
    // (those inside it are part of the window's own tiles and only change the mask)
    const int kept_tiles = (active && p.window > 0 && p.keep_first > 0)
                               ? min((p.keep_first + KEYS - 1) / KEYS, key_lo / KEYS) : 0;
    const int n_tiles = active ? kept_tiles + (key_end - key_lo + KEYS - 1) / KEYS : 0;
    auto tile_key0 = [&](int j) { return j < kept_tiles ? j * KEYS : key_lo + (j - kept_tiles) * KEYS; };

    // rows beyond the tile's (a group size that does not divide 128): zeros, like any row not stored
    for (int i = tile_rows * 8 * NH + threadIdx.x; i < ROWS * 8 * NH; i += blockDim.x) {
        const int r = i / (8 * NH), c = i % (8 * NH);
        *reinterpret_cast<uint4*>(s.q[c >> 3] + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(0, 0, 0, 0);
    }
    tc::fence_proxy_async();
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem_s = s.tmem_base;          // + 128 a buffer
    const uint32_t tmem_o = s.tmem_base + S_BUFS * 128;

    if (warp == 0) {
        // ---- loader: the warp together (a lane a page), so that scattered pages' table entries
        // and copies go out side by side -----------------------------------------------------
        // a kept tile's pages beyond the last kept token's may have gone back to the pool: their
        // keys are masked, and they are read from the last kept page instead
        const int last_kept_page = p.keep_first > 0 ? (p.keep_first - 1) >> p.page_shift : 0;
        const int pages_per_tile = KEYS >> p.page_shift;
        auto lookup = [&](int j) -> int {
            const int key0 = tile_key0(j < n_tiles ? j : 0);
            int index = (key0 >> p.page_shift) + (lane < pages_per_tile ? lane : 0);
            if (j < kept_tiles && index > last_kept_page) index = last_kept_page;
            index = index < p.table_stride ? index : p.table_stride - 1;
            const int page = table[index];
            return page < 0 ? 0 : page;               // an entry given back early: never read
        };
        // a tile's features from `feature` on, 64 to a slot's half, to `to`; N halves
        auto copy = [&](int page, bool values, int feature, uint8_t (*to)[KEYS * 128], auto halves, uint64_t* full) {
            constexpr int N = decltype(halves)::value;
            // pages that follow one another in the pool come in with one copy per half
            const int page0 = __shfl_sync(0xffffffffu, page, 0);
            const bool run = __all_sync(0xffffffffu, lane >= pages_per_tile || page == page0 + lane) && p.runs != 0 &&
                             page0 + pages_per_tile <= p.n_pages;
            if (lane == 0) tc::mbar_expect_tx(full, N * KEYS * 128);
            __syncwarp();
            if (run) {
                if (lane < N)
                    tc::tma_load_4d(to[lane], values ? &run_v : &run_k, full, feature + lane * 64, 0, kv_head, page0);
            } else if (lane < pages_per_tile) {
                const int dst = (lane << p.page_shift) * 128;
                const int y = (page * p.n_kv_heads + kv_head) << p.page_shift;
#pragma unroll
                for (int h = 0; h < N; ++h)
                    tc::tma_load_2d(to[h] + dst, values ? &map_v : &map_k, full, feature + h * 64, y);
            }
        };
        int item = 0, armed = 0;                      // the next slot's number; slots with copies sent
        auto send = [&](int page, bool values, int feature) -> bool {
            const int st = item % SLOTS;
            const int rel = BOTH ? item : item >> 1, round = rel / Store::RELEASES;
            // (A pair's first slot waits for both.  The second must not ask again: the last pair's release may
            // come round as soon as its first slot's values have been used, and the phase asked for is then
            // two behind, which reads as not over yet.)
            if (round > 0 && (BOTH || (item & 1) == 0) && !__all_sync(0xffffffffu, tc::mbar_wait(&s.empty[rel % Store::RELEASES], (round - 1) & 1, abort_flag))) {
                tc::give_up(abort_flag, p.status, tc::ST_PRODUCER_TIMEOUT);
                return false;
            }
            copy(page, values, feature, s.ring[st], std::integral_constant<int, HALVES>{}, &s.full[st]);
            armed = ++item;
            return true;
        };
        int pg0 = lookup(0), pg1 = lookup(1), pg2 = lookup(2);
        cb_pdl_wait();
        cb_pdl_trigger();     // the block holds its tensor memory: a successor that asks for some queues behind it
        bool ok = n_tiles > 0;
        if (ok && p.q_boxes && lane == 0) {
            tc::mbar_expect_tx(&s.q_full, NH * tile_rows * 128);
#pragma unroll
            for (int h = 0; h < NH; ++h)
                tc::tma_load_3d(s.q[h], &map_q, &s.q_full, h * 64, kv_head * n_rep, row_base + first_tok);
        }
        __syncwarp();
        int last_armed = 0;                           // narrow: tiles whose last 64 features have been sent
        if constexpr (NARROW) {
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int st = j % 3;
                ok = (j < 3 || __all_sync(0xffffffffu, tc::mbar_wait(&s.empty[st], (j / 3 - 1) & 1, abort_flag)));
                if (ok) {
                    copy(pg0, false, 0, &s.ring[3 * st][0], std::integral_constant<int, 3>{}, &s.full[st]);
                    armed = j + 1;
                    ok = j < 1 || __all_sync(0xffffffffu, tc::mbar_wait(&s.empty[3], (j - 1) & 1, abort_flag));
                }
                if (ok) {
                    copy(pg0, false, 192, &s.ring[9][0], std::integral_constant<int, 1>{}, &s.full[3]);
                    last_armed = j + 1;
                }
                if (!ok) tc::give_up(abort_flag, p.status, tc::ST_PRODUCER_TIMEOUT);
                pg0 = pg1, pg1 = pg2, pg2 = lookup(j + 3);
            }
        } else if (BOTH) {
            for (int j = 0; j < n_tiles && ok; ++j) {
                ok = send(pg0, false, 0) && send(pg0, false, 128);
                pg0 = pg1, pg1 = pg2, pg2 = lookup(j + 3);
            }
        } else if (ok) {
            int pg3 = lookup(3);
            ok = send(pg0, false, 0);
            if (ok && n_tiles > 1) ok = send(pg1, false, 0);
            if (ok && n_tiles > 2) ok = send(pg2, false, 0);
            for (int j = 0; j < n_tiles && ok; ++j) {
                ok = send(pg0, true, 0);
                if (ok && j + S_BUFS < n_tiles) ok = send(pg3, false, 0);
                pg0 = pg1, pg1 = pg2, pg2 = pg3, pg3 = lookup(j + 4);
            }
        }
        bool gate_sent = false;
        if (GATE == GATE_RESULT && p.q_boxes && ok) {
            // the gate's logits into the next free slots, beside the last tiles' work
            constexpr int N = BOTH ? 2 : 1;
            for (int i = 0; i < N && ok; ++i, ++item) {      // (two slots' worth: items are even by now)
                const int rel = BOTH ? item : item >> 1, round = rel / Store::RELEASES;
                ok = round == 0 || __all_sync(0xffffffffu, tc::mbar_wait(&s.empty[rel % Store::RELEASES], (round - 1) & 1, abort_flag));
                if (!ok) {
                    tc::give_up(abort_flag, p.status, tc::ST_PRODUCER_TIMEOUT);
                } else if (lane == 0) {
                    gate_sent = true;
                    if (i == 0) tc::mbar_expect_tx(&s.gate_full, NH * tile_rows * 128);
                    for (int h = 0; h < HALVES; ++h)
                        tc::tma_load_3d(s.ring[item % SLOTS][h], &map_gate, &s.gate_full, i * 128 + h * 64, kv_head * n_rep,
                                        row_base + first_tok);
                }
                __syncwarp();
            }
        }
        // an abort leaves no copy in flight behind
        if (*abort_flag && lane == 0) {
            auto drain = [&](uint64_t* bar, uint32_t parity) {
                for (uint32_t t = 0; t < tc::WAIT_LIMIT; ++t)
                    if (tc::mbar_try_wait(bar, parity)) break;
            };
            if (p.q_boxes && n_tiles > 0) drain(&s.q_full, 0);
            constexpr int AHEAD = NARROW ? 3 : SLOTS;
            for (int i = armed > AHEAD ? armed - AHEAD : 0; i < armed; ++i) drain(&s.full[i % AHEAD], (i / AHEAD) & 1);
            if (last_armed > 0) drain(&s.full[Store::FULLS - 1], (last_armed - 1) & 1);
            if (gate_sent) drain(&s.gate_full, 0);
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp walks the tiles together, one lane sends ---------------------
        // Order: the first S_BUFS tiles' scores, then O += P_t V_t and S_(t + S_BUFS) for every tile.  P lies
        // over the scores that it was made from, so the scores that take its buffer follow the second
        // product, which the tensor pipe works off in order; the softmax of the tiles between runs beside both.
        if (n_tiles > 0) {
            const bool sender = tc::elect_one();
            constexpr uint32_t idesc_qk = tc::instr_desc_bf16(ROWS, KEYS);
            constexpr uint32_t idesc_pv = tc::instr_desc_bf16_b_mn(ROWS, NARROW ? 192 : Store::PART);
            // Operand descriptors by addition: the low word carries the address in 16-byte
            // units, the high word is the same for every tile.
            const uint64_t q_desc0 = tc::smem_desc_sw128(tc::smem_u32(s.q[0]));
            const uint32_t desc_hi = (uint32_t)(q_desc0 >> 32);
            const uint32_t q_lo = (uint32_t)q_desc0;
            constexpr uint32_t HALF = KEYS * 128 >> 4, SLOT = KEYS * Store::PART * 2 >> 4;
            const uint32_t k_lo0 = (uint32_t)tc::smem_desc_sw128(tc::smem_u32(s.ring[0][0]));
            // the values, all features of a slot in one instruction: 64 of them lie together, the next 64 a
            // leading offset of HALF on
            const uint32_t v_lo0 = (k_lo0 & 0xFFFFu) | (HALF << 16);
            auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
                return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, abort_flag));
            };
            int item = 0;                         // the next slot that has not been taken
            // S_j = Q K_j^T into buffer `to`
            int to = 0;
            auto scores = [&](int j) -> bool {
                const uint32_t d_s = tmem_s + to * 128;
#pragma unroll
                for (int part = 0; part < Store::PARTS; ++part) {
                    const int st = NARROW ? (part < 3 ? 3 * (j % 3) + part : 9) : item % SLOTS;
                    if (NARROW ? part == 0 && !wait(&s.full[j % 3], (j / 3) & 1) : !wait(&s.full[st], (item / SLOTS) & 1)) return false;
                    if (NARROW && part == 3 && !wait(&s.full[3], j & 1)) return false;
                    tc::tc_fence_after_sync();
                    const uint32_t k_lo = k_lo0 + st * SLOT;
                    if (sender) {
#pragma unroll
                        for (int k = 0; k < Store::PART / 16; ++k) {
                            const uint64_t q_desc = tc::desc_of(q_lo + (part * HALVES + (k >> 2)) * HALF + 2 * (k & 3), desc_hi);
                            const uint64_t k_desc = tc::desc_of(k_lo + (k >> 2) * HALF + 2 * (k & 3), desc_hi);
                            if (k == 0 && part == 0) tc::umma_bf16(d_s, q_desc, k_desc, idesc_qk, 0u);
                            else tc::umma_bf16_add(d_s, q_desc, k_desc, idesc_qk);
                        }
                    }
                    ++item;
                }
                if (sender) {
                    tc::umma_commit(&s.s_full[to]);
                    if (NARROW) tc::umma_commit(&s.empty[3]);
                    if (!BOTH && j == 1) tc::umma_commit(&s.empty[0]);      // the pairs: K0 and K1, then K_(t+2) and V_t
                }
                if (++to == S_BUFS) to = 0;
                return true;
            };
            auto products = [&](int t) -> bool {  // O += P_t V_t: 128 keys in eight steps of 16
                const uint32_t d_o = tmem_o + (SHARED ? 0u : (uint32_t)(t & 1) * HD);
                const int b = t % S_BUFS;
                const uint32_t p_at = tmem_s + b * 128;
                const uint32_t parity = (t / S_BUFS) & 1;
#pragma unroll
                for (int part = 0; part < (NARROW ? 1 : Store::PARTS); ++part) {
                    // 256: the tile's own slots, which the scores have taken (and freed by this)
                    const int st = NARROW ? 3 * (t % 3) : BOTH ? (2 * t + part) % SLOTS : item % SLOTS;
                    if (!BOTH && !wait(&s.full[st], (item / SLOTS) & 1)) return false;
                    const uint32_t v_lo = v_lo0 + st * SLOT;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        if (part == 0 && !wait(half ? &s.p_full[b] : &s.p_half[b], parity)) return false;
                        tc::tc_fence_after_sync();
                        if (sender) {
#pragma unroll
                            for (int k = 4 * half; k < 4 * half + 4; ++k) {
                                // 16 keys further down V: 16 rows of 128 bytes = 128 descriptor units
                                const uint64_t v_desc = tc::desc_of(v_lo + 128 * k, desc_hi);
                                if (k == 0) tc::umma_bf16_ts(d_o + part * 128, p_at + 8 * k, v_desc, idesc_pv, t >= (SHARED ? 1 : GROUPS) ? 1u : 0u);
                                else tc::umma_bf16_ts_add(d_o + part * 128, p_at + 8 * k, v_desc, idesc_pv);
                            }
                        }
                    }
                    if (BOTH && sender) tc::umma_commit(&s.empty[NARROW ? t % 3 : st]);
                    if (!BOTH) ++item;
                }
                if (sender) {
                    if (BOTH) tc::umma_commit(&s.pv_done[t & 1]);
                    // (not after the last tile: the loader may still be about to ask for this barrier's phase before)
                    if (!BOTH && t + 1 < n_tiles) tc::umma_commit(&s.empty[(t + 1) % Store::RELEASES]);
                    if (t == n_tiles - 1) tc::umma_commit(&s.o_done);
                }
                return true;
            };
            bool ok = wait(&s.q_full, 0);
            for (int j = 0; j < S_BUFS && j < n_tiles && ok; ++j) ok = scores(j);
            for (int t = 0; t < n_tiles && ok; ++t) {
                ok = products(t);
                if (ok && t + S_BUFS < n_tiles) ok = scores(t + S_BUFS);
            }
            if (!ok && lane == 0) tc::give_up(abort_flag, p.status, tc::ST_MMA_TIMEOUT);
        }
    } else {
        // ---- softmax: warps 2..5 (and 6..9: the second group), one thread per row =
        // tensor-memory lane; a group takes every GROUPS-th tile -------------------------------
        const int quarter = warp & 3;
        const int group = (warp - 2) >> 2;
        const uint32_t tmem_mine = tmem_o + (SHARED ? 0u : (uint32_t)group * HD);
        const int r = quarter * 32 + lane;
        const int row = first_row + r;
        const bool real = active && r < tile_rows && row < n_rows;
        // rows that are not the request's are computed like rows that may read every key and are
        // not stored: they keep a tile's fast path open
        const int pos = real ? first_pos + row / n_rep : (1 << 30);
        const int lo = real ? first_key(p, pos) : 0;
        const uint32_t lane_bits = (uint32_t)(quarter * 32) << 16;
        cb_pdl_wait();
        // what the row needs at its end, asked for now
        __nv_bfloat16* dst = nullptr;
        const __nv_bfloat16* gate = nullptr;
        float gate_f = 1.f;
        float sink = -INFINITY;                       // in the base-2 exponent
        if (real) {
            const int tok = row_base + row / n_rep, head = kv_head * n_rep + row % n_rep;
            if (p.sinks != nullptr) sink = p.sinks[head] * LOG2E;
            dst = p.out + (size_t)tok * p.out_stride + (size_t)head * HD;
            if (GATE == GATE_RESULT) gate = p.gate + (size_t)tok * p.gate_stride + (size_t)head * HD;
            if (GATE == GATE_HEAD)
                gate_f = sigmoid(__bfloat162float(p.gate[(size_t)tok * p.gate_stride + head]));
        }
        if (!p.q_boxes && n_tiles > 0) {
            // group sizes whose tiles would leave much of the 128 rows empty: the rows by hand,
            // 16-byte pieces into the 128-byte swizzle
            for (int i = threadIdx.x - 64; i < ROWS * 8 * NH; i += 128 * GROUPS) {
                const int rr = i / (8 * NH), c = i % (8 * NH);
                const int at = first_row + rr;
                uint4 val = make_uint4(0, 0, 0, 0);
                if (at < n_rows) {
                    const int tok = row_base + at / n_rep, head = kv_head * n_rep + at % n_rep;
                    val = *reinterpret_cast<const uint4*>(p.qkv + (size_t)tok * p.qkv_stride + (size_t)head * HD + c * 8);
                }
                *reinterpret_cast<uint4*>(s.q[c >> 3] + rr * 128 + (((c & 7) ^ (rr & 7)) << 4)) = val;
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&s.q_full);
        }
        float m_ref = -INFINITY, l = 0.f;
        bool ok = true;
        auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
            bool got = tc::mbar_wait(bar, parity, abort_flag);
            if (!got && !*abort_flag) tc::give_up(abort_flag, p.status, tc::ST_EPILOGUE_TIMEOUT);
            return __all_sync(0xffffffffu, got);
        };
        const uint64_t scale2 = pair_of(p.scale_log2, p.scale_log2);
        for (int j = group; j < n_tiles; j += GROUPS) {
            const int key0 = tile_key0(j);
            const int b = j % S_BUFS;
            ok = wait_all(&s.s_full[b], (j / S_BUFS) & 1);
            if (!ok) break;
            tc::tc_fence_after_sync();
            const uint32_t at = tmem_s + b * 128 + lane_bits;
            // keys of this tile the row may read: [first, last] relative to key0, and those before
            // `kept`.  Most tiles lie wholly inside every row's range and skip the test; in the
            // others the masked scores go back where they came from.
            const int last = pos - key0, first = lo - key0;
            const int kept = p.keep_first - key0;     // keys before this one are kept first tokens (<= 0: none here)
            const bool inside = __all_sync(0xffffffffu, last >= KEYS - 1 && first <= 0);
            float mc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            // The scores are read twice, 64 at a time in a loop that is not unrolled: the code of
            // both passes over all 128 comes from memory at a block's first tile, and the registers
            // would not hold them beside the rest.
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                uint32_t sv[2][32];
                tc::tmem_ld_32x32(at + 64 * h, sv[0]);
                tc::tmem_ld_32x32(at + 64 * h + 32, sv[1]);
                tc::tmem_ld_wait();
                if (!inside) {
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int k0 = 64 * h + 32 * c;
                        const uint32_t seen = bits_below(last + 1 - k0) & (~bits_below(first - k0) | bits_below(kept - k0));
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (!(seen >> i & 1u)) sv[c][i] = __float_as_uint(-INFINITY);
                        tc::tmem_st_32x32(at + k0, sv[c]);
                    }
                    tc::tmem_st_wait();
                }
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float& m = mc[2 * c + ((i >> 1) & 1)];
                        m = max3(m, __uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1]));
                    }
            }
            float mx = fmaxf(fmaxf(mc[0], mc[1]), fmaxf(mc[2], mc[3]));
            mx *= p.scale_log2;
            // raise the reference maximum only when it is exceeded by far; the accumulator
            // in tensor memory is rescaled then, by the whole warp at once, after the second product
            // that was the last to add to it.  A shared accumulator's reference is the one of the tile before.
            float m_was = m_ref;
            if (SHARED && j > 0) {
                ok = wait_all(&s.m_full[(j - 1) & 1], ((j - 1) >> 1) & 1);
                if (!ok) break;
                m_was = s.m_row[(j - 1) & 1][r];
            }
            float m_new = m_was;
            if (mx > m_was + RAISE || (m_was == -INFINITY && mx > -INFINITY)) m_new = mx;
            if (SHARED) {
                s.m_row[j & 1][r] = m_new;
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&s.m_full[j & 1]);
            }
            if (__any_sync(0xffffffffu, m_new != m_ref)) {      // (of what this group summed, of what all have)
                const float mine = m_new == m_ref ? 1.f : m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_new);
                l *= mine;
                m_ref = m_new;
            }
            if (j >= (SHARED ? 1 : GROUPS) && __any_sync(0xffffffffu, m_new != m_was)) {
                const float corr = m_new == m_was ? 1.f : m_was == -INFINITY ? 0.f : exp2f(m_was - m_new);
                constexpr int BACK = SHARED ? 1 : GROUPS, R = Store::RELEASES;
                ok = BOTH ? wait_all(&s.pv_done[(j - BACK) & 1], ((j - BACK) >> 1) & 1)
                          : wait_all(&s.empty[(j - BACK + 1) % R], ((j - BACK + 1) / R) & 1);
                if (!ok) break;
                tc::tc_fence_after_sync();
#pragma unroll 1
                for (int c0 = 0; c0 < Store::VALUES; c0 += 32) {
                    uint32_t v[32];
                    tc::tmem_ld_32x32(tmem_mine + lane_bits + c0, v);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
                    tc::tmem_st_32x32(tmem_mine + lane_bits + c0, v);
                }
                tc::tmem_st_wait();
            }
            // P = exp2(s * scale - reference) in bf16, two a column, over the scores' own columns:
            // keys 0-63 into the first 32, 64-127 into the next (their scores, columns 64-127, are
            // read after the first half's, whose columns are 0-63)
            const float off = m_ref == -INFINITY ? 0.f : -m_ref;
            const uint64_t off2 = pair_of(off, off);
            uint64_t sum[4] = {0, 0, 0, 0};
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                uint32_t sv[2][32], pk[32];
                tc::tmem_ld_32x32(at + 64 * h, sv[0]);
                tc::tmem_ld_32x32(at + 64 * h + 32, sv[1]);
                tc::tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float e0, e1;
                        pair_to(fma2(pair_of(__uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1])), scale2, off2), e0, e1);
                        e0 = ex2_fast(e0);
                        e1 = ex2_fast(e1);
                        uint64_t& into = sum[(i >> 1) & 3];
                        into = add2(into, pair_of(e0, e1));
                        pk[16 * c + (i >> 1)] = pack_bf16(e0, e1);
                    }
                tc::tmem_st_32x32(at + 32 * h, pk);
                tc::tmem_st_wait();
                tc::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(h ? &s.p_full[b] : &s.p_half[b]);
            }
            float s0, s1;
            pair_to(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])), s0, s1);
            l += s0 + s1;
        }
        // ---- the output: O / l ------------------------------------------------------------
        const int my_tiles = n_tiles > group ? (n_tiles - group + GROUPS - 1) / GROUPS : 0;
        if (n_tiles > 0 && ok) ok = wait_all(&s.o_done, 0);
        if (GATE == GATE_RESULT && p.q_boxes && n_tiles > 0 && ok) ok = wait_all(&s.gate_full, 0);
        // where the loader put the gate's logits: behind the ring's last slot (see there)
        const int gate_item = 2 * n_tiles;
        // 32 results of the row, from feature c0 on, to the queries' place, which nothing reads any more
        auto close = [&](float (&o)[32], int c0) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
                if (GATE == GATE_RESULT) {
                    const int f = c0 + 8 * q4, piece = (f & 63) >> 3;
                    const void* from = gate + f;
                    if (p.q_boxes) {
                        const int st = (gate_item + (BOTH ? f >> 7 : 0)) % SLOTS;
                        from = s.ring[st][(f >> 6) & (HALVES - 1)] + r * 128 + ((piece ^ (r & 7)) << 4);
                    }
                    const uint4 raw = *reinterpret_cast<const uint4*>(from);
                    const __nv_bfloat16* g = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[8 * q4 + i] *= sigmoid(__bfloat162float(g[i]));
                }
                if (GATE == GATE_HEAD) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[8 * q4 + i] *= gate_f;
                }
                uint4 w;
                w.x = pack_bf16(o[8 * q4 + 0], o[8 * q4 + 1]);
                w.y = pack_bf16(o[8 * q4 + 2], o[8 * q4 + 3]);
                w.z = pack_bf16(o[8 * q4 + 4], o[8 * q4 + 5]);
                w.w = pack_bf16(o[8 * q4 + 6], o[8 * q4 + 7]);
                const int f = c0 + 8 * q4;
                *reinterpret_cast<uint4*>(s.q[f >> 6] + r * 128 + ((((f & 63) >> 3) ^ (r & 7)) << 4)) = w;
            }
        };
        // The warp's 32 rows from there to memory, several rows' pieces side by side: a store of one piece by
        // each of 32 rows touches 32 lines and takes the memory pipe 32 cycles (128 rows of 256 features
        // that way 5,200 cycles of a block, of 64 features with two groups 2,200).
        auto write_rows = [&]() {
            constexpr int MINE = Store::VALUES / GROUPS, ACROSS = MINE % 64 ? 4 : 8;      // pieces of a row side by side
            __syncwarp();
            const unsigned long long mine = real ? (unsigned long long)dst : 0ull;
#pragma unroll 4
            for (int r0 = 0; r0 < 32; r0 += 32 / ACROSS) {
                const int rr = r0 + lane / ACROSS, at = quarter * 32 + rr;
                __nv_bfloat16* to = (__nv_bfloat16*)__shfl_sync(0xffffffffu, mine, rr);
                uint4 w[MINE / (8 * ACROSS)];
#pragma unroll
                for (int i = 0; i < MINE / (8 * ACROSS); ++i) {
                    const int f = group * MINE + 8 * (i * ACROSS + lane % ACROSS);
                    w[i] = *reinterpret_cast<const uint4*>(s.q[f >> 6] + at * 128 + ((((f & 63) >> 3) ^ (at & 7)) << 4));
                }
                if (to != nullptr)
#pragma unroll
                    for (int i = 0; i < MINE / (8 * ACROSS); ++i)
                        *reinterpret_cast<uint4*>(to + group * MINE + 8 * (i * ACROSS + lane % ACROSS)) = w[i];
            }
        };
        // Each group holds the sums over its own tiles against the reference of its last one.
        // A row's two states meet in shared memory; every thread comes to the barrier,
        // whatever happened to its waits.  Then group g writes its half of the features.
        float2* const merge = reinterpret_cast<float2*>(s.ring[NARROW ? 0 : (gate_item + 2) % SLOTS][0]);     // (nothing is there any more)
        merge[group * ROWS + r] = make_float2(my_tiles > 0 ? m_ref : -INFINITY, my_tiles > 0 ? l : 0.f);
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (ok && n_tiles > 0 && !*abort_flag) {
            tc::tc_fence_after_sync();
            const float2 other = merge[(group ^ 1) * ROWS + r];
            const float m_mine = my_tiles > 0 ? m_ref : -INFINITY, m_both = fmaxf(m_mine, other.x);
            const float m_all = fmaxf(m_both, sink);
            const float f_mine = m_mine == -INFINITY ? 0.f : exp2f(m_mine - m_all);
            const float f_other = other.x == -INFINITY ? 0.f : exp2f(other.x - m_all);
            float l_all = (my_tiles > 0 ? l : 0.f) * f_mine + other.y * f_other;
            if (sink != -INFINITY) l_all += exp2f(sink - m_all);
            const float inv = l_all > 0.f ? p.out_scale / l_all : 0.f;
            // (a shared accumulator stands against the last tile's reference, the higher one)
            const float w_mine = SHARED ? fmaxf(f_mine, f_other) * inv : f_mine * inv, w_other = f_other * inv;
            // An accumulator that no MMA has written holds whatever was there and is not
            // read.  Whether a group had tiles is the same for every thread of the block,
            // as it must be: the loads are the whole warp's (.sync.aligned).  A row that
            // could read none of a group's keys has weight 0 and finite sums (zeros) there.
            const bool mine_any = SHARED || my_tiles > 0, other_any = !SHARED && n_tiles > my_tiles;
#pragma unroll 1
            for (int c0 = group * (Store::VALUES / 2); c0 < (group + 1) * (Store::VALUES / 2); c0 += 32) {
                uint32_t a[32], b[32];
                if (mine_any) tc::tmem_ld_32x32(tmem_mine + lane_bits + c0, a);
                if (other_any) tc::tmem_ld_32x32(tmem_o + (uint32_t)(group ^ 1) * HD + lane_bits + c0, b);
                tc::tmem_ld_wait();
                if (real) {
                    float o[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        o[i] = (mine_any ? __uint_as_float(a[i]) * w_mine : 0.f) +
                               (other_any ? __uint_as_float(b[i]) * w_other : 0.f);
                    close(o, c0);
                }
            }
            write_rows();
        }
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc(s.tmem_base, TMEM_COLS);
    }
}

template <int HD, int GATE, bool NARROW = false>
int launch_gate(dim3 grid, cudaStream_t st, const CUtensorMap (&maps)[6], const TcAttnParams& p) {
    constexpr int smem = (int)sizeof(Storage<HD, NARROW>);
    static_assert(smem <= 227 * 1024, "a block's shared memory");
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attention_tcgen05_kernel<HD, GATE, NARROW>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    cb_launch(attention_tcgen05_kernel<HD, GATE, NARROW>, grid, dim3(Storage<HD, NARROW>::THREADS), smem, st, maps[0],
              maps[1], maps[2], maps[3], maps[4], maps[5], p);
    return cb_last_error();
}

template <int HD>
int launch_as(int gate, dim3 grid, cudaStream_t st, const CUtensorMap (&maps)[6], const TcAttnParams& p) {
    switch (gate) {
        case GATE_NONE: return launch_gate<HD, GATE_NONE>(grid, st, maps, p);
        case GATE_RESULT: return launch_gate<HD, GATE_RESULT>(grid, st, maps, p);
    }
    return launch_gate<HD, GATE_HEAD>(grid, st, maps, p);
}

}  // namespace

// Attention for the rows of a step whose requests bring portions of prompts.
// k_cache / v_cache: [n_pages][n_kv_heads][page_tokens][head_dim] bf16; head_dim 64 or 128, or 256 where
// both are the same rows.
// keep_first (with a window): a row at position p reads j <= p with p - j < window or j < keep_first.
// chunked: `window` is a chunk's size (first_key).  sinks: [n_heads] or null.  Results times out_scale.
// n_rows: of qkv (and out, gate).  value_cols (0: all): the caller reads no result's features beyond that many; they may
// be left as they are.  lead: how many requests at the head bring a single token (as max_new_tokens is the others').
// gate: null, or logits: results times their sigmoids; laid out like `out`, rows of 16-byte pieces, or with
// gate_per_head [rows][n_heads].
CB_EXPORT int cb_attention_tcgen05_kept(const void* qkv, int qkv_stride, int n_rows, void* out, int out_stride,
                                        const void* k_cache, const void* v_cache, int n_pages,
                                        const int* req_row_start, const int* req_first_pos,
                                        const int* block_table, int table_stride, int n_requests,
                                        int max_new_tokens, int n_heads, int n_kv_heads, int head_dim,
                                        int page_tokens, float scale, int window, int chunked, int keep_first,
                                        float out_scale, const float* sinks, const void* gate, int gate_stride,
                                        int gate_per_head, int lead, int value_cols, int* status, void* stream) {
    if (n_requests <= 0 || max_new_tokens <= 0) return 0;
    if (keep_first < 0 || !(scale > 0.f)) return CB_ERR_UNSUPPORTED;
    if ((head_dim != 64 && head_dim != 128 && !(head_dim == 256 && k_cache == v_cache)) || n_heads % n_kv_heads != 0 || page_tokens < 8 || page_tokens > KEYS ||
        (page_tokens & (page_tokens - 1)) || (qkv_stride & 7) || (out_stride & 7) ||
        ((uintptr_t)qkv & 15) || ((uintptr_t)out & 15) || ((uintptr_t)k_cache & 15) ||
        ((uintptr_t)v_cache & 15) || (gate != nullptr && !gate_per_head && (((uintptr_t)gate & 15) || (gate_stride & 7))))
        return CB_ERR_UNSUPPORTED;
    int shift = 0;
    while ((1 << shift) < page_tokens) ++shift;
    CUtensorMap maps[6];
    CUtensorMap &mk = maps[0], &mv = maps[1], &rk = maps[2], &rv = maps[3];
    const uint64_t rows = (uint64_t)n_pages * n_kv_heads * page_tokens;
    if (!tc::make_map_2d(&mk, k_cache, rows, head_dim, head_dim, page_tokens)) return CB_ERR_UNSUPPORTED;
    if (!tc::make_map_2d(&mv, v_cache, rows, head_dim, head_dim, page_tokens)) return CB_ERR_UNSUPPORTED;
    // tiles of several pages: a second pair of maps that takes a run of pages at once
    rk = mk, rv = mv;
    const int pages_per_tile = KEYS / page_tokens;
    const bool runs = pages_per_tile > 1 &&
                      tc::make_map_pages(&rk, k_cache, n_pages, n_kv_heads, page_tokens, head_dim, pages_per_tile) &&
                      tc::make_map_pages(&rv, v_cache, n_pages, n_kv_heads, page_tokens, head_dim, pages_per_tile);
    // A tile takes whole tokens, all heads of the group, so that one box holds its rows.  Group sizes that
    // would leave more than an eighth of the 128 rows empty are cut anywhere and fetched by hand.
    const int n_rep = n_heads / n_kv_heads;
    TcAttnParams p;
    p.tile_rows = n_rep <= ROWS ? ROWS / n_rep * n_rep : 0;
    p.q_boxes = p.tile_rows >= ROWS - ROWS / 8;
    if (!p.q_boxes) p.tile_rows = ROWS;
    maps[4] = maps[5] = mk;
    if (p.q_boxes) {
        const uint32_t tokens = p.tile_rows / n_rep;
        if (!tc::make_map_heads(&maps[4], qkv, n_rows, n_heads, head_dim, qkv_stride, n_rep, tokens) ||
            (gate != nullptr && !gate_per_head &&
             !tc::make_map_heads(&maps[5], gate, n_rows, n_heads, head_dim, gate_stride, n_rep, tokens)))
            return CB_ERR_UNSUPPORTED;
    }
    p.n_pages = n_pages;
    p.runs = runs ? 1 : 0;
    p.qkv = (const __nv_bfloat16*)qkv;
    p.qkv_stride = qkv_stride;
    p.out = (__nv_bfloat16*)out;
    p.out_stride = out_stride;
    p.req_row_start = req_row_start;
    p.req_first_pos = req_first_pos;
    p.block_table = block_table;
    p.table_stride = table_stride;
    p.n_heads = n_heads;
    p.n_kv_heads = n_kv_heads;
    p.n_rep = n_rep;
    p.n_requests = n_requests;
    p.page_tokens = page_tokens;
    p.page_shift = shift;
    p.scale_log2 = scale * LOG2E;
    p.window = window;
    p.keep_first = window > 0 ? keep_first : 0;
    p.chunked = window > 0 && chunked ? 1 : 0;
    p.sinks = sinks;
    p.gate = (const __nv_bfloat16*)gate;
    p.gate_stride = gate_stride;
    p.out_scale = out_scale;
    p.status = status;
    const int q_tiles = (max_new_tokens * n_rep + p.tile_rows - 1) / p.tile_rows;
    if (n_requests > 65535 || q_tiles > 65535) return CB_ERR_UNSUPPORTED;
    // (single tokens of more than a tile of query heads keep ranks like a portion's)
    p.lead = lead > 0 && lead < n_requests && n_rep <= ROWS ? lead : 0;
    const int portions = n_requests - p.lead;
    p.lead_ranks = (p.lead + portions - 1) / portions;
    if (p.lead_ranks + q_tiles > 65535) return CB_ERR_UNSUPPORTED;
    const dim3 grid(n_kv_heads, portions, p.lead_ranks + q_tiles);
    const int form = gate == nullptr ? GATE_NONE : gate_per_head ? GATE_HEAD : GATE_RESULT;
    if (head_dim == 64) return launch_as<64>(form, grid, (cudaStream_t)stream, maps, p);
    if (head_dim == 256 && value_cols > 0 && value_cols <= 192 && form == GATE_NONE)
        return launch_gate<256, GATE_NONE, true>(grid, (cudaStream_t)stream, maps, p);
    if (head_dim == 256) return launch_as<256>(form, grid, (cudaStream_t)stream, maps, p);
    return launch_as<128>(form, grid, (cudaStream_t)stream, maps, p);
}
