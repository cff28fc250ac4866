// What the tcgen05 products (gemm_tcgen05.cu, gemm_waves_tcgen05.cu) are told beyond their operands.
#pragma once

namespace {

enum Epilogue { STORE_BF16 = 0, STORE_F32 = 1, ACCUM_F32 = 2, SWIGLU_BF16 = 3, ROPE_APPEND = 4 };

// What a product knows of the RMS norm on either side of it.
//   After it (ACCUM_F32 as the rows' last write before a norm): with `gain` set the epilogue
//   also leaves bf16(x * gain) of the summed rows x in `scaled` and the tile's share of every
//   row's sum of squares in `sumsq_out` [tiles along N][M] (summed in the order of the
//   columns).  The tile of C comes into shared memory by TMA while the products run, so the
//   thread that holds a row's accumulators also has the values they are added to; C itself
//   still gets its sums by TMA adds, `scaled` leaves by TMA stores of 32-column boxes (a single
//   tile of rows: in 64-byte pieces of the threads' own rows).
//   Tiles up to 128 columns, N a multiple of 32.
//   Before it (any epilogue): with `sumsq_in` set the rows of A are bf16(x * gain) of rows
//   not yet divided by their root mean square; the epilogue sums a row's `parts` shares in
//   their order and multiplies the row's accumulators by 1 / sqrt(sum / width + eps), which
//   is the same product as with normalised rows up to the rounding of A.
struct NormArgs {
    const float* gain;
    __nv_bfloat16* scaled;
    float* sumsq_out;
    int ld_scaled;
    const float* sumsq_in;
    int parts;
    float width, eps;
    // SWIGLU_BF16: limit > 0 makes the pair the capped one (tc::gated_pair), else silu(g) * u
    float glu_limit, glu_alpha, glu_offset;
    // A grouped product (form GROUPED): the rows of A lie expert by expert, W is the experts'
    // matrices one below the other (w_rows rows each), and block row y takes tile y of the plan
    // that a kernel before this one left on the device: [0] tiles in use, [2 + E + y] the tile's
    // expert, [2 + E + max_tiles + y] its first row, [2 + E + 2 max_tiles + y] its rows (at most
    // 128).  Tiles beyond those in use do nothing.
    const int* plan;
    int n_experts, max_tiles, w_rows;
    // A product per head in one launch (form PER_HEAD): block z takes head z, whose
    // columns of A start at z * head_a_cols, whose matrix is rows [z * w_rows, z * w_rows + N) of
    // W and whose results go to columns z * head_c_cols + [0, N) of C.  K is a head's K; what a
    // block of 64 columns of A holds beyond it meets columns of W outside its map, which read zero.
    // Two products of the same rows in one (form SPLIT_OUT, STORE_BF16; heads 0): the results of the first n_main rows of W (a
    // multiple of 64) go to C, those of the others to out2 in fp32 (ld2 floats between rows).  (A product of 8 to 32 columns alone
    // is a chain of K / 64 loads on few SMs, 7 to 16 us; here it mostly rides in the last column of tiles: the state-space
    // layer of width 2,048, 32 decoded tokens, 45 -> 38 us a step.)
    // These forms share their fields, as no product is both, for the size: see the assertion below.
    int heads, head_a_cols;
    union { int head_c_cols; int n_main; };
    // STORE_BF16: an activation on the way out; 0: none, 1: max(x, 0)^2.  PER_HEAD, with `gate` set (up to
    // GATED_ROWS rows): the results times the sigmoids of their logits before they are rounded, of one logit a row and head
    // (GATE_HEAD: fp32 [M][heads]) or of one a result (GATE_RESULT: bf16 [M][heads * N]).
    int act;
    union { const void* gate; void* out2; };
    union { int gate_ld; int ld2; };
};
// With 120 bytes the parameters of gemm_tcgen05_kernel are 768.  With 136 (and the kernel's code as it was) every
// gated product took 0.3 to 0.6 us more: 17 rows of 2 x 2,048 by 768 5.5 -> 5.8 us, 300 5.5 -> 5.85, 900 rows of
// 2 x 2,816 by 2,048 22.8 -> 23.5.
static_assert(sizeof(NormArgs) == 120, "the products' parameters have grown");

}  // namespace
