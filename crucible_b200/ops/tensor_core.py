"""The bfloat16 tensor-core kernels.  Each function returns True if it ran, or
False if the sizes are outside what the kernel takes, in which case the caller
runs the plain CUDA-core kernel instead.  The rule is stated here and depends
on the shapes and strides alone, never on the batch:

matrix products (tcgen05 + TMA): K, the row strides of both operands and the
row stride of a bfloat16 output must be multiples of 8 elements (TMA needs
16-byte row pitches), and the operand bases 16-byte aligned.
"""
from __future__ import annotations

import ctypes
import functools
import math

import torch

from . import LAUNCHES, TIMER, _stream, _tick, build

build.register_module("gemm_tcgen05", ["common.cuh", "tc_common.cuh", "gemm_args.cuh"])
build.register_module("gemm_waves_tcgen05", ["common.cuh", "tc_common.cuh", "gemm_args.cuh"])
build.register_module("attention_mma", ["common.cuh"])
build.register_module("gemm_skinny_tcgen05", ["common.cuh", "tc_common.cuh"])
build.register_module("attention_tcgen05", ["common.cuh", "tc_common.cuh"])
build.register_module("attention_decode_tcgen05", ["common.cuh", "tc_common.cuh"])
build.register_module("attention_short", ["common.cuh"])

# Portions of prompts with head size 64 run on the tcgen05 attention kernel; False sends
# them to the mma.sync kernel instead (the tests compare the two).
USE_TCGEN05_ATTENTION = True
USE_TCGEN05_DECODE = True

STORE_BF16, STORE_F32, ACCUM_F32, SWIGLU_BF16, ROPE_APPEND = 0, 1, 2, 3, 4
_UNSUPPORTED = 100001

_status = {}
FAILURES = [0]       # kernels that gave up so far; engines drop their captured steps when it moves


class KernelGaveUp(RuntimeError):
    """A tensor-core kernel ran out one of its bounded waits: the results of the step
    it belonged to are not valid."""


def status_word(device) -> torch.Tensor:
    """A device int the kernels write if one of their bounded waits runs out."""
    key = (device if isinstance(device, torch.device) else torch.device(device)).index or 0
    t = _status.get(key)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=device)
        _status[key] = t
    return t


def raise_if_gave_up(device, code: int) -> None:
    """`code` is a value of the status word that reached the host (read here, or relayed
    behind a step's chosen ids).  Non-zero: puts the device-side state back in order (the
    word to zero; the arrival counters of the split kernels, which a block that gave up
    leaves counted short) and raises."""
    if not code:
        return
    key = torch.device(device).index or 0
    torch.cuda.synchronize(device)
    t = _status.get(key)
    if t is not None:
        t.zero_()
    for (dev, name), buf in _buffers.items():
        if dev == key and name.endswith(".counters"):
            buf.zero_()
    FAILURES[0] += 1
    what = {1: "a TMA producer", 2: "an MMA issuer", 3: "an epilogue",
            4: "a wait made to run out on purpose"}.get(code, "a role")
    raise KernelGaveUp(f"a tensor-core kernel gave up: {what} waited past its limit "
                       f"(status {code}); the step's results are not valid")


def check_status(device) -> None:
    """Raises if a tensor-core kernel gave up a wait since the last check.
    Synchronises; call it where the host waits anyway."""
    key = torch.device(device).index or 0
    t = _status.get(key)
    if t is None:
        return
    raise_if_gave_up(device, int(t.item()))


def _count(n: int) -> None:
    LAUNCHES[0] += n
    if TIMER[0] is not None:
        import sys
        _tick("tensor cores: " + sys._getframe(1).f_code.co_name)


TILE_WIDTHS = (64, 96, 128, 160, 192, 256)
N_SMS = 148


def _tile_of(tile):
    """`tile` as callers may give it: a width, (width, blocks per SM), or
    (width, blocks per SM, shares of K)."""
    return (tile, 1) if isinstance(tile, int) else tuple(tile)


# Shares of K, measured on B200 at 33 to 512 rows: a block's chain costs about 0.32 us per
# block of 64 elements of K (0.43 us for tiles wider than 128 columns: the ring of stages
# in flight over the latency of a load, not the tile's bytes, sets it), a cluster costs
# about 2 us more than a lone block, and the first block of a cluster takes about 0.5 us
# to pull 32 KB of another block's sums.  Clusters of 3 and 4 need room to be placed inside
# one GPC, so they may not fill the SMs to the last one.
K_SPLIT_STEP_US = (0.32, 0.43)
K_SPLIT_CLUSTER_US = 2.0
K_SPLIT_PULL_US = 0.5
K_SPLIT_BLOCK_LIMIT = {2: 148, 3: 120, 4: 128}
K_SPLIT_MIN_GAIN_US = 1.0


@functools.lru_cache(maxsize=4096)
def k_splits(m: int, n_cols: int, k: int, bn: int) -> int:
    """Blocks that share one tile's K as a cluster (1: none).  A step of 33 to a few
    hundred rows has few tiles, each a chain of K / 64 loads and products on one SM while
    most SMs idle; shares of K spread the chain over the idle SMs."""
    tiles = -(-m // 128) * -(-n_cols // bn)
    k_blocks = -(-k // 64)
    step = K_SPLIT_STEP_US[1 if bn > 128 else 0]
    best, best_cost = 1, k_blocks * step - K_SPLIT_MIN_GAIN_US
    for s, limit in K_SPLIT_BLOCK_LIMIT.items():
        per = -(-k_blocks // s)
        if tiles * s > limit or (s - 1) * per >= k_blocks:
            continue
        cost = per * step + K_SPLIT_CLUSTER_US + K_SPLIT_PULL_US * (s - 1) * bn / 64
        if cost < best_cost:
            best, best_cost = s, cost
    return best


@functools.lru_cache(maxsize=4096)
def _tile_width(m: int, n_cols: int, epi: int = 1, multiple_of: int = 1):
    """Tile width in output columns: the one that needs the least time if every
    block costs (width + a fixed part) and blocks run in waves over the SMs.  A
    wide tile reuses the A tile more; a narrow one fills the last wave better.
    Widths whose output cannot leave through shared memory and TMA (bfloat16 rows
    that are no multiple of 128 bytes per tile) pay for their strided stores.  The fixed part, a
    block's start and end, weighs as much as 128 columns (of 140 products of 40 to 2,048 rows the choice
    is 2.4 % from the best width on average; with 48 it was 3.6 %: 2,048 x 5,632 x 2,048 with the gated
    pair 60 us in five waves of 128 columns, 44 in three of 256)."""
    m_tiles = -(-m // 128)
    best, best_cost = 64, None
    for bn in TILE_WIDTHS:
        if bn % multiple_of:
            continue
        blocks = m_tiles * -(-n_cols // bn)
        direct = 40 if epi == STORE_BF16 and bn % 64 else 20 if epi == SWIGLU_BF16 and bn % 128 else 0
        cost = -(-blocks // N_SMS) * (bn + 128 + direct)
        if best_cost is None or cost < best_cost or (cost == best_cost and bn > best):
            best, best_cost = bn, cost
    return best, 1


@functools.lru_cache(maxsize=4096)
def _tile_and_shares(m: int, n_cols: int, k: int, epi: int):
    """`_tile_width` for float32 results, with the shares of K where the narrowest tiles leave no room for two and
    wider ones do: a chain over a long K is longer than what a wider tile costs.  75 to 148 tiles of 64 columns ->
    two shares of 96 or 128, us: 330 x 2,048 by K = 4,096 / 5,632 / 8,192 13.3 / 17.2 / 24.9 -> 11.8 / 13.9 / 18.2 (96),
    512 rows 13.1 / 17.1 / 25.1 -> 13.0 / 15.9 / 21.4 (128), 640 x 1,024 by 4,096 13.2 -> 11.9 (96); at K = 3,072
    10.7 and 10.4, at 2,048 8.0 and 8.3.  Tiles wider than 128 columns leave the next norm's input to another launch."""
    bn, per_sm = _tile_width(m, n_cols, epi)
    if bn == 64 and epi != STORE_BF16 and k_splits(m, n_cols, k, bn) == 1:
        for wide, least in ((96, 3584), (128, 5120)):
            if k >= least and 2 * -(-m // 128) * -(-n_cols // wide) <= K_SPLIT_BLOCK_LIMIT[2]:
                return wide, 1, 2
    return bn, per_sm


TALL_MIN_ROWS = 1024        # two accumulators per block (256 x 256 of output) ...
TALL_MIN_K = 512            # ... pay where many rows meet enough 256 x 256 tiles to fill the SMs: at
TALL_MIN_FILL = 0.8         # long K they halve the operand bytes per flop, at short K the blocks' starts and ends


@functools.lru_cache(maxsize=4096)
def _tall_tiles(m: int, n_cols: int, k: int) -> bool:
    """Whether a product should run as 256 x 256 tiles (two accumulators per block).  At the
    Llama-3-8B layer sizes 148 blocks of 128 x 256 ask the L2 for 384 rows of operands per
    tile and run at half the tensor cores' rate; 256 x 256 needs 512 rows for twice the output."""
    if m < TALL_MIN_ROWS or k < TALL_MIN_K:
        return False
    blocks = -(-m // 256) * -(-n_cols // 256)
    waves = -(-blocks // N_SMS)
    return blocks / (waves * N_SMS) >= TALL_MIN_FILL


NORM_AHEAD = True    # the accumulate products may leave the next norm's input (tests switch it off)
NORM_AHEAD_MAX_TILE = 128   # widest tile whose epilogue holds a row's sums in registers


class _NormArgs(ctypes.Structure):
    """`NormArgs` of csrc/gemm_args.cuh."""
    _fields_ = [("gain", ctypes.c_void_p), ("scaled", ctypes.c_void_p), ("sumsq_out", ctypes.c_void_p),
                ("ld_scaled", ctypes.c_int), ("sumsq_in", ctypes.c_void_p), ("parts", ctypes.c_int),
                ("width", ctypes.c_float), ("eps", ctypes.c_float),
                ("glu_limit", ctypes.c_float), ("glu_alpha", ctypes.c_float), ("glu_offset", ctypes.c_float),
                ("plan", ctypes.c_void_p), ("n_experts", ctypes.c_int), ("max_tiles", ctypes.c_int),
                ("w_rows", ctypes.c_int), ("heads", ctypes.c_int), ("head_a_cols", ctypes.c_int),
                ("head_c_cols", ctypes.c_int), ("act", ctypes.c_int), ("gate", ctypes.c_void_p),
                ("gate_ld", ctypes.c_int)]


class NormEmit:
    """What an accumulate product is asked to leave for the RMS norm that reads its output
    rows next: `scaled` bf16 [rows, width] = bf16(x * gain), `sumsq` fp32 [parts, rows] = the
    tiles' shares of every row's sum of squares.  `parts` is set by the product that did it
    (None: it did not, the norm runs as a kernel of its own)."""

    def __init__(self, gain: torch.Tensor, scaled: torch.Tensor, sumsq: torch.Tensor, norm=None):
        self.gain, self.scaled, self.sumsq = gain, scaled, sumsq
        self.norm = norm              # the part the rows are left for (the caller's own reference)
        self.parts = None


def _norm_args(emit, pre, rows: int, pair=None, act: int = 0):
    """The pointer the product kernels take, and the object that keeps it alive.  `pair`:
    (limit, alpha, offset) of the capped gated pair for the SwiGLU form.  `act`: an activation
    on a bfloat16 result's way out (1: the square of relu)."""
    if emit is None and pre is None and pair is None and not act:
        return 0, None
    args = _NormArgs()
    args.act = int(act)
    if pair is not None:
        args.glu_limit, args.glu_alpha, args.glu_offset = (float(v) for v in pair)
    if emit is not None:
        args.gain, args.scaled = emit.gain.data_ptr(), emit.scaled.data_ptr()
        args.sumsq_out, args.ld_scaled = emit.sumsq.data_ptr(), emit.scaled.stride(0)
    if pre is not None:
        if pre.sumsq.stride(0) != rows or pre.sumsq.dtype != torch.float32:
            raise RuntimeError("shares of the rows' sums of squares must be float32 [parts, rows]")
        args.sumsq_in, args.parts = pre.sumsq.data_ptr(), pre.parts
        args.width, args.eps = float(pre.x.shape[1]), float(pre.eps)
    return ctypes.addressof(args), args


def _gemm(a, w, out, n, epi, bn, per_sm=1, splits=None, emit=None, pre=None, pair=None, act=0) -> bool:
    lib = build.load("gemm_tcgen05")
    if per_sm == 0:
        # 256 x 256 tiles; an output that cannot leave by TMA is refused, and the 128-row tiles run
        if _gemm(a, w, out, n, epi, 256, -1, 1, None, pre, pair, act):
            return True
        per_sm = 1
    if per_sm == -1:
        per_sm, splits = 0, 1
    m, k = a.shape
    if splits is None:
        splits = k_splits(m, 2 * n if epi == SWIGLU_BF16 else n, k, bn)
    if emit is not None and (epi != ACCUM_F32 or bn > NORM_AHEAD_MAX_TILE or per_sm == 0 or n % 32
                             or emit.sumsq.shape[0] < -(-n // bn) or emit.sumsq.stride(0) != a.shape[0]):
        emit = None
    norm_ptr, keep = _norm_args(emit, pre, m, pair, act)
    code = lib.cb_gemm_tcgen05(
        a.data_ptr(), w.data_ptr(), out.data_ptr(),
        m, n, k, a.stride(0),
        w.stride(0), out.stride(0), epi, bn, per_sm,
        splits, status_word(a.device).data_ptr(), _stream(), norm_ptr)
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core matrix product failed to launch (CUDA error {code})")
    if emit is not None:
        emit.parts = -(-n // bn)
    _count(1)
    return True


WAVES_MIN_TILES = 200       # tiles of 128 x 256 from which one block an SM walks them (`_gemm_waves`)
F32_WAVES_MIN_TILES = 210   # ... for float32 results by a long K
TALL_COST = 711             # a wave of tall tiles, where a wave of tiles of bn columns costs bn + 128


@functools.lru_cache(maxsize=4096)
def _waves_width(m: int, n_cols: int, k: int, epi: int) -> int:
    """The tile width with which a product runs through `_gemm_waves`, 0: not at all.  That kernel hides every
    tile's way out behind the next tile's products, but has fewer stages, a longer start, and no second
    accumulator row for tall tiles.  us at 2,048 rows, 128-row tiles or tall ones -> waves: the gated pair of
    2 x 2,048 by K = 768 15.8 -> 13.3, of 2 x 2,816 by 2,048 43.2 -> 35.3; float32 results of 4,096
    by 128 10.2 -> 8.6, of 50,304 by 768 204 -> 160.  From 1.35 waves on: at 1,100 rows of
    2 x 2,816 (198 tiles) 23.7 -> 24.4.  bfloat16 results gain 3 to 7 % at the width that a block a tile would
    have: with 256 columns from two waves on (8,192 by 2,048 at 1,100 / 1,600 rows 28.2 / 43.0 -> 26.4 / 39.9),
    with 192 from three on or at a short K (2,048 rows of 5,120 by 2,048 34.0 -> 32.9, of 3,072 by 1,024 14.6 ->
    13.6; two waves by 2,048, 1,100 rows of 4,608, 21.5 -> 21.9), and beyond K = 2,048 from four (by 4,096, 1,600 rows of
    6,144 64.6 -> 67.7, 1,800 79.5 -> 75.0).
    float32 results of more than 128 rows by a K of more than 1,024 want 1.4 waves (1,300 rows of 4,096 by 2,048, 1.2 waves,
    23.2 -> 24.4, by 4,096 37.8 -> 43.3), and from K = 1,024 on stay with one to three waves of tall tiles unless that many
    waves here cost clearly less (2,048 rows of 4,096 by 2,048 27.1 -> 27.9, of 8,192 56.4 -> 62.8; 1,100 of 6,144 28.2 -> 24.5,
    1,300 of 16,384 91.0 -> 76.9)."""
    m_tiles = -(-m // 128)
    waves = lambda bn: -(-m_tiles * -(-n_cols // bn) // N_SMS)
    if epi == STORE_F32 and waves(256) > 1:
        if k > 1024 and m_tiles > 1 and m_tiles * -(-n_cols // 256) < F32_WAVES_MIN_TILES:
            return 0
        cost, bn = min((waves(bn) * (bn + 64), bn) for bn in (192, 256))
        if k >= 1024 and _tall_tiles(m, n_cols, k):
            tall = -(--(-m // 256) * -(-n_cols // 256) // N_SMS)
            if tall <= 3 and cost > 0.83 * tall * TALL_COST:
                return 0
        return bn
    if epi == SWIGLU_BF16:
        return 256 if m_tiles * -(-n_cols // 256) >= WAVES_MIN_TILES else 0
    if epi == STORE_BF16:
        bn = _tile_width(m, n_cols, epi)[0]
        least = {256: 2, 192: 2 if k <= 1024 else 3 if k <= 2048 else 4}.get(bn)
        return bn if least is not None and waves(bn) >= least else 0
    return 0


def _gemm_waves(a, w, out, n, epi, bn, pre=None, pair=None, act=0, plan=None) -> bool:
    """The product with one block an SM over the tiles (`csrc/gemm_waves_tcgen05.cu`).  `plan`: the arguments of
    a grouped product.  False: sizes it does not take."""
    norm_ptr, keep = _norm_args(None, pre, a.shape[0], pair, act)
    if plan is not None:
        keep, norm_ptr = plan, ctypes.addressof(plan)
    code = build.load("gemm_waves_tcgen05").cb_gemm_waves(
        a.data_ptr(), w.data_ptr(), out.data_ptr(),
        a.shape[0], n, a.shape[1], a.stride(0), w.stride(-2),
        out.stride(0), epi, bn, status_word(a.device).data_ptr(), _stream(), norm_ptr)
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core product in waves failed to launch (CUDA error {code})")
    _count(1)
    return True


_buffers = {}        # (device, name) -> tensor; grown by doubling, old ones kept alive because
_retired = []        # captured CUDA graphs may still hold their addresses


def _buffer(device, name: str, numel: int, dtype, zero: bool = False) -> torch.Tensor:
    key = (torch.device(device).index or 0, name)
    t = _buffers.get(key)
    if t is None or t.numel() < numel:
        if t is not None:
            _retired.append(t)
        make = torch.zeros if zero else torch.empty
        t = make(max(2 * numel, 1024), dtype=dtype, device=device)
        _buffers[key] = t
    return t


def skinny_splits(m: int, n_tiles: int, k: int) -> int:
    """Blocks along K per 128-row tile of W: as many as give every SM one block, never more
    blocks than SMs (a launch of at most one block per SM runs with eight stages, and every
    further split is a partial tile more for the last block to sum: 50 MB at 8 rows 13.7 us with
    3 x 48 blocks, 15.9 us with 4 x 48), and never so many that the partial tiles outweigh the
    weights they stand for."""
    k_blocks = -(-k // 64)
    want = max(1, N_SMS // n_tiles)
    cap = max(1, k // (4 * m))
    return max(1, min(want, k_blocks, cap))


def _gemm_skinny(a, w, out, n, epi, splits=None) -> bool:
    lib = build.load("gemm_skinny_tcgen05")
    m, k = a.shape
    n_tiles = int(lib.cb_gemm_skinny_tiles(n, epi))
    if splits is None:
        splits = skinny_splits(m, n_tiles, k)
    partial = counters = None
    if splits > 1:
        nbytes = int(lib.cb_gemm_skinny_partial_bytes(m, n, epi,
                                                      splits))
        partial = _buffer(a.device, "skinny.partial", nbytes // 4, torch.float32)
        counters = _buffer(a.device, "skinny.counters", n_tiles, torch.int32, zero=True)
    code = lib.cb_gemm_skinny(
        a.data_ptr(), w.data_ptr(), out.data_ptr(),
        m, n, k, a.stride(0), w.stride(0),
        out.stride(0), epi, splits,
        partial.data_ptr() if partial is not None else 0,
        counters.data_ptr() if counters is not None else 0,
        status_word(a.device).data_ptr(), _stream())
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core matrix product failed to launch (CUDA error {code})")
    _count(1)
    return True


SKINNY_ROWS = 16     # products with at most this many rows run with W on the MMA's M side ...
SKINNY_MIN_BYTES = 40 << 20   # ... if W is at least this large (it streams: 3.6-5.5 TB/s; smaller
                              # ones are latency-bound: at 33 MB and 16 rows the 128-row tiles, with
                              # K shared by clusters, take 12.7 us, these 12.4, the few-row kernel 12.1
                              # at 8 rows).
SKINNY_MID_ROWS = 32          # ... and up to this many rows between that size and SKINNY_MID_BYTES
SKINNY_MID_BYTES = 128 << 20  # (50 MB at 32 rows: 16.2 against 17.6 us for the tiles, 117 MB: 29.2
                              # against 33.3; 235 MB: 46.8 against 44.4).  From 33 rows on the
                              # 128-row tiles are as fast or faster at every size.
SKINNY_WIDE_N = 8192 # ... and up to 64 rows if W has at least this many rows (the LM head)


def _operands_ok(a, w) -> bool:
    (a_row, a_col), (w_row, w_col) = a.stride(), w.stride()
    return (a_col == 1 and w_col == 1 and not (a.shape[1] | a_row | w_row) & 7 and not (a.data_ptr() | w.data_ptr()) & 15
            and a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and a.is_cuda)


def linear(a, w, out, *, accumulate=False, tile=None, emit=None, pre=None, act=0) -> bool:
    """`emit` (`NormEmit`): with accumulate, also leave the next norm's input if this product's
    form can (`emit.parts` says whether it did).  `pre` (`small_batch.LazyNorm` with `scaled`):
    `a` is that norm input, the rows' factors are applied in the epilogue.  `act` 1 (a bfloat16
    result through the 128-row tiles): the square of relu in the epilogue."""
    if not _operands_ok(a, w) or out.stride(1) != 1:
        return False
    if act and out.dtype != torch.bfloat16:
        return False
    if out.dtype == torch.bfloat16:
        if accumulate:
            return False
        epi = STORE_BF16
    elif out.dtype == torch.float32:
        epi = ACCUM_F32 if accumulate else STORE_F32
    else:
        return False
    m, k = a.shape
    n = w.shape[0]
    if tile is None and m <= 64:
        w_bytes = w.numel() * 2
        if ((m <= SKINNY_ROWS and w_bytes >= SKINNY_MIN_BYTES)
                or (m <= SKINNY_MID_ROWS and SKINNY_MIN_BYTES <= w_bytes <= SKINNY_MID_BYTES) or n >= SKINNY_WIDE_N):
            if pre is not None or act:
                return False
            return _gemm_skinny(a, w, out, n, epi)
    if tile is None:
        tall = _tall_tiles(m, n, k)
        waves = 0 if emit is not None or pre is not None or (tall and epi != STORE_F32) else _waves_width(m, n, k, epi)
        if waves and _gemm_waves(a, w, out, n, epi, waves, act=act):
            return True
        tile = (256, 0) if tall else None
    bn, per_sm, *splits = _tile_of(tile) if tile else _tile_and_shares(m, n, k, epi)
    return _gemm(a, w, out, n, epi, bn, per_sm, splits[0] if splits else None, emit, pre, None, act)


def _product_cost(m: int, n_cols: int, k: int):
    """The cost by which `_tile_width` chooses, of its choice or of tall tiles, and the tile."""
    if _tall_tiles(m, n_cols, k):
        return -(--(-m // 256) * -(-n_cols // 256) // N_SMS) * TALL_COST, (256, 0)
    bn, per_sm = _tile_width(m, n_cols, STORE_BF16, 64)
    return -(--(-m // 128) * -(-n_cols // bn) // N_SMS) * (bn + 128), (bn, per_sm)


@functools.lru_cache(maxsize=4096)
def _split_tile(m: int, n_main: int, n_second: int, k: int):
    """The tile of two products of the same rows in one launch, or None where apart they take less: the second
    often fits into the first's last column of tiles or an SM that its wave leaves idle (2,048 rows of 5,120 +
    32 columns by 2,048: 34.0 and 8.7 us apart), but where it opens a wave more that costs more than a launch
    (4,608 + 16: tall tiles of the first take 25.2)."""
    joint, tile = _product_cost(m, n_main + n_second, k)
    return tile if joint <= _product_cost(m, n_main, k)[0] + _product_cost(m, n_second, k)[0] else None


def linear_split(a, w, out, out2) -> bool:
    """[out | out2] = a . w^T for bfloat16 rows `out` of a multiple of 64 columns and float32 rows `out2`, in one
    launch.  False: not taken."""
    m, k = a.shape
    n, n_main = w.shape[0], out.shape[1]
    if (not _operands_ok(a, w) or out.dtype != torch.bfloat16 or out2.dtype != torch.float32 or n_main % 64
            or out.stride(1) != 1 or out2.stride(1) != 1 or out2.shape[1] != n - n_main or out2.stride(0) % 4
            or out.stride(0) % 8 or (out.data_ptr() | out2.data_ptr()) & 15):
        return False
    if m <= 64 and ((m <= SKINNY_MID_ROWS and w.numel() * 2 >= SKINNY_MIN_BYTES) or n >= SKINNY_WIDE_N):
        return False                              # (the few-row kernel's)
    tile = _split_tile(m, n_main, n - n_main, k)
    if tile is None:
        return False
    args = _NormArgs()
    args.gate, args.head_c_cols, args.gate_ld = out2.data_ptr(), n_main, out2.stride(0)      # (out2, n_main, ld2 there)
    bn, per_sm = tile
    code = build.load("gemm_tcgen05").cb_gemm_tcgen05(
        a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, a.stride(0), w.stride(0), out.stride(0), STORE_BF16, bn, per_sm,
        1 if per_sm == 0 else k_splits(m, n, k, bn), status_word(a.device).data_ptr(), _stream(), ctypes.addressof(args))
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core product with two results failed to launch (CUDA error {code})")
    _count(1)
    return True


@functools.lru_cache(maxsize=4096)
def grouped_tile(pairs: int, n_experts: int, n_cols: int, gated: bool):
    """(tile width, blocks to an SM) of a grouped product over `n_cols` rows of an expert's matrix.  Blocks
    run in waves over the SMs and a block costs its width and a fixed part of 160 columns, which here
    is mostly the operands' way in.  Tiles of 128 rows: one an expert while few experts have more rows than
    that, then a half-filled one each beside the full ones.  Over 16 to 4,096 pairs of 8 experts of 2,816 x 2,048
    and 1,408 x 1,024 the choice is 0.5 % from the best width on average, 14 % at worst; 128 columns
    throughout 16 %, 67 % at worst (4,096 pairs, gate/up of 2,816: 106 us with 256 columns, 150 with
    128; 512 pairs: gate/up 36 with 192 and 42 with 128, down 17.5 with 128 and 23.8 with 256).
    A couple of pairs an expert: not all experts have rows, and with two blocks to an SM all blocks of
    the wide gate/up find a place at once (16 pairs: 24.7 us, 31.2 with 192 columns)."""
    if gated and pairs < 3 * n_experts:
        return 128, 2
    tiles = n_experts if pairs <= 112 * n_experts else pairs / 128 + n_experts / 2
    return min((-(-int(math.ceil(tiles * -(-n_cols // bn))) // N_SMS) * (bn + 160), bn) for bn in (128, 192, 256))[1], 1


def grouped_waves(pairs: int, n_experts: int, n_cols: int) -> bool:
    """Whether a grouped product over `n_cols` rows of an expert's matrix goes by `_gemm_waves`: full tiles beside a
    half-filled one an expert (4,096 pairs of 8 experts of 2,816 x 2,048 gate/up 99.8 -> 90.6 us, down 53.8 -> 49.2;
    2,048 pairs 56.6 -> 53.8 and, below the line, 39.0 -> 45.7)."""
    return (pairs / 128 + n_experts / 2) * -(-n_cols // 256) >= WAVES_MIN_TILES and pairs >= 64 * n_experts


def tiles_by_chance(pairs: int, n_experts: int) -> float:
    """The tiles of 128 rows that `pairs` rows fill if every expert has each of them with the same chance: the experts, times
    the mean of the whole tiles of a number of rows that is about normal."""
    mean = pairs / n_experts
    return n_experts * sum(0.5 * math.erfc((128 * j + 0.5 - mean) / math.sqrt(2 * mean))
                           for j in range(int((mean + 4 * math.sqrt(mean)) / 128) + 1))


def _grouped_cost(pairs: int, n_experts: int, tiles: float, n_cols: int, gated: bool) -> int:
    """What a grouped product over `tiles` tiles costs in the unit of `_tile_width`: its waves, each the tile's
    width and a fixed part, less of it where a block takes several tiles and hides a tile's end behind the next."""
    bn, fixed = (256, 64) if grouped_waves(pairs, n_experts, n_cols) else (grouped_tile(pairs, n_experts, n_cols, gated)[0], 112)
    return -(-math.ceil(tiles * -(-n_cols // bn)) // N_SMS) * (bn + fixed)


def _dense_cost(m: int, n_cols: int, k: int, epi: int) -> int:
    bn = _waves_width(m, n_cols, k, epi)
    return -(--(-m // 128) * -(-n_cols // bn) // N_SMS) * (bn + 64) if bn else _product_cost(m, n_cols, k)[0]


@functools.lru_cache(maxsize=4096)
def riding_pays(rows: int, width: int, ff: int, n_experts: int, top: int) -> bool:
    """Whether one more expert of the same size that all `rows` rows choose goes with the grouped products of the
    others, `top` of `n_experts` a row, instead of by two products of its own: by the waves that the four products
    take and the two would.  Its rows fill tiles of their own, which may cost a wave more than the dense products do.
    Riding saves two launches (100,000 of the unit times K).  16 sizes (4 to 64 experts of 512 x 768 to 4,096 x 1,536, top 1
    to 8) at 136 to 4,096 rows, 512 measured both replayed and eagerly, against apart: where the reckoned cost is 7 % less,
    0.955 and 0.936 on average, 10 of them more than 1.5 % slower (3.9 % at worst).  Riding
    always is 0.958 and 0.937, 13 % slower at worst, by two limits on the rows as before 0.965 and 0.946.  us apart and
    riding: 8 of 2,048 x 2,816, top 2, 320 rows 100 and 100, 600 135 and 121, 2,048 223 and 217, 4,096 381 and 394; 32 of
    2,048 x 1,408, top 4, 450 rows 150 and 134; 8 of 4,096 x 1,536, top 1, 384 rows 107 and 121.  Of 5,000 to 8,192 rows
    neither is ahead (the mean of 18: 0.2 % behind)."""
    if rows > 4096:
        return False
    pairs = rows * top
    tiles = tiles_by_chance(pairs, n_experts)
    more = tiles + -(-rows // 128)
    apart = (width * (_grouped_cost(pairs, n_experts, tiles, 2 * ff, True) + _dense_cost(rows, 2 * ff, width, SWIGLU_BF16))
             + ff * (_grouped_cost(pairs, n_experts, tiles, width, False) + _dense_cost(rows, width, ff, ACCUM_F32)))
    riding = (width * _grouped_cost(pairs + rows, n_experts + 1, more, 2 * ff, True)
              + ff * _grouped_cost(pairs + rows, n_experts + 1, more, width, False))
    return riding <= 0.93 * (apart + 100_000)


def grouped_linear(a, w, out, plan, n_experts: int, tiles: int, gated: bool, pair=None, tile=None) -> bool:
    """The grouped product of a mixture of experts (`cb_gemm_tcgen05_grouped`): `a` [pairs, K]
    bfloat16 rows expert by expert, `w` [experts, rows, K] a declared weight, `plan` the int32
    plan on the device with `tiles` tile entries of 128 rows.  gated: out [pairs, rows / 2]
    bfloat16 with the gated pair; else out float32 or bfloat16 [pairs, rows]."""
    if (a.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or w.dim() != 3 or not w.is_contiguous()
            or a.stride(1) != 1 or out.stride(1) != 1 or a.shape[1] != w.shape[2]):
        return False
    if gated and out.dtype != torch.bfloat16:
        return False
    epi = SWIGLU_BF16 if gated else (STORE_F32 if out.dtype == torch.float32 else STORE_BF16)
    n = w.shape[1] // 2 if gated else w.shape[1]
    args = _NormArgs()
    if pair is not None:
        args.glu_limit, args.glu_alpha, args.glu_offset = (float(v) for v in pair)
    args.plan, args.n_experts, args.max_tiles, args.w_rows = plan.data_ptr(), n_experts, tiles, w.shape[1]
    if (tile is None and grouped_waves(a.shape[0], n_experts, w.shape[1]) and _gemm_waves(a, w, out, n, epi, 256, plan=args)):
        return True
    bn, per_sm = tile or grouped_tile(a.shape[0], n_experts, w.shape[1], gated)
    lib = build.load("gemm_tcgen05")
    code = lib.cb_gemm_tcgen05_grouped(
        a.data_ptr(), w.data_ptr(), out.data_ptr(),
        a.shape[0], n, a.shape[1], a.stride(0), w.stride(1),
        out.stride(0), epi, bn, per_sm, status_word(a.device).data_ptr(),
        _stream(), ctypes.addressof(args))
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"grouped tensor-core product failed to launch (CUDA error {code})")
    _count(1)
    return True




GATE_HEAD, GATE_RESULT = 2, 3


def heads_linear(a, a_head: int, w, out, out_head: int, gate=None) -> bool:
    """out[t, h * out_head + n] = sum_k a[t, h * a_head + k] * w[h, n, k] for every head of `w`
    [heads, N, K] (a declared bfloat16 weight) in ONE launch (`cb_gemm_tcgen05_heads`: the head is
    the grid's third axis).  `gate` (bfloat16 results of up to 16 rows alone): float32 logits [rows, heads] or bfloat16 ones
    [rows, heads * N] whose sigmoids the results are multiplied by before they are rounded.  Refuses
    what the tiles cannot take (the caller then runs a product per head)."""
    heads, n, k = w.shape
    if (a.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or not w.is_contiguous() or not a.is_cuda
            or a.stride(1) != 1 or out.stride(1) != 1 or out.dtype not in (torch.bfloat16, torch.float32)
            or k % 8 or a_head % 8 or a.stride(0) % 8
            or a.data_ptr() % 16 or w.data_ptr() % 16 or out.data_ptr() % 16
            or (out_head * out.element_size()) % 16 or (out.stride(0) * out.element_size()) % 16
            or a.shape[1] < (heads - 1) * a_head + k or out.shape[1] < (heads - 1) * out_head + n):
        return False
    epi = STORE_F32 if out.dtype == torch.float32 else STORE_BF16
    bn = 128 if n > 96 else (96 if n > 64 else 64)
    lib = build.load("gemm_tcgen05")
    code = lib.cb_gemm_tcgen05_heads(
        a.data_ptr(), w.data_ptr(), out.data_ptr(), a.shape[0],
        n, k, a.shape[1], a.stride(0), w.stride(1),
        out.stride(0), heads, a_head, out_head, epi, bn,
        gate.data_ptr() if gate is not None else 0, gate.stride(0) if gate is not None else 0,
        GATE_HEAD if gate is not None and gate.dtype == torch.float32 else GATE_RESULT,
        status_word(a.device).data_ptr(), _stream())
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core product per head failed to launch (CUDA error {code})")
    _count(1)
    return True


def linear_swiglu(h, gate_up, out, tile=None, pre=None, pair=None) -> bool:
    """`pair`: (limit, alpha, offset): the capped gated pair instead of silu(g) * u."""
    if not _operands_ok(h, gate_up) or out.dtype != torch.bfloat16 or out.stride(1) != 1:
        return False
    inter = gate_up.shape[0] // 2
    if tile is None and h.shape[0] <= SKINNY_ROWS and gate_up.numel() * 2 >= SKINNY_MIN_BYTES:
        if pre is not None or pair is not None:      # (the few-row split product has the silu pair only)
            return False
        return _gemm_skinny(h, gate_up, out, inter, SWIGLU_BF16)
    if tile is None:
        waves = _waves_width(h.shape[0], 2 * inter, h.shape[1], SWIGLU_BF16)
        if waves and _gemm_waves(h, gate_up, out, inter, SWIGLU_BF16, waves, pre, pair):
            return True
        tile = (256, 0) if _tall_tiles(h.shape[0], 2 * inter, h.shape[1]) else None
    bn, per_sm, *splits = _tile_of(tile) if tile else _tile_width(h.shape[0], 2 * inter, SWIGLU_BF16)
    return _gemm(h, gate_up, out, inter, SWIGLU_BF16, bn, per_sm, splits[0] if splits else None, None, pre, pair)


ROPE_TALL = None     # tests may fix the form of the q/k/v product (True: 256 x 256 tiles)


def linear_rope_append(h, wqkv, qkv, n_heads, n_kv_heads, head_dim, cos, sin, rotary_dim, ctx, cache,
                       binding, pre=None) -> bool:
    """The q/k/v projection with the rotation and the cache write in the product's
    epilogue (whole head rotated, head size a multiple of 64).  Rotated q lands in the
    first columns of `qkv`; k and v only in the cache.  False: not taken."""
    if (not _operands_ok(h, wqkv) or qkv.dtype != torch.bfloat16 or qkv.stride(1) != 1
            or cos is None or rotary_dim != head_dim or head_dim % 64 or head_dim > 256
            or h.shape[0] <= SKINNY_ROWS):
        return False
    k_cache, v_cache = cache.keys(binding.slot), cache.values(binding.slot)
    if k_cache.dtype != torch.bfloat16:
        return False
    table = ctx.block_table(binding.group)
    bn, _ = _tile_width(h.shape[0], wqkv.shape[0], ROPE_APPEND, multiple_of=head_dim)
    tall = 256 % head_dim == 0 and _tall_tiles(h.shape[0], wqkv.shape[0], h.shape[1])
    if ROPE_TALL is not None:
        tall = ROPE_TALL
    if tall:
        bn = 256
    if bn % head_dim:
        return False
    lib = build.load("gemm_tcgen05")
    norm_ptr, keep = _norm_args(None, pre, h.shape[0])
    code = lib.cb_gemm_tcgen05_rope(
        h.data_ptr(), wqkv.data_ptr(), qkv.data_ptr(),
        h.shape[0], h.shape[1], h.stride(0), wqkv.stride(0),
        qkv.stride(0), bn, cos.data_ptr(), sin.data_ptr(),
        ctx.positions.data_ptr(), ctx.row_request.data_ptr(),
        table.data_ptr(), table.shape[1], k_cache.data_ptr(),
        v_cache.data_ptr(), n_heads, n_kv_heads, head_dim,
        cache.page_tokens, 1 if binding.write else 0,
        1 if tall else k_splits(h.shape[0], wqkv.shape[0], h.shape[1], bn), 1 if tall else 0,
        status_word(h.device).data_ptr(), _stream(), norm_ptr)
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core q/k/v product failed to launch (CUDA error {code})")
    _count(1)
    return True


class _Requests:
    """A run of consecutive requests of the step, as the attention kernels see one:
    the metadata arrays from its first request on, how many there are, the most new
    tokens any of them brings, the context bucket that covers them, and the number of
    the step's rows up to its end (the split form's scratch is indexed by row)."""

    def __init__(self, ctx, table, first: int, count: int, max_new: int, bucket: int, rows_end: int, reach=None):
        self.row_start = ctx.req_row_start.data_ptr() + 4 * first         # (addresses of int32)
        self.first_pos = ctx.req_first_pos.data_ptr() + 4 * first
        self.table_stride = table.shape[1]
        self.table = table.data_ptr() + 4 * first * table.stride(0)
        self.first, self.whole_table = first, table
        self.count, self.max_new, self.bucket, self.rows_end = count, max_new, bucket, rows_end
        self.reach = bucket if reach is None else reach


def _tcgen05_rows(head_dim, k_cache, v_cache) -> bool:
    """Head sizes the tcgen05 prompt attention takes: 64 and 128, and 256 where a cached row is key and
    value at once."""
    return head_dim in (64, 128) or (head_dim == 256 and k_cache.data_ptr() == v_cache.data_ptr())


def _attention_tcgen05(qkv, out, k_cache, v_cache, reqs, n_heads, n_kv_heads, head_dim, scale,
                       window, cache, keep_first: int = 0, chunked: bool = False, sinks=None, out_scale: float = 1.0,
                       gate=None, gate_per_head: bool = False, lead: int = 0, value_cols=None) -> bool:
    """tcgen05 attention for portions of prompts: head sizes of `_tcgen05_rows`, page size a
    power of two from 8 to 128.  `keep_first` (with a window): keys before that position stay
    visible.  `chunked`: the window is a chunk's size.  `sinks`: float32 per query head or None.
    `gate`: rows laid out like `out` (`gate_per_head`: one logit a head) whose sigmoids the results are
    multiplied by before they are rounded, or None.  `lead`: how many requests at the head of `reqs` bring a
    single token.  `value_cols`: the features of a result that are read (None: all).  Returns False for anything else."""
    pt = cache.page_tokens
    if pt < 8 or pt > 128 or pt & (pt - 1):
        return False
    lib = build.load("attention_tcgen05")
    code = lib.cb_attention_tcgen05_kept(
        qkv.data_ptr(), qkv.stride(0), qkv.shape[0], out.data_ptr(),
        out.stride(0), k_cache.data_ptr(), v_cache.data_ptr(),
        k_cache.shape[0], reqs.row_start,
        reqs.first_pos, reqs.table,
        reqs.table_stride, reqs.count, reqs.max_new,
        n_heads, n_kv_heads, head_dim, pt,
        scale, window or 0, 1 if chunked else 0, keep_first if window else 0,
        out_scale, sinks.data_ptr() if sinks is not None else 0,
        gate.data_ptr() if gate is not None else 0, gate.stride(0) if gate is not None else 0,
        1 if gate_per_head else 0, lead, value_cols or 0, status_word(qkv.device).data_ptr(), _stream())
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tcgen05 attention failed to launch (CUDA error {code})")
    _count(1)
    return True


def _attention_decode_tcgen05(qkv, out, k_cache, v_cache, reqs, n_heads, n_kv_heads, head_dim,
                              scale, window, cache, partial, counters, n_chunks,
                              chunk_keys) -> bool:
    """tcgen05 attention for decoded tokens (at most 16 packed rows per request and
    KV head): head size 64 or 128, page size a power of two from 8 to 128.  Returns False
    for anything else."""
    pt = cache.page_tokens
    if pt < 8 or pt > 128 or pt & (pt - 1):
        return False
    lib = build.load("attention_decode_tcgen05")
    code = lib.cb_attention_decode_tcgen05(
        qkv.data_ptr(), qkv.stride(0), out.data_ptr(),
        out.stride(0), k_cache.data_ptr(), v_cache.data_ptr(),
        k_cache.shape[0], reqs.row_start,
        reqs.first_pos, reqs.table,
        reqs.table_stride, reqs.count, reqs.max_new,
        n_heads, n_kv_heads, head_dim, pt,
        scale, window or 0, partial.data_ptr(),
        counters.data_ptr(), n_chunks, chunk_keys,
        status_word(qkv.device).data_ptr(), _stream())
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tcgen05 decode attention failed to launch (CUDA error {code})")
    _count(1)
    return True


SHORT_ATTENTION = True       # tests switch it off to reach the split kernels with the same inputs


# A sink or a gate, by (features of a head, whether more than four query heads share a key/value head): the blocks from
# which contexts of up to so many keys go by one block each.
SHORT_SINK_BLOCKS = {(64, False): ((1024, 0), (1536, 32), (2048, 48), (3840, 64), (8192, 80)),
                     (64, True): ((512, 0), (768, 24), (1024, 64), (2048, 96)),
                     (128, False): ((1024, 0), (2048, 48), (8192, 80)),
                     (128, True): ((256, 0), (512, 32), (768, 64), (1536, 96))}


def short_attention_pays(blocks: int, reach: int, head_dim: int, plain: bool, heads_a_group: int = 1, tokens: int = 1) -> bool:
    """Whether single tokens that read up to `reach` keys (the longest context's class, or the window) take one block a
    request and key/value head (`blocks` of them) instead of keys split over blocks.  Without splitting
    nothing is merged, but a block walks its keys alone: 1.7 us a 256 keys of 64 features and 2.9 of 128, with more
    than four heads a group 2.6 and 4.8.  `reach` is the longest of the step, so every line was measured with
    all contexts as long and with one so long among others of 200 keys, and lies where both are as fast or faster.

    `plain`: against the tcgen05 kernel, which has nothing to merge up to 128 keys.  us, split and short: a pass of a prompt and
    eight steps of the 120M shape (12 heads of 64, 4 key/value heads), 4 tokens, behind 100 keys 2,355 and 2,432, behind 180
    2,610 and 2,497; 16 behind 40 3,046 and 3,120, 17 3,727 and 3,718; 32 (128 blocks) behind 180 4,504 and 4,323, 48 (192) 4,809 and
    4,820; whole layers of 16 heads of 128 and 4 key/value heads: 1 token behind 100 keys 33.4 and 31.6, 250 keys 36.7
    and 31.8, 400 keys 4 tokens 37.3 and 38.2, 16 (64 blocks) 52.9 and 48.1, 1,000 keys 24 tokens (96) 73.8 and 72.4, 48
    (192) 89.8 and 90.0; eight heads a group, 4 tokens behind 250 keys 39.6 and 38.2, 400 40.0 and 43.3.
    Else against the mma.sync kernel, whose launch and merge cost more: 8 tokens of 128 behind 240 keys 30.9 and 22.6, 1,000
    33.5 and 30.8, 2,000 (32 blocks) 41.4 and 43.3; 16 (64) behind 2,000 59.4 and 47.1; 40 (160) behind 3,700 248 and 104; one
    of 24 behind 8,000 keys and the others behind 200 (96) 1.5 times as fast, 16 tokens (64) all behind 8,000 0.89."""
    many = heads_a_group > 4
    if not plain:
        return any(reach <= keys and blocks >= least for keys, least in SHORT_SINK_BLOCKS[head_dim, many])
    if reach <= 128 and (many if head_dim == 128 else tokens <= 16):
        return False
    if head_dim == 64:
        return blocks <= N_SMS and (reach <= 256 or (reach <= 512 and (not many or blocks >= 24)))
    if many:
        return reach <= 256
    return (reach <= 256 or (reach <= 512 and blocks >= 48) or (reach <= 768 and blocks >= 80)
            or (reach <= 1024 and 80 <= blocks <= N_SMS))


def short_attention(q, out, k_cache, v_cache, ctx, table, count: int, reach: int, n_heads: int, n_kv_heads: int, head_dim: int,
                    scale: float, window, page_tokens: int, sinks=None, out_scale: float = 1.0, gate=None,
                    gate_per_head: bool = False, plain: bool = False) -> bool:
    """`csrc/attention_short.cu` for the step's first `count` requests, which bring one token each and whose contexts
    (`reach` at most), or windows, are short.  A rule of the step's shape and of the sizes.  False: not taken."""
    if (not SHORT_ATTENTION or head_dim not in (64, 128) or n_heads > 8 * n_kv_heads or q.stride(0) % 8 or q.data_ptr() % 16
            or k_cache.shape[-1] != head_dim or v_cache.shape[-1] != head_dim or k_cache.dtype != torch.bfloat16
            # (a short window's keys may lie in two of the split kernel's chunks, a short context's do not)
            or not short_attention_pays(count * n_kv_heads, reach if window is None or reach <= 128 else
                                        min(reach, max(window, 129)), head_dim, plain, n_heads // n_kv_heads, count)):
        return False
    code = build.load("attention_short").cb_attention_short(
        q.data_ptr(), q.stride(0), out.data_ptr(), out.stride(0), gate.data_ptr() if gate is not None else 0,
        gate.stride(0) if gate is not None else 0, 1 if gate_per_head else 0, k_cache.data_ptr(), v_cache.data_ptr(),
        sinks.data_ptr() if sinks is not None else 0, ctx.req_row_start.data_ptr(), ctx.req_first_pos.data_ptr(),
        table.data_ptr(), table.shape[1], count, n_heads, n_kv_heads, head_dim, page_tokens, scale, window or 0,
        out_scale, _stream())
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"short attention failed to launch (CUDA error {code})")
    _count(1)
    return True


DECODE_TC_TARGET_BLOCKS = 3 * N_SMS // 2  # two blocks of the tcgen05 decode kernel fit an SM, but they
                                          # start under the q/k/v product, whose blocks each take one
                                          # block's place until they end: a launch of more than about
                                          # one and a half blocks per SM starts in two waves
DECODE_TC_SHORT_BLOCKS = 22 * N_SMS // 10 # chunks of at most two tiles run with two K/V stages, three
                                          # blocks to an SM: a launch of up to this many finds its place
DECODE_MMA_TARGET_BLOCKS = 4 * N_SMS


def decode_chunk_keys(blocks_per_chunk: int, context_bucket: int, tcgen05: bool, head_dim: int = 64) -> int:
    """Keys per block of the split attention for decoded tokens: a function of the step's
    shape alone (so a captured step replays).  `blocks_per_chunk`: blocks that one chunk of
    every request takes (requests x KV heads x groups of 16 packed rows).  `context_bucket`:
    the longest context rounded up to a multiple of 256.

    tcgen05 form, from sweeps on B200 (120M shape, batch 1 to 64, contexts of 512 to 3,700):
    one tile of 128 keys per block while that is at most eight chunks (one round of the
    merge) and the launch finds its place at once; else two tiles per block while the launch
    finds its place (these short chunks run with two K/V stages, three blocks to an SM);
    else the bucket divided into as many equal parts as bring the launch nearest to one and
    a half blocks per SM, in whole tiles (batch 4 / 8 / 32 at 2,048 tokens: 0.307 / 0.321 /
    0.624 ms per step against 0.322 / 0.331 / 0.706 ms with chunks for 296 or 148 blocks).
    With heads of more than 64 features a block's three K/V stages are 192 KB, one block to an
    SM, and a launch of more blocks than SMs runs in two waves: the same rule with one block
    per SM as the most (Llama-3-8B layer sizes, 2,048 tokens, batch 4 / 8 / 16: 0.714 / 0.753 /
    0.824 ms per step of four layers against 0.736 / 0.773 / 0.854 ms).
    mma.sync form: the parts that bring the launch nearest to four blocks per SM."""
    unit = 128 if tcgen05 else 256
    whole = -(-context_bucket // unit) * unit
    one_per_sm = tcgen05 and head_dim > 64
    if tcgen05:
        short = N_SMS if one_per_sm else DECODE_TC_SHORT_BLOCKS
        n_one, n_two = -(-context_bucket // 128), -(-context_bucket // 256)
        if n_one <= 8 and blocks_per_chunk * n_one <= short:
            return min(128, whole)
        if blocks_per_chunk * n_two <= short:
            return min(256, whole)
    target = DECODE_TC_TARGET_BLOCKS if tcgen05 else DECODE_MMA_TARGET_BLOCKS
    if one_per_sm:
        parts = max(1, N_SMS // max(1, blocks_per_chunk))
    else:
        parts = max(1, (2 * target + blocks_per_chunk) // (2 * max(1, blocks_per_chunk)))
    chunk = -(-context_bucket // parts)
    chunk = -(-chunk // unit) * unit
    return min(max(chunk, unit), whole)


WIDE_ROW_TARGET_BLOCKS = 2 * N_SMS


def wide_row_chunk_keys(blocks_per_chunk: int, context_bucket: int, window) -> int:
    """Keys per block of the mma.sync split attention over rows of more than 128 features (one
    block to an SM; each of its four warps walks its sub-tiles of 16 keys one memory round trip
    after the other, so short chunks are what hides the latency).  Chunks lie at fixed places
    of the context; with a window only those that it touches work, so the working blocks are
    counted over the window's reach: as many parts as bring them nearest to two per SM, in
    whole tiles of 64 keys (one sub-tile a warp).  A function of the step's shape alone."""
    unit = 64
    reach = context_bucket if not window else min(context_bucket, window + unit)
    parts = max(1, (2 * WIDE_ROW_TARGET_BLOCKS + blocks_per_chunk) // (2 * max(1, blocks_per_chunk)))
    chunk = -(-reach // parts)
    chunk = -(-chunk // unit) * unit
    whole = -(-context_bucket // unit) * unit
    return min(max(chunk, unit), whole)


MIXED_REACH = 2048 * 256     # keys times features
MIXED_FEW = 12               # decoded tokens


def tiles_first(host, n_requests, head_dim, window, keep_first) -> int:
    """The first request of a step that the tcgen05 tiles take (`n_requests`: none): 0, or behind the
    single decoded tokens at its head, which the caller then runs with their keys dealt to several
    blocks.  A decoded token is a block of 128 rows like another in the tiles' launch and walks its keys
    alone, 10 us a thousand keys of 64 features, 12 of 128 and 21 of 256: it rides along unless few tokens
    have long to walk; the more there are, the longer the launch of their own takes.  (One launch and two,
    16 heads: of 128, 4 tokens behind 3,000 keys beside 2,000 of a prompt 48 and 70 us, 48 behind 3,500 beside 500
    62 and 242; of 256, 12 behind 3,500 beside 200 72 and 52, 24 behind 3,000 beside 300 62 and 66.)"""
    lead = host.lead_single
    if lead == 0 or lead == n_requests:
        return lead
    reach = host.lead_context_bucket
    if window is not None:
        reach = min(reach, window + 128 + (keep_first or 0))
    return 0 if reach * head_dim <= MIXED_REACH * (1 if lead <= MIXED_FEW else 4) else lead


def prompt_attention(q, out, k_cache, v_cache, n_heads, n_kv_heads, head_dim, scale, window, keep_first,
                     ctx, cache, table, chunked: bool = False, sinks=None, out_scale: float = 1.0,
                     gate=None, gate_per_head: bool = False, value_cols=None) -> int:
    """The tcgen05 attention for the requests of a step from `tiles_first` on, over keys and values of
    one size (`_tcgen05_rows`), with a window that may keep the first tokens or (`chunked`) is the size of
    chunks, and with a sink per head in the softmax (`sinks`) or none; `gate`: a logit for every result or
    (`gate_per_head`) head, or None.  `q`: rows of n_heads * head_dim.  Returns the first request taken (`ctx.n_requests`: none)."""
    host, none = getattr(ctx, "host", None), ctx.n_requests
    n_rep = n_heads // n_kv_heads
    if (not USE_TCGEN05_ATTENTION or host is None or q.dtype != torch.bfloat16
            or not _tcgen05_rows(head_dim, k_cache, v_cache) or k_cache.dtype != torch.bfloat16
            or q.stride(0) % 8 or out.stride(0) % 8 or q.data_ptr() % 16 or out.data_ptr() % 16
            or (gate is not None and (gate.dtype != q.dtype or (not gate_per_head and (
                gate.stride(0) % 8 or gate.data_ptr() % 16))))
            or k_cache.shape[-1] != head_dim or v_cache.shape[-1] != head_dim):
        return none
    first = tiles_first(host, none, head_dim, window, keep_first)
    if first == none or host.max_new_tokens * n_rep < 64:
        return none
    reqs = _Requests(ctx, table, first, none - first, host.max_new_tokens, host.context_bucket, ctx.n_tokens)
    taken = _attention_tcgen05(q, out, k_cache, v_cache, reqs, n_heads, n_kv_heads, head_dim, scale, window, cache,
                               keep_first=keep_first, chunked=chunked, sinks=sinks, out_scale=out_scale, gate=gate,
                               gate_per_head=gate_per_head, lead=host.lead_single if first == 0 else 0,
                               value_cols=value_cols)
    return first if taken else none


SPLIT_ROWS = 16          # packed rows (new tokens x heads of a group) the split form takes


def _attend(qkv, out, k_cache, v_cache, reqs, n_heads, n_kv_heads, head_dim, scale, window, ctx,
            cache, value_cols=None) -> bool:
    """One run of requests through the kernel that suits it.  A function of the run's
    shape (count, most new tokens, bucket) and of the sizes only."""
    n_rep = n_heads // n_kv_heads
    if (reqs.max_new == 1 and reqs.first == 0 and USE_TCGEN05_DECODE
            and short_attention(qkv, out, k_cache, v_cache, ctx, reqs.whole_table, reqs.count, reqs.reach, n_heads,
                                n_kv_heads, head_dim, scale, window, cache.page_tokens, plain=True)):
        return True
    split = reqs.max_new * n_rep <= SPLIT_ROWS
    pt = cache.page_tokens
    decode_tc = (USE_TCGEN05_DECODE and split and head_dim in (64, 128) and out.stride(0) % 2 == 0
                 and 8 <= pt <= 128 and pt & (pt - 1) == 0)
    partial = counters = None
    n_chunks, chunk_keys = 0, 256
    if split:
        groups = -(-reqs.max_new * n_rep // 16)
        blocks_per_chunk = reqs.count * n_kv_heads * groups
        if head_dim > 128:
            chunk_keys = wide_row_chunk_keys(blocks_per_chunk, reqs.bucket, window)
        else:
            chunk_keys = decode_chunk_keys(blocks_per_chunk, reqs.bucket, decode_tc, head_dim)
        n_chunks = -(-reqs.bucket // chunk_keys)
        floats = reqs.rows_end * n_heads * n_chunks * (head_dim + 2)
        partial = ctx.scratch("attn.partial", (floats,), torch.float32)
        if decode_tc:
            counters = _buffer(qkv.device, "attn.counters", blocks_per_chunk, torch.int32, zero=True)
    if (decode_tc
            and _attention_decode_tcgen05(qkv, out, k_cache, v_cache, reqs, n_heads, n_kv_heads,
                                          head_dim, scale, window, cache, partial, counters,
                                          n_chunks, chunk_keys)):
        return True
    if (USE_TCGEN05_ATTENTION and not split and _tcgen05_rows(head_dim, k_cache, v_cache)
            and reqs.max_new * n_rep >= 64 and out.stride(0) % 8 == 0
            and _attention_tcgen05(qkv, out, k_cache, v_cache, reqs, n_heads, n_kv_heads,
                                   head_dim, scale, window, cache, value_cols=value_cols)):
        return True
    if split and head_dim <= 128 and chunk_keys % 256:
        # the mma.sync split form of rows up to 128 features walks whole tiles of 256 keys
        chunk_keys = -(-chunk_keys // 256) * 256
        n_chunks = -(-reqs.bucket // chunk_keys)
    lib = build.load("attention_mma")
    code = lib.cb_attention_mma(
        qkv.data_ptr(), qkv.stride(0), out.data_ptr(),
        out.stride(0), k_cache.data_ptr(), v_cache.data_ptr(),
        ctx.positions.data_ptr(), reqs.row_start,
        reqs.first_pos, reqs.table,
        reqs.table_stride, reqs.rows_end, reqs.count,
        reqs.max_new, n_heads, n_kv_heads, head_dim,
        cache.page_tokens, scale, window or 0,
        partial.data_ptr() if partial is not None else 0, n_chunks,
        chunk_keys, _stream())
    if code == _UNSUPPORTED:
        return False
    if code != 0:
        raise RuntimeError(f"tensor-core attention failed to launch (CUDA error {code})")
    _count(1)                                    # (one of the step's attention forms, its merge with it)
    return True


def paged_attention(qkv, out, n_heads, n_kv_heads, head_dim, scale, window, ctx, cache,
                    binding, value_cols=None) -> bool:
    """Tensor-core attention over the paged cache.  Takes head sizes that are
    multiples of 16 up to 256 and any head counts, group sizes and page sizes;
    refuses anything else (the plain kernel then runs).

    The kernel is chosen per request, not per step: requests that bring at most 16
    query rows per KV head (decoded tokens, tiny portions) run split over chunks of
    keys, merged by a kernel of their own (heads of 64 and 128: by the last block of a row
    group to arrive); longer portions run as tiles (the tcgen05 kernel for head sizes 64 and
    128, and 256 where a cached row is key and value at once, the mma.sync kernel of 64-row
    tiles else).  A step that holds both kinds (single decoded tokens first, as the
    scheduler orders them, then portions) is two launches over disjoint runs of its
    requests; the shapes of both are functions of the step's shape."""
    if (qkv.dtype != torch.bfloat16 or head_dim % 16 != 0 or head_dim > 256
            or n_heads % n_kv_heads != 0 or qkv.stride(0) % 8 != 0 or out.stride(0) % 2 != 0):
        return False
    k_cache, v_cache = cache.keys(binding.slot), cache.values(binding.slot)
    table = ctx.block_table(binding.group)
    host = ctx.host
    n_rep = n_heads // n_kv_heads
    args = (n_heads, n_kv_heads, head_dim, scale, window, ctx, cache, value_cols)
    lead = host.lead_single
    if 0 < lead < ctx.n_requests and host.max_new_tokens * n_rep > SPLIT_ROWS:
        decoding = _Requests(ctx, table, 0, lead, 1, host.lead_context_bucket, lead, host.lead_context_reach)
        portions = _Requests(ctx, table, lead, ctx.n_requests - lead, host.max_new_tokens,
                             host.context_bucket, ctx.n_tokens)
        if not _attend(qkv, out, k_cache, v_cache, decoding, *args):
            return False
        if not _attend(qkv, out, k_cache, v_cache, portions, *args):
            raise RuntimeError("the attention kernels took the step's decoded tokens but "
                               "refused its portions: a rule of sizes is inconsistent")
        return True
    whole = _Requests(ctx, table, 0, ctx.n_requests, host.max_new_tokens, host.context_bucket,
                      ctx.n_tokens, host.context_reach)
    return _attend(qkv, out, k_cache, v_cache, whole, *args)


def run_wait_probe(device, limit: int = 4096) -> None:
    """Launches a kernel whose only thread waits, bounded by `limit` polls, on a barrier
    nothing arrives at, and then records its give-up code in the status word: the failure
    path of the tensor-core kernels, made to happen without a fault (for tests)."""
    lib = build.load("gemm_tcgen05")
    code = lib.cb_tc_wait_probe(status_word(device).data_ptr(), limit, _stream())
    if code != 0:
        raise RuntimeError(f"wait probe failed to launch (CUDA error {code})")
