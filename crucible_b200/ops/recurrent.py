"""Wrappers of `csrc/recurrent.cu`: mixers that carry a matrix per head from token to
token in the request's state slot (the gated delta rule, the mLSTM, the wkv rule, the
state-space rule, the delta rule with a decay per key channel)."""
from __future__ import annotations

import functools

import torch

from . import LAUNCHES, KernelError, _check, _code, _need_cuda, _ptr, _stream, build, tensor_core

DELTA, MLSTM, WKV, SSD, CHANNEL = 0, 1, 2, 3, 4
GATE_SILU, GATE_SIGMOID = 0, 1
CHUNKS = True                # tests switch it off to reach the token-by-token walk with the same inputs
STEP = True                  # likewise, for the form of a token each


# us of the walk over tokens (a launch, a token of the longest portion, a token and head of 128, a portion and head) with
# 1, 2 and 4 columns of a matrix a lane, fitted over 4 to 32 heads of 64 and 128 and 1 to 48 uneven portions of up to 4
# to 490 tokens, and of the chunks (their launches, a chunk and head of 128), fitted over 4 to 32 heads and 1 to 12 portions of
# 24 to 900 tokens on average
_DELTA_WALK = {1: (3.43, 0.183, 0.0060, 0.0553), 2: (3.49, 0.227, 0.0037, 0.0460), 4: (4.55, 0.337, 0.0032, 0.0383)}
COSTS = {DELTA: (_DELTA_WALK, (14.0, 0.188)), CHANNEL: (_DELTA_WALK, (14.5, 0.236)),
         MLSTM: ({1: (3.49, 0.192, 0.0072, 0.0613), 2: (4.35, 0.240, 0.0046, 0.0430), 4: (5.75, 0.350, 0.0036, 0.0361)},
                 (21.5, 0.124)),
         WKV: ({1: (3.28, 0.148, 0.0068, 0.0647), 2: (3.55, 0.172, 0.0037, 0.0515), 4: (3.50, 0.296, 0.0035, 0.0419)},
               (19.5, 0.120)),
         SSD: ({1: (3.60, 0.127, 0.0038, 0.0635), 2: (4.41, 0.142, 0.0026, 0.0446), 4: (5.84, 0.181, 0.0027, 0.0341)},
               (18.0, 0.112))}


@functools.lru_cache(maxsize=4096)
def walk_columns(rule, requests: int, rows: int, longest: int, n_heads: float, key_dim: int, value_dim: int):
    """How many columns of its matrix a lane of the walk takes, and the walk's us.  Every lane of a column's eight reads
    the token's k and q out of shared memory, which is what many portions wait for: with 2 or 4 columns a
    lane half or a quarter of it, and the state's rows come in 8 or 16 bytes; but fewer blocks, and a token of a
    lone portion takes longer.  32 portions of up to 24 tokens, 16 heads of 128, with 1, 2 and 4: delta rule 78, 61
    and 57 us, state space 67, 50 and 48; one of 90 27, 28 and 41, 21, 23 and 33.  Up to a block an SM, and where
    nobody knows the longest portion (0), one is taken, else what costs least, if that is clearly less than one costs:
    by a twentieth; by more than a fifth where one portion is over a third of the rows, whose blocks, dealt out between
    the others', come to lie on a few of the SMs (portions of 180, 130, 75, 40, 9 and 1, 16 heads of 128 by the delta rule,
    1 and 2: reckoned 83 and 75 us, measured 86 and 98).  The mLSTM's one column has three blocks of 128 channels an SM, not
    four: an eighth (330 and 290, 32 heads: 218 and 149).  Of 500 steps measured 4 are more than 1.5 % behind one
    column as it was before there were more (up to 4 %), the mean 11 % ahead."""
    heads = n_heads * key_dim / 128
    cost = {c: start + token * longest + (work * rows + portion * requests) * heads
            for c, (start, token, work, portion) in COSTS[rule][0].items()}
    us, columns = min((us, c) for c, us in cost.items())
    clearly = 0.95 if rows >= 3 * longest else 0.87 if rule == MLSTM else 0.78
    if longest <= 0 or requests * n_heads * -(-value_dim // 16) <= 148 or us > clearly * cost[1]:
        return 1, cost[1]
    return columns, us


def chunks_pay(rule, rows: int, requests: int, longest: int, heads: float) -> bool:
    """Whether a bfloat16 step's portions (`rows` tokens of `requests`, without the single tokens at the
    step's head; the longest; `heads` of 128 key channels) go in chunks.  The walk takes its time a token of the
    longest portion until the requests fill the GPU, then a time a token; a chunk that holds few tokens
    costs what a full one does, and every portion ends in one such.  16 heads of 128, chunks and walk: delta rule
    1 portion of 110 tokens 27 and 30 us, 24 of up to 300 514 and 450; state space 1 of 140 35 and 31, of 500 45 and
    103; 24 of up to 60 101 and 90.
    The chunks' launches and workspaces are some 30 us of host work, which a step that runs eagerly pays and whose
    host time covers either form of little work (wkv, a portion of 150: 37 and 36 us on the device, the layer
    eagerly 275 and 242): less than 96 tokens a request of the delta rules, or less than 160 of a few of the others,
    are walked, and more where the costs say that the walk is ahead.  Of 532 steps
    measured that are enough work for that, the choice is 0.7 % from the quicker form on average (46 % at worst), and none
    is slower than by one column or by the chunks as they were before there were more."""
    if requests <= 0:
        return False
    if rule in (DELTA, CHANNEL):
        if rows < 96 * requests:
            return False
    elif longest < 160 and (longest < 48 or rows < 24 * requests or rows * heads < 4096):
        return False
    first, chunk = COSTS[rule][1]
    walk = walk_columns(rule, requests, rows, longest, heads, 128, 128)[1]      # of the form that would be launched
    return walk > first + chunk * (rows / 32 + requests / 2) * heads


CHUNK_SPACE = 256 << 20      # bytes of the chunks' workspaces


@functools.lru_cache(maxsize=256)
def _space_of(rule, n_heads: int, key_dim: int, value_dim: int):
    """Bytes that a row and that a chunk take in the chunks' workspaces."""
    delta, vector = rule in (DELTA, CHANNEL), rule in (WKV, CHANNEL)
    return (4 * n_heads * (key_dim * ((delta or vector) + delta + (rule == CHANNEL)) + value_dim * delta + 4),
            4 * n_heads * (key_dim * (vector + (rule == MLSTM)) + (0 if delta else key_dim * value_dim) + 1))


@functools.lru_cache(maxsize=4096)
def _chunk_room(rule, rows: int, requests: int, n_heads: int, key_dim: int, value_dim: int, slices: bool):
    """The chunks' workspaces in one buffer: its floats, and where wq, ww, wk, wu, ws, wg, wl, wn, wm and the
    slices' n and m begin (-1: the rule has none)."""
    delta, vector, mlstm = rule in (DELTA, CHANNEL), rule in (WKV, CHANNEL), rule == MLSTM
    row, chunk = rows * n_heads, (rows // 32 + requests) * n_heads
    sizes = (row * key_dim * (delta or vector), row * key_dim * delta, row * key_dim * (rule == CHANNEL),
             row * value_dim * delta, row * 4, chunk * key_dim * vector, 0 if delta else chunk * key_dim * value_dim,
             chunk * key_dim * mlstm, chunk * mlstm, 2 * requests * n_heads * (key_dim + 1) * (mlstm and slices))
    floats, begins = 0, []
    for size in sizes:
        begins.append(floats if size else -1)
        floats += -(-size // 4) * 4                 # (16-byte boundaries)
    return floats, tuple(begins)


def slice_tokens(rows: int, requests: int, longest: int, row_bytes: int, chunk_bytes: int) -> int:
    """Tokens of each of `requests` portions (`rows` tokens in all) that go through the chunks at a time: all of
    the longest if the workspaces then stay within CHUNK_SPACE, else what does, in whole chunks and one
    at least.  (16 heads of 128 x 128 take 25 to 33 KB a token, so that up to 8,000 tokens go at once;
    a longer step's slices each fill the GPU.)"""
    if rows * row_bytes + (rows // 32 + requests) * chunk_bytes <= CHUNK_SPACE:
        return longest
    per_token = requests * (row_bytes + chunk_bytes / 32)
    return max(32, int((CHUNK_SPACE - requests * chunk_bytes) / per_token) // 32 * 32)


def _state_args(state: torch.Tensor):
    if state.dtype != torch.uint8 or state.dim() != 2 or state.stride(1) != 1:
        raise KernelError("a mixer's state is a uint8 view [slots, bytes]")
    if state.data_ptr() % 16:
        raise KernelError("a mixer's state must start on a 16-byte boundary")
    return _ptr(state), state.stride(0)


def delta_prepare(proj, conv_w, taps, gates, a_log, dt_bias, ctx, state, tail_off, qkv, beta,
                  decay, n_heads, n_kv_heads, key_dim, value_dim, update_tail: bool = False) -> bool:
    """`update_tail`: the convolution's inputs in the state may be replaced here; returns whether they
    were (else `conv_tail_update` does it)."""
    _need_cuda(proj, conv_w, gates, a_log, dt_bias, state, qkv, beta, decay)
    if _conv_prepare(proj, conv_w, None, taps, gates, a_log, dt_bias, ctx, state, tail_off, qkv, decay, beta, n_heads,
                     qkv.shape[1], 2 * n_kv_heads, key_dim, False, update_tail):
        return update_tail
    sp, stride = _state_args(state)
    lib = build.load("recurrent")
    _check(lib.cb_delta_prepare(
        _ptr(proj), proj.stride(0), _code(proj.dtype), _ptr(conv_w), taps,
        _ptr(gates), gates.stride(0), _ptr(a_log), _ptr(dt_bias), _ptr(ctx.row_request), _ptr(ctx.req_row_start),
        _ptr(ctx.req_state_slot), sp, stride, tail_off, _ptr(qkv), _ptr(beta), _ptr(decay),
        proj.shape[0], n_heads, n_kv_heads, key_dim,
        value_dim, _stream()), "delta_prepare")
    return False


def _conv_prepare(proj, conv_w, conv_b, taps, gates, a_log, dt_bias, ctx, state, tail_off, dst, num0, num1, n_heads,
                  channels, unit_heads, head_size, is_ssd: bool, update: bool) -> bool:
    """The preparations' form of 16 bytes a lane; `proj`: rows that start with the convolution's channels.
    A rule of the sizes alone.  False: not taken."""
    host = getattr(ctx, "host", None)
    if (host is None or proj.stride(1) != 1 or not dst.is_contiguous() or not num0.is_contiguous()
            or not num1.is_contiguous() or not conv_w.is_contiguous() or conv_w.shape[1] != taps):
        return False
    sp, stride = _state_args(state)
    lib = build.load("recurrent")
    code = lib.cb_conv_prepare(
        _ptr(proj), proj.stride(0), _code(proj.dtype), _ptr(conv_w), _ptr(conv_b), taps,
        _ptr(gates), gates.stride(0), _ptr(a_log), _ptr(dt_bias), _ptr(ctx.req_row_start),
        _ptr(ctx.req_state_slot), sp, stride, tail_off, _ptr(dst), _ptr(num0), _ptr(num1),
        ctx.n_requests, host.max_new_tokens, n_heads, channels, unit_heads,
        head_size, 1 if is_ssd else 0, 1 if update else 0, _stream())
    if code == build.UNSUPPORTED:
        return False
    _check(code, "conv_prepare")
    return True


def channel_delta_prepare(proj, conv_w, rate, beta_logit, a_log, dt_bias, ctx, state, tail_off, qkv, beta,
                          n_heads, n_qk_heads, key_dim, value_dim) -> None:
    """`proj` rows [q: G*D | k: G*D | v: H*E | ...], `conv_w` float32 [taps, channels], `rate`
    float32 rows of H*D decay logits, `beta_logit` float32 rows of H.  qkv = float32
    [unit q * D^-1/2 | unit k | v | exp(-exp(a_log) softplus(rate + dt_bias))], beta = sigmoid; the
    convolution's inputs in the state (float32 [taps - 1, channels] at `tail_off`) are read and
    rewritten."""
    _need_cuda(proj, conv_w, rate, beta_logit, a_log, dt_bias, state, qkv, beta)
    C = 2 * n_qk_heads * key_dim + n_heads * value_dim
    f32 = torch.float32
    if (proj.stride(1) != 1 or proj.shape[1] < C or conv_w.dtype != f32 or not conv_w.is_contiguous()
            or conv_w.shape[1] != C or rate.dtype != f32 or rate.stride(1) != 1 or rate.shape[1] < n_heads * key_dim
            or beta_logit.dtype != f32 or beta_logit.stride(1) != 1 or qkv.dtype != f32 or not qkv.is_contiguous()
            or qkv.shape[1] != C + n_heads * key_dim or beta.dtype != f32 or not beta.is_contiguous()
            or a_log.numel() != n_heads or dt_bias.numel() != n_heads * key_dim):
        raise KernelError("channel_delta_prepare: rows [q | k | v], float32 taps [taps, channels], logits and outputs")
    sp, stride = _state_args(state)
    lib = build.load("recurrent")
    _check(lib.cb_channel_delta_prepare(
        _ptr(proj), proj.stride(0), _code(proj.dtype), _ptr(conv_w), conv_w.shape[0],
        _ptr(rate), rate.stride(0), _ptr(beta_logit), beta_logit.stride(0), _ptr(a_log),
        _ptr(dt_bias), _ptr(ctx.req_row_start), _ptr(ctx.req_state_slot), sp, stride, tail_off, _ptr(qkv),
        _ptr(beta), ctx.n_requests, ctx.host.max_new_tokens, n_heads, n_qk_heads,
        key_dim, value_dim, _stream()), "channel_delta_prepare")


def conv_tail_update(proj, taps, channels, ctx, state, tail_off) -> None:
    _need_cuda(proj, state)
    sp, stride = _state_args(state)
    lib = build.load("recurrent")
    _check(lib.cb_conv_tail_update(
        _ptr(proj), proj.stride(0), _code(proj.dtype), taps, channels,
        _ptr(ctx.req_row_start), _ptr(ctx.req_state_slot), sp, stride, tail_off,
        ctx.n_requests, _stream()), "conv_tail_update")


def mlstm_prepare(proj, gates, bias_i, bias_f, cap, qkv, log_keep, log_in, n_heads, key_dim,
                  value_dim, ctx=None, state=None, n_off=0, m_off=0, kept=None) -> None:
    """`kept` (with `ctx`, `state` and the offsets of n and m in it): float32 [requests, H*D + H] that
    receives the requests' n and m as the step begins, for `matrix_memory`."""
    _need_cuda(proj, gates, bias_i, bias_f, qkv, log_keep, log_in, state, kept)
    sp, stride = _state_args(state) if kept is not None else (_ptr(None), 0)
    if kept is not None and (kept.dtype != torch.float32 or not kept.is_contiguous()
                             or tuple(kept.shape) != (ctx.n_requests, n_heads * (key_dim + 1))
                             or proj.shape[0] < ctx.n_requests):
        raise KernelError("mlstm_prepare: kept is float32 [requests, H*D + H]")
    lib = build.load("recurrent")
    _check(lib.cb_mlstm_prepare(
        _ptr(proj), proj.stride(0), _code(proj.dtype), _ptr(gates), gates.stride(0), _ptr(bias_i),
        _ptr(bias_f), cap, _ptr(qkv), _ptr(log_keep), _ptr(log_in), proj.shape[0],
        n_heads, key_dim, value_dim, _ptr(kept),
        _ptr(ctx.req_state_slot if kept is not None else None), sp, stride, n_off, m_off,
        ctx.n_requests if kept is not None else 0, _stream()), "mlstm_prepare")


def retention_prepare(proj, freq, rotary_dim: int, split_halves: bool, ctx, head_decay, k_scale: float,
                      qkv, keep, step, n_heads: int, key_dim: int, value_dim: int) -> None:
    """Rows of `proj` are [q: H*D | k: H*D | v: H*E | ...]: the first `rotary_dim` features of
    every q and k head turn by position * freq (float32), k times `k_scale` afterwards; qkv =
    float32 [q | k | v]; keep[t, h] = head_decay[h], step[t, h] = 1 (what the state-space rule
    of `matrix_memory` reads for S <- decay S + k v^T)."""
    _need_cuda(proj, freq, head_decay, qkv, keep, step)
    if (proj.stride(1) != 1 or qkv.dtype != torch.float32 or not qkv.is_contiguous()
            or qkv.shape[1] != n_heads * (2 * key_dim + value_dim)
            or head_decay.dtype != torch.float32 or head_decay.numel() != n_heads
            or keep.dtype != torch.float32 or step.dtype != torch.float32
            or not keep.is_contiguous() or not step.is_contiguous()):
        raise KernelError("retention_prepare: contiguous rows, float32 outputs [rows, H (2D + E)] and "
                          "[rows, H], one float32 decay per head")
    if rotary_dim and (freq is None or freq.dtype != torch.float32 or freq.numel() * 2 != rotary_dim):
        raise KernelError("retention_prepare: freq is float32 [rotary_dim / 2]")
    lib = build.load("recurrent")
    _check(lib.cb_retention_prepare(
        _ptr(proj), proj.stride(0), _code(proj.dtype), _ptr(freq), rotary_dim,
        1 if split_halves else 0, _ptr(ctx.positions), _ptr(head_decay), k_scale,
        _ptr(qkv), _ptr(keep), _ptr(step), proj.shape[0], n_heads, key_dim,
        value_dim, _stream()), "retention_prepare")


def matrix_memory(rule, qkv, q_off, k_off, v_off, sc0, sc1, ctx, state, s_off, n_off, m_off, out,
                  n_heads, n_qk_heads, key_dim, value_dim, w_off=0, per_head=None, kept=None) -> None:
    """Walks every request's tokens in order through its heads' matrices (see the kernel).
    `w_off`: where the wkv and channel rules' decay vectors (one a head) lie in the rows of `qkv`; `per_head`: float32
    constants, the wkv rule's bonus [heads, key_dim] or the state-space rule's skip [heads]; `kept`: the
    mLSTM's n and m as `mlstm_prepare` left them (None: they are copied here)."""
    _need_cuda(qkv, sc0, sc1, state, out, per_head, kept)
    if rule == MLSTM and kept is None:
        nd, slots = n_heads * key_dim, ctx.req_state_slot.long()
        kept = torch.cat([state[:, n_off:n_off + 4 * nd][slots].contiguous().view(torch.float32),
                          state[:, m_off:m_off + 4 * n_heads][slots].contiguous().view(torch.float32)], 1)
    if per_head is not None and (per_head.dtype != torch.float32 or not per_head.is_contiguous()):
        raise KernelError("matrix_memory: the per-head constants are contiguous float32")
    if qkv.dtype != torch.float32 or out.dtype != torch.float32 or not qkv.is_contiguous():
        raise KernelError("matrix_memory takes prepared float32 rows")
    sp, stride = _state_args(state)
    n, walked = ctx.n_requests, ctx.n_requests
    # (without the host's counts of the step, or in 32 bits: the walk alone)
    counts = getattr(ctx, "host", None)
    host = counts if getattr(ctx, "dtype", None) == torch.bfloat16 else None
    starts, slots, kept_at = (t.data_ptr() if t is not None else 0 for t in (ctx.req_row_start, ctx.req_state_slot, kept))
    w_off_read = w_off if rule in (WKV, CHANNEL) else 0
    if (CHUNKS and host is not None and chunks_pay(
                rule, qkv.shape[0] - host.lead_single, n - host.lead_single, host.max_new_tokens, n_heads * key_dim / 128)
            and key_dim <= 128 and (qkv.shape[1] | q_off | k_off | v_off | key_dim | value_dim | w_off_read) % 4 == 0
            and (s_off | state.stride(0) | qkv.data_ptr() | out.data_ptr() | state.data_ptr()) % 16 == 0):
        # prompts' portions in chunks; the requests at the head of the step that bring one token are walked
        walked = host.lead_single
        longest, requests = host.max_new_tokens, n - walked
        limit = slice_tokens(qkv.shape[0] - walked, requests, longest, *_space_of(rule, n_heads, key_dim, value_dim))
        rows = min(qkv.shape[0] - walked, requests * limit)
        floats, begins = _chunk_room(rule, rows, requests, n_heads, key_dim, value_dim, limit < longest)
        room = ctx.scratch("memory.chunks", (floats,), torch.float32).data_ptr()
        wq, ww, wk, wu, ws, wg, wl, wn, wm, kept_room = (room + 4 * at if at >= 0 else 0 for at in begins)
        lib = build.load("recurrent_chunks")
        code = lib.cb_matrix_memory_chunks(
            rule, _ptr(qkv), qkv.shape[1], q_off, k_off, v_off,
            _ptr(sc0), _ptr(sc1), starts + 4 * walked, slots + 4 * walked, sp, stride,
            s_off, n_off, m_off, _ptr(out), requests,
            longest, n_heads, n_qk_heads, key_dim, value_dim,
            w_off, _ptr(per_head),
            kept_at + 4 * walked * n_heads * (key_dim + 1) if kept is not None else 0,
            limit, kept_room, wq, ww, wk, wu, ws, wg, wl, wn, wm,
            qkv.shape[0], rows, tensor_core.status_word(qkv.device).data_ptr(), _stream())
        if code == build.UNSUPPORTED:            # the walk's
            walked = n
        else:
            _check(code, "matrix_memory (chunks)")
            LAUNCHES[0] += (2 if rule in (DELTA, CHANNEL) else 3) * -(-longest // limit) - 1
    if walked == 0:
        return
    lib = build.load("recurrent")
    # decoded tokens of the bfloat16 engine: a token each, S read and written once
    step = (STEP and host is not None and host.lead_single >= walked
            and (qkv.shape[1] | v_off | value_dim) % 4 == 0 and (s_off | state.stride(0)) % 16 == 0)
    args = (rule, _ptr(qkv), qkv.shape[1], q_off, k_off, v_off,
            _ptr(sc0), _ptr(sc1), starts, slots, sp, stride,
            s_off, n_off, m_off, _ptr(out), walked,
            n_heads, n_qk_heads, key_dim, value_dim, w_off,
            _ptr(per_head), kept_at, _stream())
    code = lib.cb_matrix_memory_step(*args) if step else build.UNSUPPORTED
    if code == build.UNSUPPORTED:
        rows, longest = ((walked, 1) if walked < n else (qkv.shape[0], counts.max_new_tokens if counts is not None else 0))
        columns = walk_columns(rule, walked, rows, longest, n_heads, key_dim, value_dim)[0]
        code = lib.cb_matrix_memory(*args[:-1], columns, args[-1])
    _check(code, "matrix_memory")


def head_norm_gate(o, gain, gain_per_head, gate, out, gate_kind, n_heads, value_dim, eps,
                   out_scale) -> None:
    """out = o / rms(o over a head) * gain * act(gate) * out_scale; `out` is a view of rows in
    the engine dtype, `gate` one in the engine dtype or in float32.  `gain` None: a norm without a weight."""
    _need_cuda(o, gain, gate, out)
    if (o.dtype != torch.float32 or gate.dtype not in (out.dtype, torch.float32) or gate.stride(1) != 1
            or out.stride(1) != 1):
        raise KernelError("head_norm_gate: float32 input, gate rows of the output's dtype or float32")
    lib = build.load("recurrent")
    _check(lib.cb_head_norm_gate(
        _ptr(o), _ptr(gain), value_dim if gain_per_head else 0, _ptr(gate),
        gate.stride(0), _code(gate.dtype), _ptr(out), out.stride(0),
        _code(out.dtype), gate_kind, o.shape[0], n_heads, value_dim, eps,
        out_scale, _stream()), "head_norm_gate")


def shift_mix(h, mu, ctx, state, prev_off, out) -> None:
    """out[s, t] = h[t] + (h[t-1] - h[t]) * mu[s]; the row before a portion's first row is the
    request's state (float32 [width] at `prev_off`), which then becomes the portion's last row."""
    _need_cuda(h, mu, state, out)
    if (mu.dtype != torch.float32 or not mu.is_contiguous() or h.stride(1) != 1 or out.dtype != h.dtype
            or not out.is_contiguous() or tuple(out.shape) != (mu.shape[0], h.shape[0], h.shape[1])):
        raise KernelError("shift_mix: float32 mixes [n, width], rows of one dtype, output [n, rows, width]")
    sp, stride = _state_args(state)
    lib = build.load("recurrent")
    _check(lib.cb_shift_mix(
        _ptr(h), h.stride(0), _code(h.dtype), _ptr(mu), mu.shape[0],
        _ptr(ctx.row_request), _ptr(ctx.req_row_start), _ptr(ctx.req_state_slot), sp, stride,
        prev_off, _ptr(out), h.shape[0], h.shape[1], _stream()), "shift_mix")


def wkv_prepare(rkv, logit, w0, qkv, n_channels) -> None:
    """`rkv`: [>= 3, rows, channels] (r, k, v); qkv = float32 [r | k | v | exp(-exp(logit + w0))],
    each of `n_channels` columns."""
    _need_cuda(rkv, logit, w0, qkv)
    if (logit.dtype != torch.float32 or qkv.dtype != torch.float32 or not logit.is_contiguous()
            or not qkv.is_contiguous() or rkv.dim() != 3 or rkv.shape[0] < 3 or not rkv.is_contiguous()
            or rkv.shape[2] != n_channels or qkv.shape[1] != 4 * n_channels):
        raise KernelError("wkv_prepare: planes [3, rows, channels], float32 logits and output "
                          "[rows, 4 * channels]")
    lib = build.load("recurrent")
    _check(lib.cb_wkv_prepare(_ptr(rkv), rkv.stride(0), _code(rkv.dtype), _ptr(logit),
                              _ptr(w0), _ptr(qkv), rkv.shape[1], n_channels, _stream()),
           "wkv_prepare")


def ssd_prepare(proj, conv_at, conv_w, conv_b, taps, gates, a_log, dt_bias, ctx, state, tail_off, xbc,
                decay, step, n_heads, channels, update_tail: bool = False) -> bool:
    """Causal convolution with bias + SiLU over `channels` columns of `proj` from `conv_at`
    on; step size softplus(gate + dt_bias) and decay exp(-exp(A_log) * step) per head.
    `update_tail` and the result as in `delta_prepare`."""
    _need_cuda(proj, conv_w, conv_b, gates, a_log, dt_bias, state, xbc, decay, step)
    if proj.stride(1) != 1 or gates.dtype != torch.float32 or xbc.dtype != torch.float32:
        raise KernelError("ssd_prepare: contiguous rows, float32 gates and output")
    if _conv_prepare(proj[:, conv_at:conv_at + channels], conv_w, conv_b, taps, gates, a_log, dt_bias, ctx, state,
                     tail_off, xbc, decay, step, n_heads, channels, 0, 0, True, update_tail):
        return update_tail
    sp, stride = _state_args(state)
    lib = build.load("recurrent")
    _check(lib.cb_ssd_prepare(
        _ptr(proj), proj.stride(0), conv_at, _code(proj.dtype), _ptr(conv_w),
        _ptr(conv_b), taps, _ptr(gates), gates.stride(0), _ptr(a_log), _ptr(dt_bias),
        _ptr(ctx.row_request), _ptr(ctx.req_row_start), _ptr(ctx.req_state_slot), sp, stride,
        tail_off, _ptr(xbc), _ptr(decay), _ptr(step), proj.shape[0], n_heads,
        channels, _stream()), "ssd_prepare")
    return False


def gate_group_norm(y, gate, gain, out, parts, eps) -> None:
    """out = unit-rms, in `parts` equal parts of a row, of y * silu(gate), times gain."""
    _need_cuda(y, gate, gain, out)
    if (y.dtype != torch.float32 or not y.is_contiguous() or gate.dtype != out.dtype
            or gate.stride(1) != 1 or out.stride(1) != 1 or y.shape[1] % parts):
        raise KernelError("gate_group_norm: float32 input, gate and output rows of one dtype, "
                          "a width that the parts divide")
    lib = build.load("recurrent")
    _check(lib.cb_gate_group_norm(_ptr(y), _ptr(gate), gate.stride(0), _ptr(gain), _ptr(out),
                                  out.stride(0), _code(out.dtype), y.shape[0],
                                  y.shape[1], parts, eps, _stream()),
           "gate_group_norm")
