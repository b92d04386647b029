"""Torch-tensor front end of libb200_mixers.so (include/b200_mixers.h): ragged-batch mixers and feed-forward pieces.

Same rules as ``ops``: shapes are checked on the host, raw device pointers and torch's current stream go to the
library, nothing here computes and nothing falls back to torch.  Activations of a step are packed ``[n_tok, ...]``.
"""
from __future__ import annotations

import functools
from typing import Optional

import torch

from . import _lib
from .ops import DTYPE_ID, _need_cuda, _stream


# benchmark instrumentation: when set to a list, every op appends (name, start event, end event) recorded on the
# launching stream around its C-ABI call
EVENTS: Optional[list] = None


def _timed(fn):
    @functools.wraps(fn)
    def wrapper(*args, **kwargs):
        if EVENTS is None:
            return fn(*args, **kwargs)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        out = fn(*args, **kwargs)
        b.record()
        EVENTS.append((fn.__name__, a, b))
        return out

    return wrapper


def _lib_():
    return _lib.load_mixers()


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _rows2(x: torch.Tensor) -> int:
    """Row stride of a 2-D view whose last dimension is contiguous."""
    if x.dim() != 2 or (x.shape[1] > 1 and x.stride(1) != 1):
        raise ValueError("expected a 2-D tensor with a contiguous last dimension")
    return x.stride(0) if x.shape[0] > 1 else max(x.stride(0), x.shape[1])


@_timed
def offset_rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """``x * rsqrt(mean(x^2) + eps) * (1 + weight)``: fp32 ``[rows, width]`` in, the weight's dtype out."""
    _need_cuda(x, weight)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2:
        raise ValueError("the residual stream is a contiguous fp32 [rows, width] tensor")
    out = torch.empty(x.shape, dtype=weight.dtype, device=x.device)
    rc = _lib_().b200_offset_rmsnorm(out.data_ptr(), x.data_ptr(), weight.data_ptr(), float(eps), x.shape[0], x.shape[1],
                                     DTYPE_ID[weight.dtype], _stream())
    _lib.check_mixers(rc, "b200_offset_rmsnorm")
    return out


@_timed
def postnorm_residual(x: torch.Tensor, y: torch.Tensor, w_post: torch.Tensor, mult: float, eps: float,
                      w_next: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """In place ``x += mult * offset_norm(y; w_post)`` (fp32); returns ``offset_norm(x; w_next)`` in the weights'
    dtype when ``w_next`` is given.  ``y``: the weights' dtype or fp32."""
    _need_cuda(x, y, w_post)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or y.shape != x.shape:
        raise ValueError("x must be contiguous fp32 [rows, width] and y of the same shape")
    if y.dtype not in (w_post.dtype, torch.float32):
        raise TypeError("y must have the weights' dtype or be fp32")
    out = torch.empty(x.shape, dtype=w_post.dtype, device=x.device) if w_next is not None else None
    rc = _lib_().b200_postnorm_residual(x.data_ptr(), y.data_ptr(), _rows2(y), int(y.dtype == torch.float32 and
                                        w_post.dtype != torch.float32), w_post.data_ptr(), float(mult), _ptr(w_next),
                                        _ptr(out), float(eps), x.shape[0], x.shape[1], DTYPE_ID[w_post.dtype], _stream())
    _lib.check_mixers(rc, "b200_postnorm_residual")
    return out


@_timed
def value_prep_append(k: torch.Tensor, v: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor,
                      slot_mapping: torch.Tensor, eps: float, v_prev: Optional[torch.Tensor] = None, lam: float = 0.0,
                      v_keep: Optional[torch.Tensor] = None) -> None:
    """Unit-RMS values per head (optionally mixed with ``v_prev``), then k / v into the pools at ``slot_mapping``.
    ``k [n, G*dk]``, ``v [n, G*dv]`` (column slices of a projection are fine); pools ``[blocks, G, bs, dk|dv]``."""
    _need_cuda(k, v, k_pool, v_pool, slot_mapping)
    nb, G, bs, dk = k_pool.shape
    dv = v_pool.shape[3]
    n = k.shape[0]
    if k.shape[1] != G * dk or v.shape != (n, G * dv) or tuple(v_pool.shape[:3]) != (nb, G, bs):
        raise ValueError("k / v do not match the pools")
    if slot_mapping.dtype != torch.int64 or slot_mapping.numel() != n:
        raise ValueError("slot_mapping must be int64 [n_tok]")
    for t in (v_prev, v_keep):
        if t is not None and (tuple(t.shape) != (n, G * dv) or not t.is_contiguous() or t.dtype != v.dtype):
            raise ValueError("v_prev / v_keep must be contiguous [n_tok, G*dv] in the storage dtype")
    rc = _lib_().b200_value_prep_append(k.data_ptr(), _rows2(k), v.data_ptr(), _rows2(v), _ptr(v_prev), _ptr(v_keep),
                                        float(lam), float(eps), k_pool.data_ptr(), v_pool.data_ptr(),
                                        slot_mapping.data_ptr(), n, G, dk, dv, bs, nb, DTYPE_ID[k_pool.dtype], _stream())
    _lib.check_mixers(rc, "b200_value_prep_append")


def attn_tile_tokens(n_tokens: int, H: int, G: int) -> int:
    return int(_lib_().b200_biased_attn_tile_tokens(int(n_tokens), H, G))


@_timed
def biased_paged_attention(q: torch.Tensor, gate: Optional[torch.Tensor], k_pool: torch.Tensor, v_pool: torch.Tensor,
                           block_tables: torch.Tensor, tiles: torch.Tensor, max_tile_tokens: int, tok_pos: torch.Tensor,
                           bias_lut: torch.Tensor, scale: float, temp_coef: float, temp_every: int, H: int,
                           out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal attention of packed rows ``q [n, H*dk]`` over the paged cache with a distance-bias table
    ``bias_lut [H, L]`` (fp32), a query temperature and a sigmoid gate ``gate [n, H]``; returns ``[n, H*dv]``
    (the tiles' rows of ``out`` when given)."""
    _need_cuda(q, k_pool, v_pool, block_tables, tiles, tok_pos, bias_lut)
    nb, G, bs, dk = k_pool.shape
    dv = v_pool.shape[3]
    n = q.shape[0]
    if q.shape[1] != H * dk or (gate is not None and tuple(gate.shape) != (n, H)):
        raise ValueError("q / gate do not match the head layout")
    if block_tables.dtype != torch.int32 or tiles.dtype != torch.int32 or tok_pos.dtype != torch.int32:
        raise TypeError("block tables, tiles and positions are int32")
    if tiles.dim() != 2 or tiles.shape[1] != 3 or not tiles.is_contiguous():
        raise ValueError("tiles must be contiguous int32 [n_tiles, 3]")
    if bias_lut.dtype != torch.float32 or bias_lut.shape[0] != H or not bias_lut.is_contiguous():
        raise ValueError("bias_lut must be contiguous fp32 [H, L]")
    if out is None:
        out = torch.empty((n, H * dv), dtype=q.dtype, device=q.device)
    rc = _lib_().b200_biased_paged_attn(out.data_ptr(), q.data_ptr(), _rows2(q), _ptr(gate),
                                        _rows2(gate) if gate is not None else 0, k_pool.data_ptr(), v_pool.data_ptr(),
                                        block_tables.data_ptr(), block_tables.stride(0), tiles.data_ptr(), tiles.shape[0],
                                        int(max_tile_tokens), tok_pos.data_ptr(), bias_lut.data_ptr(), bias_lut.shape[1],
                                        float(scale), float(temp_coef), int(temp_every), H, G, dk, dv, bs,
                                        DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_biased_paged_attn")
    return out


def prompt_tile_tokens(H: int, G: int) -> int:
    """Tokens of one sequence a CTA of the tensor-core kernel serves: 64 rows over the heads of a kv group."""
    return int(_lib_().b200_biased_prompt_attn_tile_tokens(int(H), int(G)))


def prompt_attention_supported(dk: int, dv: int, dtype: torch.dtype) -> bool:
    return bool(_lib_().b200_biased_prompt_attn_supported(int(dk), int(dv), DTYPE_ID[dtype]))


# Bytes up to which ``biased_prompt_attention`` divides keys over CTAs.  Steps beyond (256 sequences of 16 heads, one of them at 130000
# tokens) have CTAs enough without; dividing always at multiples of the same size is what keeps a row's sums its own.
SPLIT_WORKSPACE = 1 << 30


@_timed
def biased_prompt_attention(out: torch.Tensor, q: torch.Tensor, gate: Optional[torch.Tensor], k_pool: torch.Tensor,
                            v_pool: torch.Tensor, block_tables: torch.Tensor, tiles: torch.Tensor, tok_pos: torch.Tensor,
                            bias_lut: torch.Tensor, scale: float, temp_coef: float, temp_every: int, H: int,
                            max_tile_tokens: int = 0, max_context: int = 0) -> None:
    """``biased_paged_attention`` on the tensor cores, for prompt portions and decoded tokens alike; writes the tiles'
    rows of ``out`` ``[n, H*dv]`` (16-bit dtypes, see ``prompt_attention_supported``).  ``tiles``: up to
    ``prompt_tile_tokens(H, G)`` tokens each; ``max_tile_tokens``: the largest tile (0 = unknown) — steps of decoded
    tokens only take the variant whose warps split the keys; with ``max_context`` (a bound on the tiles' contexts) its CTAs do too."""
    _need_cuda(out, q, k_pool, v_pool, block_tables, tiles, tok_pos, bias_lut)
    nb, G, bs, dk = k_pool.shape
    dv = v_pool.shape[3]
    n = q.shape[0]
    if q.shape[1] != H * dk or tuple(out.shape) != (n, H * dv) or not out.is_contiguous() or out.dtype != q.dtype:
        raise ValueError("q / out do not match the head layout")
    if gate is not None and tuple(gate.shape) != (n, H):
        raise ValueError("gate must be [n, H]")
    if tiles.dtype != torch.int32 or tiles.dim() != 2 or tiles.shape[1] != 3 or not tiles.is_contiguous():
        raise ValueError("tiles must be contiguous int32 [n_tiles, 3]")
    if bias_lut.dtype != torch.float32 or bias_lut.shape[0] != H or not bias_lut.is_contiguous():
        raise ValueError("bias_lut must be contiguous fp32 [H, L]")
    lib = _lib_()
    ws = None
    if 0 < max_tile_tokens * (H // G) <= 16 and max_context > lib.b200_biased_attn_split_keys():
        splits = -(-max_context // lib.b200_biased_attn_split_keys())
        rows = tiles.shape[0] * max_tile_tokens     # the tiles' own: a step's prompts beside them are another launch's
        if splits * rows * H * (dv + 2) * 4 <= SPLIT_WORKSPACE:
            ws = torch.empty((splits, rows, H, dv + 2), dtype=torch.float32, device=q.device)
    rc = lib.b200_biased_prompt_attn_ext(out.data_ptr(), q.data_ptr(), _rows2(q), _ptr(gate),
                                         _rows2(gate) if gate is not None else 0, k_pool.data_ptr(), v_pool.data_ptr(),
                                         block_tables.data_ptr(), block_tables.stride(0), tiles.data_ptr(), tiles.shape[0],
                                         int(max_tile_tokens), tok_pos.data_ptr(), bias_lut.data_ptr(), bias_lut.shape[1], float(scale),
                                         float(temp_coef), int(temp_every), H, G, dk, dv, bs, int(max_context), _ptr(ws), DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_biased_prompt_attn")


# Tokens of a step's longest portion from which the recurrences (gated, delta, retention) may run in chunks on the tensor cores.  B200, bf16,
# 64 x 128 states, us token by token / in chunks: 8 x 96 tokens of 4 heads gated 15.4 / 15.8, delta 21.9 / 21.4, retention 16.9 / 18.6; 192
# tokens 27.4 / 22.2, 38.5 / 30.5, 25.2 / 24.9; 2048 tokens 248 / 154, 382 / 233, 191 / 151.
SPLIT_SCAN_FROM = (96, 96, 160)
# Chunks take 8 - 10 us more of the host (a workspace, two launches): a step whose mixer leaves the device waiting walks until the walk is
# longer than that, from ``SPLIT_SCAN_ALONE`` tokens in one portion or ``SPLIT_SCAN_WORK`` = longest portion x tokens x heads on.  The mixers
# called from Python, us walking / in chunks: gated, width 512, 1 portion of 200 64 / 73, 300 64 / 73, 448 74 / 74, 576 89 / 75; width 2048, 4 of
# 200 65 / 74, 4 of 300 87 / 78, 8 of 200 95 / 89.  Delta, width 512, 1 of 300 119 / 129, 448 128 / 130, 576 151 / 130; width 2048, 4 of 300
# 151 / 132.  Retention, width 512, 1 of 448 140 / 148, 576 (in segments) 155 / 149; width 2048, 2 of 448 137 / 142, 4 of 448 192 / 178.
SPLIT_SCAN_ALONE = (448, 448, 512)
SPLIT_SCAN_WORK = (3600000, 3600000, 6500000)
SPLIT_SCAN_WORKSPACE = 1 << 30      # bytes of chunk operands at most (one head's if that is more); the heads go in groups beyond, smaller
                                    # ones where memory is short, and token by token where one head's do not fit


def split_scan_pays(rule: int, longest: int, n: int, n_seqs: int, H: int, dk: int, dv: int) -> bool:
    """Whether chunks are ahead for a step of ``n`` tokens in ``n_seqs`` portions, the longest of ``longest`` (rule 0: gated, 1: delta, 2:
    retention; ``H`` states of ``dk`` x ``dv``).  A chunk's work does not shrink with the state (padded to 64 keys and 64-column blocks) nor
    with the portion (a single token takes a chunk), what chunks shorten is the chain of a long portion.  B200, bf16, us token by token / in
    chunks (gated):

    64 x 128 states, whose chunks cost less than their tokens: 64 portions of 96, 16 heads 163 / 136; 512 beside 63 single tokens 107 / 74; but
    96 beside 255, of 4, 16, 32 heads 38 / 46, 122 / 179, 232 / 351, 160 beside 63, 32 heads 77 / 97.
    64 x 64, 16 heads: 8 of 512 77 / 70, 512 beside 63 95 / 59, but 64 of 96 85 / 100, of 256 205 / 222.  Smaller ones likewise from longer
    portions on: 32 x 128 8 of 192 38 / 38, 64 of 256 284 / 316; 16 x 16 1 of 512 71 / 45, 8 of 192 29 / 33, 256 of 96 224 / 387.
    Retention of up to 32 keys walks at 63 ns a token: 1 of 512 39 / 42, 8 of 2048 of 32 x 32 133 / 243."""
    chunks = n // 16 + n_seqs
    if longest < SPLIT_SCAN_ALONE[rule] and (longest < SPLIT_SCAN_FROM[rule] or longest * n * H < SPLIT_SCAN_WORK[rule]):
        return False
    if dk > 32 and 13 * dv >= 64 * (8 + 7 * -(-dv // 64)):
        return 16 * chunks <= 2 * n or 8 * longest >= H * chunks
    if dk <= 32 and rule == 2:
        return False
    return 2 * longest >= 3 * SPLIT_SCAN_FROM[rule] and 16 * chunks <= 4 * n and (16 if dv > 32 else 4) * longest >= H * chunks


def split_scan_takes(rule: int, max_count: int, n: int, n_seqs: int, H: int, dk: int, dv: int, dtype: torch.dtype) -> bool:
    """Whether such a step runs in chunks (``split_scan_pays``): ``max_count`` tokens in its longest portion, 0 or more than ``n``: unknown."""
    return max_count <= n and split_scan_pays(rule, max_count, n, n_seqs, H, dk, dv) and _split_scan_supported(dk, dtype)


@functools.lru_cache(maxsize=None)
def _split_scan_supported(dk: int, dtype: torch.dtype) -> bool:
    return bool(_lib_().b200_split_scan_supported(dk, DTYPE_ID[dtype]))


@functools.lru_cache(maxsize=None)
def _chunk_bytes(rule: int) -> int:
    """Workspace of one chunk and head."""
    return int(_lib_().b200_split_scan_workspace(rule, 0, 1, 1))


def _chunk_workspace(one: int, H: int, device: torch.device) -> Optional[torch.Tensor]:
    """Room for the chunk operands (``one`` bytes a head) of as many of ``H`` heads as the device still holds; None: not for one."""
    heads = max(1, min(H, SPLIT_SCAN_WORKSPACE // one))
    while heads:
        try:
            return torch.empty(heads * one, dtype=torch.uint8, device=device)
        except torch.OutOfMemoryError:
            heads //= 2
    return None


def split_scan_segment(rule: int, longest: int, n: int, n_seqs: int, H: int, dv: int) -> int:
    """Chunks per segment of a step in chunks; 0: its sequences in one piece.  Segments make the walk shorter and the work 1.4 times as much (the
    state of the middle ones is walked twice), so they pay where the sequences leave SMs idle and the longest takes twice as long as an SM's share
    of the work.  Not for the delta rule, whose decay is no diagonal.  B200, bf16, 64 x 128 states, us in one piece / in segments,
    operands included: 4 heads, 1 of 2048 124 / 36, 8 of 2048 160 / 124, 8 of 512 45 / 44, 16 of 400 44 / (58), 1 of 512 38 / 24; 8 heads, 6 of 720 -
    1780 139 / 105, 8 of 1024 102 / (118); 16 heads, 2 of 1000 79 / 67.  (More CTAs than SMs: 16 heads, 6 of 720 - 1780 225 / 181 in a graph by
    themselves, but the gated mixer around them 361 / 362; hardly fewer CTAs: 16 heads, 2 of 900 103 / 105 with the mixer, 2 of 1150 125 / 122.)
    Under 48 chunks they save less than the 7 us of host time that they take (8 heads, 6 of 210 - 690: 58 / 51).  Their length: short ones fill the
    chip from little work, long ones start seldom and add fewer ends up (4 heads, 1 of 2048: 4 chunks 38, 8 35, 16 47; 16 heads, 1 of 8192: 8
    chunks 321, 16 239, 32 239)."""
    chunks, blocks = (longest + 15) // 16, H * -(-dv // 64)
    if rule == 1 or chunks < 48 or n_seqs * blocks > 148:
        return 0
    share = (n // 16 + n_seqs) * blocks / 148
    return int(max(4 + share / 8, chunks / 32)) if chunks >= 2 * share + 8 else 0


def split_segments_wait(rule: int, longest: int, n: int, H: int) -> bool:
    """Whether a step of 48 chunks and more is better off without segments, which cost the host 6.5 us (a launch, a tensor): the mixer around
    them takes the device less time in one piece than the host needs for it with segments, by the longest walk and, for what stands beside it,
    the tokens and heads.  B200, bf16, 64 x 128 states, called from Python, us in one piece / in segments: gated, width 512, 1 of 760 77 / 84,
    1000 78 / 85, 1300 93 / 85, 8 of up to 840 80 / 85, 940 90 / 85; width 1024, 1 of 1000 81 / 85, 1150 88 / 85, 2 of 900 84 / 85, 1000 90 / 86;
    width 2048, 1 of 760 83 / 85, 900 93 / 86.  Attention beside retention, whose host side is longer: width 512, 1 of 1500 147 / 152, 2000 157 /
    152, 4 of up to 1250 146 / 152, 1670 171 / 153; width 1024, 2 of 1150 147 / 154, 1300 162 / 153; width 2048, 1 of 1000 148 / 154, 1150 163 /
    155."""
    chunks = (longest + 15) // 16
    return chunks >= 48 and (chunks + n * H * (37 + H) / 17000 < 128 if rule == 2 else chunks + n * H * (20 + H) / 20000 < 80)


@functools.lru_cache(maxsize=None)
def _end_floats() -> int:
    """What a segment leaves per head and 64 value columns."""
    return int(_lib_().b200_split_scan_ends(1, 0, 1, 1, 64)) // 4


def _split_scan(rule: int, o, q, k, v, stride: int, beta, a, bias, rate, decay, per_channel: bool, state, seqs, G: int, eps: float,
                scale: float, longest: int = 0) -> bool:
    """``b200_split_scan`` into ``o``; ``beta`` and ``a`` are (tensor or None, row stride).  False, with nothing done, where the device
    has no memory left for its workspace: the token-by-token scans need none."""
    _, H, dk, dv = state.shape
    lib, n, n_seqs = _lib_(), q.shape[0], seqs.shape[0]
    ws = _chunk_workspace((n // 16 + n_seqs) * _chunk_bytes(rule), H, q.device)
    if ws is None:
        return False
    segment, ends = split_scan_segment(rule, longest, n, n_seqs, H, dv), None
    if segment and split_segments_wait(rule, longest, n, H):
        segment = 0
    if segment:
        try:
            ends = torch.empty((n // 16 + n_seqs) // segment * H * -(-dv // 64) * _end_floats(), dtype=torch.float32, device=q.device)
        except torch.OutOfMemoryError:
            segment = 0
    rc = lib.b200_split_scan_ext(rule, o.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), stride, _ptr(beta[0]), beta[1], _ptr(a[0]), a[1],
                             _ptr(bias), _ptr(rate), _ptr(decay), int(per_channel), state.data_ptr(), seqs.data_ptr(), n_seqs, n, H, G, dk,
                             dv, float(eps), float(scale), ws.data_ptr(), ws.numel(), segment, _ptr(ends),
                                 4 * ends.numel() if segment else 0, DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_split_scan")
    return True


@_timed
def gated_scan(zq: torch.Tensor, zf: torch.Tensor, v: torch.Tensor, f_bias: torch.Tensor, lower: torch.Tensor,
               state: torch.Tensor, seqs: torch.Tensor, H: int, max_count: int = 1 << 20) -> torch.Tensor:
    """Gated linear recurrence over each sequence's tokens; ``state`` fp32 ``[slots, H, dk, dv]`` is read (unless the
    sequence is fresh) and written back.  ``zq / zf [n, H*dk]``, ``v [n, H*dv]`` are column slices of ONE projection
    (same row stride).  ``max_count``: the largest token count in ``seqs`` (picks the kernel; a hint, not a bound; beyond ``n``: unknown):
    16-bit steps with long portions (``split_scan_pays``) and keys of up to 64 run in chunks on the tensor cores, others token by token.
    Returns the raw read-outs, fp32 ``[n, H, dv]``."""
    _need_cuda(zq, zf, v, state, seqs)
    n = zq.shape[0]
    _, Hs, dk, dv = state.shape
    if Hs != H or zq.shape[1] != H * dk or zf.shape != zq.shape or v.shape != (n, H * dv):
        raise ValueError("projections do not match the state's shape")
    stride = _rows2(zq)
    if n > 1 and (zf.stride(0) != stride or v.stride(0) != stride):
        raise ValueError("zq, zf and v must share a row stride")
    if state.dtype != torch.float32 or not state.is_contiguous():
        raise TypeError("the recurrent state is contiguous fp32")
    if seqs.dtype != torch.int32 or seqs.dim() != 2 or seqs.shape[1] != 4 or not seqs.is_contiguous():
        raise ValueError("seqs must be contiguous int32 [n_seqs, 4]")
    o = torch.empty((n, H, dv), dtype=torch.float32, device=zq.device)
    if split_scan_takes(0, max_count, n, seqs.shape[0], H, dk, dv, zq.dtype) and _split_scan(
            0, o, zq, zf, v, stride, (None, 0), (None, 0), f_bias, lower, None, False, state, seqs, H, 0.0, 0.0, max_count):
        return o
    rc = _lib_().b200_gated_scan(o.data_ptr(), zq.data_ptr(), zf.data_ptr(), v.data_ptr(), stride, f_bias.data_ptr(),
                                 lower.data_ptr(), state.data_ptr(), seqs.data_ptr(), seqs.shape[0], int(max_count), H, dk, dv,
                                 DTYPE_ID[zq.dtype], _stream())
    _lib.check_mixers(rc, "b200_gated_scan")
    return o


@_timed
def head_rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """fp32 ``[..., dv]`` rows -> ``x * rsqrt(mean(x^2) + eps) * weight`` in the weight's dtype."""
    _need_cuda(x, weight)
    if x.dtype != torch.float32 or not x.is_contiguous():
        raise ValueError("x must be contiguous fp32")
    dv = x.shape[-1]
    out = torch.empty(x.shape, dtype=weight.dtype, device=x.device)
    rc = _lib_().b200_head_rmsnorm(out.data_ptr(), x.data_ptr(), weight.data_ptr(), float(eps), x.numel() // dv, dv,
                                   DTYPE_ID[weight.dtype], _stream())
    _lib.check_mixers(rc, "b200_head_rmsnorm")
    return out


@_timed
def polynorm(z: torch.Tensor, coef: torch.Tensor, eps: float) -> torch.Tensor:
    _need_cuda(z, coef)
    out = torch.empty(z.shape, dtype=z.dtype, device=z.device)
    rc = _lib_().b200_polynorm(out.data_ptr(), z.data_ptr(), _rows2(z), coef.data_ptr(), float(eps), z.shape[0],
                               z.shape[1], DTYPE_ID[z.dtype], _stream())
    _lib.check_mixers(rc, "b200_polynorm")
    return out


@_timed
def sigmoid_topk(logits: torch.Tensor, top: int):
    """fp32 ``[n, E]`` logits -> ``(ids int32 [n, top], weights fp32 [n, top])``; weights are sigmoid(logit)."""
    _need_cuda(logits)
    if logits.dtype != torch.float32 or not logits.is_contiguous() or logits.dim() != 2:
        raise ValueError("router logits are contiguous fp32 [n, E]")
    n, E = logits.shape
    ids = torch.empty((n, top), dtype=torch.int32, device=logits.device)
    w = torch.empty((n, top), dtype=torch.float32, device=logits.device)
    rc = _lib_().b200_sigmoid_topk(ids.data_ptr(), w.data_ptr(), logits.data_ptr(), n, E, int(top), _stream())
    _lib.check_mixers(rc, "b200_sigmoid_topk")
    return ids, w


def zero_blocks(pools, slots) -> None:
    """Blocks ``slots`` (a host list) of every tensor of ``pools`` (contiguous ``[blocks, ...]`` on one device) set to zero in one launch
    there, whatever the current device is."""
    import ctypes

    n, m = len(pools), len(slots)
    if not n or not m:
        return
    _need_cuda(*pools)
    if any(p.device != pools[0].device or not p.is_contiguous() for p in pools):
        raise ValueError("pools are contiguous and on one device")
    if min(slots) < 0 or max(slots) >= min(p.shape[0] for p in pools):
        raise IndexError(f"block slots {min(slots)} .. {max(slots)} of pools of {min(p.shape[0] for p in pools)} blocks")
    with torch.cuda.device(pools[0].device):
        rc = _lib_().b200_zero_blocks((ctypes.c_void_p * n)(*[p.data_ptr() for p in pools]),
                                      (ctypes.c_int64 * n)(*[p.stride(0) * p.element_size() for p in pools]), n,
                                      (ctypes.c_int32 * m)(*slots), m, _stream())
    _lib.check_mixers(rc, "b200_zero_blocks")


@_timed
def expert_order(ids: torch.Tensor, n_experts: int):
    """``(order int64 [n * top], where int64 [n * top], offsets int32 [n_experts + 1])`` for ``ids`` int32 ``[n, top]`` in ``0 ..
    n_experts - 1``: the pairs in stable expert order, the inverse, and where each expert's rows start.  Other ids come behind the last
    expert, so that ``order`` and ``where`` are permutations whatever the ids are.  Nothing travels to the host."""
    _need_cuda(ids)
    if ids.dtype != torch.int32 or not ids.is_contiguous():
        raise TypeError("expert ids are contiguous int32")
    n, lib = ids.numel(), _lib_()
    if not lib.b200_expert_order_supported(n, int(n_experts)):     # more pairs or experts than the one-CTA sort holds
        flat = ids.reshape(-1).clamp(-1, n_experts).remainder_(n_experts + 1)     # ids of no expert: n_experts
        sorted_ids, order = torch.sort(flat.to(torch.int16) if n_experts < 1 << 15 else flat, stable=True)
        where = torch.empty_like(order)
        where[order] = torch.arange(n, device=ids.device)
        bounds = torch.arange(n_experts + 1, device=ids.device).to(sorted_ids.dtype)
        return order, where, torch.searchsorted(sorted_ids, bounds).to(torch.int32)
    order = torch.empty((n,), dtype=torch.int64, device=ids.device)
    where = torch.empty_like(order)
    offsets = torch.empty((n_experts + 1,), dtype=torch.int32, device=ids.device)
    rc = lib.b200_expert_order(order.data_ptr(), where.data_ptr(), offsets.data_ptr(), ids.data_ptr(), n, int(n_experts), _stream())
    _lib.check_mixers(rc, "b200_expert_order")
    return order, where, offsets


@_timed
def scaled_gather(h: torch.Tensor, weights: torch.Tensor, src: torch.Tensor, top: int) -> torch.Tensor:
    _need_cuda(h, weights, src)
    if not h.is_contiguous() or src.dtype != torch.int64 or weights.dtype != torch.float32:
        raise ValueError("h contiguous, src int64, weights fp32")
    xs = torch.empty((src.numel(), h.shape[1]), dtype=h.dtype, device=h.device)
    rc = _lib_().b200_scaled_gather(xs.data_ptr(), h.data_ptr(), weights.data_ptr(), src.data_ptr(), src.numel(), int(top),
                                    h.shape[1], DTYPE_ID[h.dtype], _stream())
    _lib.check_mixers(rc, "b200_scaled_gather")
    return xs


def grouped_linear_supported(K: int, dtype: torch.dtype) -> bool:
    return bool(_lib_().b200_grouped_linear_supported(int(K), DTYPE_ID[dtype]))


@_timed
def grouped_linear(xs: torch.Tensor, w: torch.Tensor, offsets: torch.Tensor) -> torch.Tensor:
    """``out[r] = xs[r] @ w[e].T`` for ``offsets[e] <= r < offsets[e + 1]``: ``xs [rows, K]`` sorted by expert,
    ``w [E, N, K]``, ``offsets`` int32 ``[E + 1]`` on the device (no host copy).  16-bit dtypes."""
    _need_cuda(xs, w, offsets)
    E, N, K = w.shape
    if xs.dim() != 2 or xs.shape[1] != K or not xs.is_contiguous() or not w.is_contiguous() or xs.dtype != w.dtype:
        raise ValueError("xs [rows, K] and w [E, N, K] must be contiguous and of one dtype")
    if offsets.dtype != torch.int32 or offsets.numel() != E + 1 or not offsets.is_contiguous():
        raise ValueError("offsets must be contiguous int32 [E + 1]")
    out = torch.empty((xs.shape[0], N), dtype=xs.dtype, device=xs.device)
    rc = _lib_().b200_grouped_linear(out.data_ptr(), xs.data_ptr(), w.data_ptr(), offsets.data_ptr(), xs.shape[0], E, N, K,
                                     DTYPE_ID[xs.dtype], _stream())
    _lib.check_mixers(rc, "b200_grouped_linear")
    return out


@_timed
def clamped_glu(gu: torch.Tensor, limit: float, alpha: float) -> torch.Tensor:
    _need_cuda(gu)
    if not gu.is_contiguous() or gu.shape[1] % 2:
        raise ValueError("gu must be contiguous [rows, 2*ff]")
    ff = gu.shape[1] // 2
    y = torch.empty((gu.shape[0], ff), dtype=gu.dtype, device=gu.device)
    rc = _lib_().b200_clamped_glu(y.data_ptr(), gu.data_ptr(), gu.shape[0], ff, float(limit), float(alpha),
                                  DTYPE_ID[gu.dtype], _stream())
    _lib.check_mixers(rc, "b200_clamped_glu")
    return y


@_timed
def expert_combine(ys: torch.Tensor, where: torch.Tensor, n_tok: int, top: int) -> torch.Tensor:
    _need_cuda(ys, where)
    if not ys.is_contiguous() or where.dtype != torch.int64 or where.numel() != n_tok * top:
        raise ValueError("ys contiguous, where int64 [n_tok * top]")
    out = torch.empty((n_tok, ys.shape[1]), dtype=torch.float32, device=ys.device)
    rc = _lib_().b200_expert_combine(out.data_ptr(), ys.data_ptr(), where.data_ptr(), n_tok, int(top), ys.shape[1],
                                     DTYPE_ID[ys.dtype], _stream())
    _lib.check_mixers(rc, "b200_expert_combine")
    return out


# ---- pieces for hybrid designs (csrc/b200_hybrid_ops.cu) ---------------------------------------------------------------
@_timed
def rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float, weight_offset: float = 0.0) -> torch.Tensor:
    """``x * rsqrt(mean(x^2) + eps) * (weight_offset + weight)`` over the last dimension of 2-D rows (fp32 or the
    weight's dtype, column slices are fine); the weight's dtype out."""
    _need_cuda(x, weight)
    if x.dtype not in (torch.float32, weight.dtype) or weight.numel() != x.shape[1]:
        raise ValueError("x must be fp32 or of the weight's dtype, [rows, width] with width = weight.numel()")
    out = torch.empty(x.shape, dtype=weight.dtype, device=x.device)
    rc = _lib_().b200_rms_norm(out.data_ptr(), out.shape[1], x.data_ptr(), _rows2(x),
                               int(x.dtype == torch.float32 and weight.dtype != torch.float32), weight.data_ptr(),
                               float(weight_offset), float(eps), x.shape[0], x.shape[1], DTYPE_ID[weight.dtype], _stream())
    _lib.check_mixers(rc, "b200_rms_norm")
    return out


@_timed
def residual_add2_norm(x: torch.Tensor, a: torch.Tensor, b: Optional[torch.Tensor], w_next: Optional[torch.Tensor],
                       eps: float, weight_offset: float = 0.0) -> Optional[torch.Tensor]:
    """In place ``x += (a + b)`` on the fp32 residual (``b`` may be None); returns ``rms_norm(x; w_next)`` in the
    branches' dtype when ``w_next`` is given."""
    _need_cuda(x, a)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or a.shape != x.shape:
        raise ValueError("x must be contiguous fp32 [rows, width] and the branches of the same shape")
    if b is not None and (b.shape != x.shape or b.dtype != a.dtype):
        raise ValueError("both branches must have one shape and dtype")
    out = torch.empty(x.shape, dtype=a.dtype, device=x.device) if w_next is not None else None
    rc = _lib_().b200_residual_add2_norm(x.data_ptr(), a.data_ptr(), _rows2(a), _ptr(b), _rows2(b) if b is not None else 0,
                                         _ptr(w_next), float(weight_offset), _ptr(out), float(eps), x.shape[0], x.shape[1],
                                         DTYPE_ID[a.dtype], _stream())
    _lib.check_mixers(rc, "b200_residual_add2_norm")
    return out


@_timed
def xielu(z: torch.Tensor, pq: torch.Tensor) -> torch.Tensor:
    """``z > 0: softplus(p) z^2 + z/2;  z <= 0: (1/2 + softplus(q)) (exp(z) - 1 - z) + z/2`` with ``pq = (p, q)``."""
    _need_cuda(z, pq)
    if pq.numel() != 2 or pq.dtype != z.dtype:
        raise ValueError("pq holds the two numbers (p, q) in the activations' dtype")
    out = torch.empty(z.shape, dtype=z.dtype, device=z.device)
    rc = _lib_().b200_xielu(out.data_ptr(), z.data_ptr(), _rows2(z), pq.data_ptr(), z.shape[0], z.shape[1],
                            DTYPE_ID[z.dtype], _stream())
    _lib.check_mixers(rc, "b200_xielu")
    return out


@_timed
def rotary_kv_append(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor,
                     slot_mapping: torch.Tensor, tok_pos: torch.Tensor, H: int, rot_dims: int, rot_base: float,
                     rotate_values: bool, interleaved: bool = False, want_table: bool = False) -> Optional[torch.Tensor]:
    """Rotary positions on q (in place) and k over their first ``rot_dims`` dimensions, optionally the values turned
    over their whole width; k and v are stored in the pools at ``slot_mapping``.  With ``want_table`` returns fp32
    ``[n, dv // 2, 2]`` = (cos, sin) of the value pairs' angles (what ``mixed_prompt_attention`` turns outputs back
    with)."""
    _need_cuda(q, k, v, k_pool, v_pool, slot_mapping, tok_pos)
    nb, G, bs, dk = k_pool.shape
    dv = v_pool.shape[3]
    n = q.shape[0]
    if q.shape[1] != H * dk or k.shape != (n, G * dk) or v.shape != (n, G * dv):
        raise ValueError("q / k / v do not match the pools")
    if slot_mapping.dtype != torch.int64 or tok_pos.dtype != torch.int32:
        raise TypeError("slot_mapping is int64, tok_pos int32")
    table = (torch.empty((n, dv // 2, 2), dtype=torch.float32, device=q.device)
             if want_table and rotate_values else None)
    rc = _lib_().b200_rotary_kv_append(q.data_ptr(), _rows2(q), k.data_ptr(), _rows2(k), v.data_ptr(), _rows2(v),
                                       k_pool.data_ptr(), v_pool.data_ptr(), slot_mapping.data_ptr(), tok_pos.data_ptr(),
                                       n, H, G, dk, dv, int(rot_dims), float(rot_base), int(rotate_values),
                                       int(interleaved), bs, nb, _ptr(table), DTYPE_ID[k_pool.dtype], _stream())
    _lib.check_mixers(rc, "b200_rotary_kv_append")
    return table


@_timed
def norm_append(x: torch.Tensor, weight: torch.Tensor, eps: float, pool: torch.Tensor, slot_mapping: torch.Tensor,
                weight_offset: float = 0.0) -> None:
    """``pool[slot] = rms_norm(x[n]; weight)``: latent rows into a one-head pool ``[blocks, 1, bs, width]``."""
    _need_cuda(x, weight, pool, slot_mapping)
    if pool.shape[1] != 1 or pool.shape[3] != x.shape[1] or x.dtype != pool.dtype or slot_mapping.dtype != torch.int64:
        raise ValueError("the pool must be [blocks, 1, block size, width] in the rows' dtype; slots int64")
    rc = _lib_().b200_norm_append(x.data_ptr(), _rows2(x), weight.data_ptr(), float(weight_offset), float(eps),
                                  pool.data_ptr(), slot_mapping.data_ptr(), x.shape[0], x.shape[1], DTYPE_ID[x.dtype],
                                  _stream())
    _lib.check_mixers(rc, "b200_norm_append")


def _gate_kind(gate: Optional[torch.Tensor], n: int, H: int, dv: int, dtype: torch.dtype) -> int:
    """0: no gate, or one per head (``[n, H]``); 1: one per output channel (``[n, H*dv]``)."""
    if gate is None:
        return 0
    if gate.dtype != dtype or tuple(gate.shape) not in ((n, H), (n, H * dv)):
        raise ValueError("gate must be [n, H] or [n, H*dv] in the activations' dtype")
    return int(gate.shape[1] != H)


def _value_layout(k_pool: torch.Tensor, v_pool: torch.Tensor, value_width: Optional[int], value_div: int):
    """``(value size, elements between value rows)`` of an attention call, after checking the pools against each other."""
    if v_pool.dim() != 4 or v_pool.shape[0] != k_pool.shape[0] or v_pool.shape[2] != k_pool.shape[2]:
        raise ValueError("the pools must agree on blocks and block size")
    if value_div < 1 or v_pool.shape[1] * value_div != k_pool.shape[1]:
        raise ValueError("v_pool holds one head per `value_div` key heads")
    v_row = v_pool.shape[3]
    dv = v_row if value_width is None else int(value_width)
    if dv < 1 or dv > v_row:
        raise ValueError("value_width exceeds the rows of v_pool")
    return dv, v_row


@_timed
def mixed_paged_attention(out: torch.Tensor, q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor,
                          block_tables: torch.Tensor, tok_row: torch.Tensor, tok_pos: torch.Tensor, scale: float,
                          talk: Optional[torch.Tensor] = None, sink: Optional[torch.Tensor] = None, window: int = 0,
                          keep_first: int = 0, unrotate_base: Optional[float] = None, interleaved: bool = False,
                          gate: Optional[torch.Tensor] = None, softcap: float = 0.0, chunk: int = 0,
                          value_width: Optional[int] = None, value_div: int = 1) -> None:
    """Softmax attention of packed query rows over the paged cache.  ``q`` and ``out`` are 3-D ``[n, H, dk | dv]``
    VIEWS with a contiguous last dimension (any token / head strides); ``talk`` fp32 ``[H, H]`` mixes the heads'
    scores before the softmax, ``sink`` fp32 ``[H]`` adds exp(sink) to the denominator, ``window`` > 0 limits a
    position to its last ``window`` tokens plus the sequence's first ``keep_first``, ``unrotate_base`` turns the
    output back by the position over the value width, ``gate`` holds the logits of a sigmoid gate per head (``[n, H]``) or
    per output channel (``[n, H*dv]``, not with ``unrotate_base``), ``softcap`` > 0
    bounds the scores by ``softcap * tanh(score / softcap)`` before the mask, ``chunk`` > 0 lets a position see only
    the keys of its own block of ``chunk`` positions, ``value_width`` says that the values are the first that many
    columns of the (wider) rows of ``v_pool``, ``value_div`` that ``v_pool`` holds one value head per that many key
    heads (several score maps over the same values).  ``out`` may be fp32 whatever the storage dtype (results that are
    combined before they are rounded; not with ``unrotate_base``)."""
    _need_cuda(out, q, k_pool, v_pool, block_tables, tok_row, tok_pos)
    nb, G, bs, dk = k_pool.shape
    dv, v_row = _value_layout(k_pool, v_pool, value_width, value_div)
    n, H = q.shape[0], q.shape[1]
    if q.dim() != 3 or q.shape[2] != dk or tuple(out.shape) != (n, H, dv) or q.stride(2) != 1 or out.stride(2) != 1:
        raise ValueError("q must be [n, H, dk] and out [n, H, dv] with contiguous last dimensions")
    if out.dtype not in (q.dtype, torch.float32) or k_pool.dtype != q.dtype or v_pool.dtype != q.dtype:
        raise TypeError("q and the pools share one dtype; out has it too, or is fp32")
    out_f32 = int(out.dtype == torch.float32 and q.dtype != torch.float32)
    for t in (block_tables, tok_row, tok_pos):
        if t.dtype != torch.int32:
            raise TypeError("block tables, token rows and positions are int32")
    for t, shape in ((talk, (H, H)), (sink, (H,))):
        if t is not None and (t.dtype != torch.float32 or tuple(t.shape) != shape or not t.is_contiguous()):
            raise ValueError("talk is contiguous fp32 [H, H], sink fp32 [H]")
    per_channel = _gate_kind(gate, n, H, dv, q.dtype)
    rc = _lib_().b200_mixed_paged_attn_ext2(out.data_ptr(), out.stride(0), out.stride(1), q.data_ptr(), q.stride(0),
                                           q.stride(1), _ptr(gate), _rows2(gate) if gate is not None else 0, per_channel,
                                           k_pool.data_ptr(), v_pool.data_ptr(), block_tables.data_ptr(),
                                           block_tables.stride(0), tok_row.data_ptr(), tok_pos.data_ptr(), n, _ptr(talk),
                                           _ptr(sink), float(scale), float(softcap), int(window), int(keep_first),
                                           int(chunk), int(unrotate_base is not None), int(interleaved),
                                           float(unrotate_base or 0.0), H, G, dk, dv, v_row, int(value_div), out_f32, bs,
                                           DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_mixed_paged_attn")


def mixed_prompt_attention_supported(H: int, G: int, dk: int, dv: int, has_talk: bool, same_pool: bool, unrotate: bool,
                                     dtype: torch.dtype) -> bool:
    return bool(_lib_().b200_mixed_prompt_attn_supported(int(H), int(G), int(dk), int(dv), int(has_talk), int(same_pool),
                                                         int(unrotate), DTYPE_ID[dtype]))


def heads_as_rows_supported(H: int, dk: int, dv: int, dtype: torch.dtype) -> bool:
    """Whether ``mixed_prompt_attention(heads_as_rows=True)`` takes ``H`` heads over one kv head."""
    return bool(_lib_().b200_mixed_prompt_attn_rows_supported(int(H), int(dk), int(dv), DTYPE_ID[dtype]))


PROMPT_TILE_TOKENS = 16     # tokens of one sequence a CTA of ``mixed_prompt_attention`` serves


@_timed
def mixed_prompt_attention(out: torch.Tensor, q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor,
                           block_tables: torch.Tensor, tiles: torch.Tensor, tok_pos: torch.Tensor, scale: float,
                           talk: Optional[torch.Tensor] = None, sink: Optional[torch.Tensor] = None, window: int = 0,
                           keep_first: int = 0, value_rot: Optional[torch.Tensor] = None, interleaved: bool = False,
                           gate: Optional[torch.Tensor] = None, max_context: int = 0, softcap: float = 0.0,
                           chunk: int = 0, value_width: Optional[int] = None, value_div: int = 1,
                           heads_as_rows: bool = False, max_tile_tokens: int = PROMPT_TILE_TOKENS) -> None:
    """``mixed_paged_attention`` on the tensor cores for prompt portions and decoded tokens alike (16-bit dtypes, see
    ``mixed_prompt_attention_supported``).  ``tiles`` int32 ``[n_tiles, 3]``: up to ``PROMPT_TILE_TOKENS`` consecutive
    tokens of one sequence each (``max_tile_tokens`` bounds them); only their rows of ``out`` are written; ``value_rot``: the table
    ``rotary_kv_append`` returned for this step's tokens; ``max_context``: the longest context of the tiles (a hint: few tokens
    over long contexts divide the keys over several CTAs and merge); ``chunk``, ``value_width`` and ``value_div`` as in
    ``mixed_paged_attention``, as are the kinds of ``gate``.  ``heads_as_rows`` (steps of single tokens over one kv head,
    no talk / value_rot; see ``heads_as_rows_supported``): the 16 rows of a tensor-core tile are 16 query heads of one token
    instead of 16 tokens of one head."""
    _need_cuda(out, q, k_pool, v_pool, block_tables, tiles, tok_pos)
    nb, G, bs, dk = k_pool.shape
    dv, v_row = _value_layout(k_pool, v_pool, value_width, value_div)
    n, H = q.shape[0], q.shape[1]
    if q.dim() != 3 or q.shape[2] != dk or tuple(out.shape) != (n, H, dv) or q.stride(2) != 1 or out.stride(2) != 1:
        raise ValueError("q must be [n, H, dk] and out [n, H, dv] with contiguous last dimensions")
    if out.dtype not in (q.dtype, torch.float32) or k_pool.dtype != q.dtype or v_pool.dtype != q.dtype:
        raise TypeError("q and the pools share one dtype; out has it too, or is fp32")
    out_f32 = int(out.dtype == torch.float32 and q.dtype != torch.float32)
    if tiles.dtype != torch.int32 or tiles.dim() != 2 or tiles.shape[1] != 3 or not tiles.is_contiguous():
        raise ValueError("tiles must be contiguous int32 [n_tiles, 3]")
    for t, shape in ((talk, (H, H)), (sink, (H,))):
        if t is not None and (t.dtype != torch.float32 or tuple(t.shape) != shape or not t.is_contiguous()):
            raise ValueError("talk is contiguous fp32 [H, H], sink fp32 [H]")
    if value_rot is not None and (tuple(value_rot.shape) != (n, dv // 2, 2) or value_rot.dtype != torch.float32
                                  or not value_rot.is_contiguous()):
        raise ValueError("value_rot must be contiguous fp32 [n, dv // 2, 2]")
    per_channel = _gate_kind(gate, n, H, dv, q.dtype)
    if heads_as_rows and (G != 1 or talk is not None or value_rot is not None):
        raise ValueError("heads_as_rows needs one kv head and no talk or value_rot")
    if not 1 <= max_tile_tokens <= PROMPT_TILE_TOKENS:
        raise ValueError(f"tiles have 1 to {PROMPT_TILE_TOKENS} tokens")
    if heads_as_rows:
        max_tile_tokens = 1
    lib = _lib_()
    seen = min(max_context, window + keep_first + PROMPT_TILE_TOKENS) if window > 0 else max_context
    if chunk > 0:
        seen = min(seen, chunk + PROMPT_TILE_TOKENS)
    splits = lib.b200_mixed_prompt_attn_splits(tiles.shape[0], (seen + 31) // 32, (H + 15) // 16 if heads_as_rows else H, G,
                                               dk, dv, int(talk is not None),
                                               int(k_pool.data_ptr() == v_pool.data_ptr()), int(value_rot is not None),
                                               DTYPE_ID[q.dtype]) if max_context > 0 else 1
    ws = None
    if splits > 1:
        ws = torch.empty(lib.b200_mixed_prompt_attn_workspace(splits, tiles.shape[0] * max_tile_tokens, H, dv) // 4, dtype=torch.float32,
                         device=q.device)
    rc = lib.b200_mixed_prompt_attn_ext3(out.data_ptr(), out.stride(0), out.stride(1), q.data_ptr(), q.stride(0),
                                        q.stride(1), _ptr(gate), _rows2(gate) if gate is not None else 0, per_channel, k_pool.data_ptr(),
                                        v_pool.data_ptr(), block_tables.data_ptr(), block_tables.stride(0),
                                        tiles.data_ptr(), tiles.shape[0], int(max_tile_tokens), tok_pos.data_ptr(), n, _ptr(talk), _ptr(sink),
                                        float(scale), float(softcap), int(window), int(keep_first), int(chunk),
                                        _ptr(value_rot), int(interleaved), H, G, dk, dv, v_row, int(value_div),
                                        int(heads_as_rows), out_f32, bs, int(splits), _ptr(ws), DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_mixed_prompt_attn")


def tile_rows(H: int, G: int, dk: int, n_tokens: int, heavy: bool = False, page: int = 16) -> int:
    """Query rows (tokens x heads of a kv group) of a ``tile_attention`` tile for portions of ``n_tokens`` tokens in all (``heavy``: with
    distance biases or a soft cap) over pages of ``page`` tokens."""
    by_row = 2 if page % 8 or 64 % page else 0      # pages that the copy engine cannot fetch whole
    return int(_lib_().b200_tile_attn_rows_ext(H // G, int(G), int(dk), int(n_tokens), int(heavy) | by_row))


def tile_attention_supported(H: int, G: int, dk: int, dv: int, same_pool: bool, bias: bool, dtype: torch.dtype) -> bool:
    """Whether ``tile_attention`` serves this head layout (aligned query rows are checked per call)."""
    return bool(_lib_().b200_tile_attn_supported(int(H), int(G), int(dk), int(dv), int(same_pool), int(bias), DTYPE_ID[dtype]))


def tile_attention_from(H: int, G: int, bias: bool = False) -> int:
    """Tokens from which a portion goes to ``tile_attention``.  Most of the 128 rows of a product are padding for a few tokens, but the walk
    is as long as one of the 16-row kernels and divides the keys over CTAs.  Without biases: from two tokens and 8 rows (tokens x heads of
    a kv group) on (B200, 16 heads over 4, two tokens per sequence, 16-row kernel against tile: 8 sequences at 500 32 and 21 us, at 2000 55
    and 37; 48 sequences at 2000 177 and 79).  With biases the 16-row kernel divides the keys of its 16 rows over CTAs too and starts sooner,
    so that it keeps them (as above: 8 sequences at 100 10 and 12 us, at 2000 23 and 42; 48 at 2000 85 and 113; from 17 rows on 145 and 46),
    except where every head has its own keys (12 over 12, 8 sequences at 100: 15 and 11; 48 at 2000: 363 and 210)."""
    rep = H // G
    return 16 // rep + 1 if bias and rep > 1 else max(2, 8 // rep)


# A portion of up to 16 tokens whose context is up to 32 keys is one step of the 16-row kernel's walk; the tile kernel's fixed beginning (tensor
# memory, more warps, more shared memory) is hidden while an SM holds one or two of its CTAs.  B200, 16-row against tile, 8 tokens
# each: 16 heads over 4, 20 sequences 7.6 and 7.1 us, 40: 7.7 and 8.9, 160: 15.6 and 20.3; 16 over 16, 12 sequences 11.2 and 8.9, 40: 11.4
# and 20.0.  With more heads per kv head, or one kv head, the tile kernel has as few CTAs and stays level or ahead: 16 over 2, 200 sequences
# 14.7 and 15.1; 16 over 1 19.1 and 11.2; latent 320 of 16 heads 34.9 and 25.9.
TINY_TOKENS, TINY_CONTEXT = 16, 32


def tiny_to_tiles(n_portions: int, H: int, G: int) -> bool:
    """Whether ``n_portions`` of up to ``TINY_TOKENS`` tokens and ``TINY_CONTEXT`` keys still go to ``tile_attention``."""
    rep = H // G
    return G == 1 or rep > 4 or n_portions * G <= (148 if rep > 2 else 296)


@_timed
def tile_attention(out: torch.Tensor, q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, block_tables: torch.Tensor,
                   tiles: torch.Tensor, tok_pos: torch.Tensor, scale: float, sink: Optional[torch.Tensor] = None, window: int = 0,
                   keep_first: int = 0, gate: Optional[torch.Tensor] = None, max_context: int = 0, softcap: float = 0.0, chunk: int = 0,
                   value_width: Optional[int] = None, value_div: int = 1, bias_lut: Optional[torch.Tensor] = None,
                   temp_coef: float = 0.0, temp_every: int = 1, rows: int = 128) -> None:
    """``mixed_prompt_attention`` (or, with ``bias_lut``, ``biased_prompt_attention``) for prompt portions in tiles of up to
    ``rows`` rows (see ``tile_rows``): ``tiles`` int32 ``[n_tiles, 3]`` with up to ``rows // (H // G)`` consecutive tokens of one sequence each.
    Only the tiles' rows of ``out`` are written, so the other portions of a step may go through another kernel."""
    _need_cuda(out, q, k_pool, v_pool, block_tables, tiles, tok_pos)
    nb, G, bs, dk = k_pool.shape
    dv, v_row = _value_layout(k_pool, v_pool, value_width, value_div)
    n, H = q.shape[0], q.shape[1]
    if q.dim() != 3 or q.shape[2] != dk or tuple(out.shape) != (n, H, dv) or q.stride(2) != 1 or out.stride(2) != 1:
        raise ValueError("q must be [n, H, dk] and out [n, H, dv] with contiguous last dimensions")
    if out.dtype not in (q.dtype, torch.float32) or k_pool.dtype != q.dtype or v_pool.dtype != q.dtype:
        raise TypeError("q and the pools share one dtype; out has it too, or is fp32")
    if tiles.dtype != torch.int32 or tiles.dim() != 2 or tiles.shape[1] != 3 or not tiles.is_contiguous():
        raise ValueError("tiles must be contiguous int32 [n_tiles, 3]")
    if block_tables.dtype != torch.int32 or tok_pos.dtype != torch.int32:
        raise TypeError("block tables and positions are int32")
    if sink is not None and (sink.dtype != torch.float32 or tuple(sink.shape) != (H,) or not sink.is_contiguous()):
        raise ValueError("sink is contiguous fp32 [H]")
    if bias_lut is not None and (bias_lut.dtype != torch.float32 or bias_lut.shape[0] != H or not bias_lut.is_contiguous()):
        raise ValueError("bias_lut must be contiguous fp32 [H, L]")
    per_channel = _gate_kind(gate, n, H, dv, q.dtype)
    lib = _lib_()
    seen = min(max_context, window + keep_first + 128) if window > 0 else max_context
    if chunk > 0:
        seen = min(seen, chunk + 128)
    n_tiles, rows = tiles.shape[0], int(rows)
    splits = lib.b200_tile_attn_splits_ext(n_tiles, (seen + 63) // 64, G, dk, rows, n * H) if max_context > 0 else 1
    if H * dv * 4 > 227 * 1024:     # more than the merge of splits holds
        splits = 1
    ws = torch.empty((splits, n_tiles * (rows // (H // G)), H, dv + 2), dtype=torch.float32, device=q.device) if splits > 1 else None
    rc = lib.b200_tile_attn(out.data_ptr(), out.stride(0), out.stride(1), q.data_ptr(), q.stride(0), q.stride(1), _ptr(gate),
                            _rows2(gate) if gate is not None else 0, per_channel, k_pool.data_ptr(), v_pool.data_ptr(),
                            block_tables.data_ptr(), block_tables.stride(0), tiles.data_ptr(), n_tiles, rows, tok_pos.data_ptr(),
                            _ptr(sink), _ptr(bias_lut), bias_lut.shape[1] if bias_lut is not None else 0, float(scale), float(softcap),
                            float(temp_coef), int(temp_every), int(window), int(keep_first), int(chunk), H, G, dk, dv, v_row,
                            int(value_div), int(out.dtype == torch.float32), bs, int(splits), _ptr(ws), DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_tile_attn")


@_timed
def causal_conv_silu(x: torch.Tensor, weight: torch.Tensor, tail: torch.Tensor, seqs: torch.Tensor,
                     max_count: int, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Short causal convolution per channel over each sequence's tokens (plus ``bias [C]``), then SiLU.  ``x [n, C]`` (a
    column slice is fine), ``weight [C, taps]`` (last column = the current token), ``tail`` fp32 ``[slots, taps - 1, C]``
    carries each live sequence's last inputs between steps and is updated."""
    _need_cuda(x, weight, tail, seqs)
    C, taps = weight.shape
    if x.shape[1] != C or tail.dtype != torch.float32 or tuple(tail.shape[1:]) != (taps - 1, C) or not tail.is_contiguous():
        raise ValueError("x [n, C], weight [C, taps], tail fp32 [slots, taps - 1, C]")
    if seqs.dtype != torch.int32 or seqs.dim() != 2 or seqs.shape[1] != 4 or not seqs.is_contiguous():
        raise ValueError("seqs must be contiguous int32 [n_seqs, 4]")
    if bias is not None and (bias.numel() != C or bias.dtype != x.dtype or not bias.is_contiguous()):
        raise ValueError("bias is contiguous [C] in the activations' dtype")
    if weight.dtype != x.dtype or not weight.is_contiguous():
        raise ValueError("weight is contiguous [C, taps] in the activations' dtype")
    out = torch.empty((x.shape[0], C), dtype=x.dtype, device=x.device)
    rc = _lib_().b200_causal_conv_silu_ext(out.data_ptr(), C, x.data_ptr(), _rows2(x), weight.data_ptr(), _ptr(bias),
                                           tail.data_ptr(), seqs.data_ptr(), seqs.shape[0], int(max_count), C, taps,
                                           DTYPE_ID[x.dtype], _stream())
    _lib.check_mixers(rc, "b200_causal_conv_silu")
    return out


@_timed
def delta_scan(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, beta_logit: torch.Tensor, a_logit: torch.Tensor,
               dt_bias: torch.Tensor, a_log: torch.Tensor, state: torch.Tensor, seqs: torch.Tensor, G: int,
               unit_eps: float, q_scale: float, max_count: int = 0) -> torch.Tensor:
    """Gated delta rule with a decay per key channel (``a_logit [n, H*dk]``, ``dt_bias [H*dk]``) or per head (``[n, H]``,
    ``[H]``) over each sequence's tokens; ``state`` fp32 ``[slots, H, dk, dv]``
    is read (unless the sequence is fresh) and written back.  ``q / k [n, G*dk]`` and ``v [n, H*dv]`` are column
    slices of ONE tensor (same row stride), ``beta_logit [n, H]``.  Returns fp32 ``[n, H, dv]``.  ``max_count``: the
    largest token count in ``seqs`` (0: unknown), picks the kernel.  One decay per head: steps of single tokens, and bf16 steps with a
    portion of ``CHUNK_SCAN_FROM`` tokens or more in chunks of 64 on the tensor cores; otherwise, 16-bit steps with long
    portions (``split_scan_pays``) and keys of up to 64 in chunks of 16 at fp32 precision; others token by token."""
    _need_cuda(q, k, v, beta_logit, a_logit, dt_bias, a_log, state, seqs)
    n = q.shape[0]
    _, H, dk, dv = state.shape
    if q.shape[1] != G * dk or k.shape != q.shape or v.shape != (n, H * dv) or beta_logit.shape != (n, H) \
            or a_log.numel() != H or (tuple(a_logit.shape), dt_bias.numel()) not in (((n, H * dk), H * dk), ((n, H), H)):
        raise ValueError("inputs do not match the state's shape")
    if any(t.dtype != q.dtype for t in (k, v, beta_logit, a_logit, dt_bias, a_log)):
        raise TypeError("inputs and constants share one dtype")
    stride = _rows2(q)
    if n > 1 and (k.stride(0) != stride or v.stride(0) != stride):
        raise ValueError("q, k and v must share a row stride")
    if state.dtype != torch.float32 or not state.is_contiguous():
        raise TypeError("the recurrent state is contiguous fp32")
    if seqs.dtype != torch.int32 or seqs.dim() != 2 or seqs.shape[1] != 4 or not seqs.is_contiguous():
        raise ValueError("seqs must be contiguous int32 [n_seqs, 4]")
    o = torch.empty((n, H, dv), dtype=torch.float32, device=q.device)
    lib, dt, n_seqs = _lib_(), DTYPE_ID[q.dtype], seqs.shape[0]
    head = (o.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), stride, beta_logit.data_ptr(), _rows2(beta_logit),
            a_logit.data_ptr(), _rows2(a_logit), dt_bias.data_ptr(), a_log.data_ptr())
    tail = (H, G, dk, dv, float(unit_eps), float(q_scale))
    one_decay = a_logit.shape[1] == H
    if one_decay and max_count == 1 and n_seqs == n:
        rc = lib.b200_delta_step(*head, state.data_ptr(), seqs.data_ptr(), n_seqs, *tail, dt, _stream())
        _lib.check_mixers(rc, "b200_delta_step")
    elif one_decay and max_count >= CHUNK_SCAN_FROM and lib.b200_delta_chunk_scan_supported(dk, dv, dt):
        ws = torch.empty(lib.b200_delta_chunk_workspace(n, n_seqs, H), dtype=torch.uint8, device=q.device)
        rc = lib.b200_delta_chunk_scan(*head, state.data_ptr(), seqs.data_ptr(), n_seqs, int(max_count), *tail, ws.data_ptr(), dt,
                                       _stream())
        _lib.check_mixers(rc, "b200_delta_chunk_scan")
    elif not (split_scan_takes(1, max_count, n, n_seqs, H, dk, dv, q.dtype) and _split_scan(
            1, o, q, k, v, stride, (beta_logit, _rows2(beta_logit)), (a_logit, _rows2(a_logit)), dt_bias, a_log, None, not one_decay,
            state, seqs, G, unit_eps, q_scale)):
        rc = lib.b200_delta_scan_ext(*head, int(not one_decay), state.data_ptr(), seqs.data_ptr(), n_seqs, *tail, dt, _stream())
        _lib.check_mixers(rc, "b200_delta_scan")
    return o


@_timed
def head_rmsnorm_gated(x: torch.Tensor, weight: torch.Tensor, gate: Optional[torch.Tensor], eps: float) -> torch.Tensor:
    """fp32 ``[n, H, dv]`` -> ``x * rsqrt(mean(x^2) + eps) * weight * sigmoid(gate)`` as ``[n, H*dv]`` in the weight's
    dtype; ``gate [n, H*dv]`` holds logits."""
    _need_cuda(x, weight)
    n, H, dv = x.shape
    if x.dtype != torch.float32 or not x.is_contiguous() or weight.numel() != dv:
        raise ValueError("x must be contiguous fp32 [n, H, dv] and weight [dv]")
    if gate is not None and (tuple(gate.shape) != (n, H * dv) or gate.dtype != weight.dtype):
        raise ValueError("gate must be [n, H*dv] in the weight's dtype")
    out = torch.empty((n, H * dv), dtype=weight.dtype, device=x.device)
    rc = _lib_().b200_head_rmsnorm_gated(out.data_ptr(), x.data_ptr(), weight.data_ptr(), _ptr(gate),
                                         _rows2(gate) if gate is not None else 0, float(eps), n, H, dv,
                                         DTYPE_ID[weight.dtype], _stream())
    _lib.check_mixers(rc, "b200_head_rmsnorm_gated")
    return out


# ---- side-by-side mixers, post-norm sublayers, grouped softmax routing (csrc/b200_parallel_ops.cu) ---------------------
def _check_seqs(seqs: torch.Tensor) -> None:
    if seqs.dtype != torch.int32 or seqs.dim() != 2 or seqs.shape[1] != 4 or not seqs.is_contiguous():
        raise ValueError("seqs must be contiguous int32 [n_seqs, 4]")


@_timed
def qknorm_rotary_append(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, q_norm: Optional[torch.Tensor],
                         k_norm: Optional[torch.Tensor], eps: float, freqs: Optional[torch.Tensor], k_pool: torch.Tensor,
                         v_pool: torch.Tensor, slot_mapping: torch.Tensor, tok_pos: torch.Tensor, H: int,
                         interleaved: bool = True, unit_norm: bool = False) -> None:
    """Per-head RMS norm of q (in place) and k (weights ``[dk]``; None: no norm, or with ``unit_norm`` a norm without a
    weight, which a rotation leaves as it is), rotary positions over the first
    ``2 * len(freqs)`` dimensions of every head with angle ``pos * freqs[i]`` (``freqs`` float64 on the device), k and v
    stored in the pools at ``slot_mapping``.  ``v_pool`` may hold fewer heads than ``k_pool`` (several score maps over the
    same values)."""
    _need_cuda(q, k, v, k_pool, v_pool, slot_mapping, tok_pos)
    nb, G, bs, dk = k_pool.shape
    Gv, dv = v_pool.shape[1], v_pool.shape[3]
    n = q.shape[0]
    if q.shape[1] != H * dk or k.shape != (n, G * dk) or v.shape != (n, Gv * dv) or v_pool.shape[0] != nb \
            or v_pool.shape[2] != bs:
        raise ValueError("q / k / v do not match the pools")
    if slot_mapping.dtype != torch.int64 or tok_pos.dtype != torch.int32:
        raise TypeError("slot_mapping is int64, tok_pos int32")
    for w in (q_norm, k_norm):
        if w is not None and (w.numel() != dk or w.dtype != q.dtype or not w.is_contiguous()):
            raise ValueError("norm weights are contiguous [dk] in the activations' dtype")
    rot_dims = 0
    if freqs is not None:
        if freqs.dtype != torch.float64 or not freqs.is_contiguous() or not freqs.is_cuda:
            raise ValueError("freqs is a contiguous float64 tensor on the device")
        rot_dims = 2 * freqs.numel()
    rc = _lib_().b200_qknorm_rotary_append_ext2(q.data_ptr(), _rows2(q), k.data_ptr(), _rows2(k), v.data_ptr(), _rows2(v),
                                               _ptr(q_norm), _ptr(k_norm), int(unit_norm), float(eps), _ptr(freqs), rot_dims,
                                               int(interleaved), k_pool.data_ptr(), v_pool.data_ptr(),
                                               slot_mapping.data_ptr(), tok_pos.data_ptr(), n, H, G, Gv, dk, dv, bs, nb,
                                               DTYPE_ID[k_pool.dtype], _stream())
    _lib.check_mixers(rc, "b200_qknorm_rotary_append")


@_timed
def retention_scan(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, decay: torch.Tensor, k_scale: float,
                   state: torch.Tensor, seqs: torch.Tensor, plan=None, max_count: int = 0) -> torch.Tensor:
    """Fixed-decay linear attention over each sequence's tokens: ``S <- decay[h] S + (k_scale k) v^T``, ``o = S^T q``;
    ``state`` fp32 ``[slots, H, dk, dv]`` is read (unless the sequence is fresh) and written back.  ``q / k [n, H*dk]``
    and ``v [n, H*dv]`` are column slices of ONE tensor.  Returns fp32 ``[n, H, dv]``.

    ``plan`` (``RaggedBatchState.scan_plan()``; None: every sequence runs token by token in one launch) names the long
    portions of the step as parallel segments: each segment runs as a fresh sequence against a scratch state, one launch
    chains the segments' end states into the state at every segment's start and the sequence's final state, and one adds
    what each token missed, ``decay^(t - t0 + 1) P^T q_t``.  Short sequences of the same step run as before.  Without a plan, ``max_count``
    (the largest token count in ``seqs``, 0: unknown) picks the kernel as in ``gated_scan``."""
    _need_cuda(q, k, v, decay, state, seqs)
    n = q.shape[0]
    _, H, dk, dv = state.shape
    if q.shape[1] != H * dk or k.shape != q.shape or v.shape != (n, H * dv):
        raise ValueError("projections do not match the state's shape")
    stride = _rows2(q)
    if n > 1 and (k.stride(0) != stride or v.stride(0) != stride):
        raise ValueError("q, k and v must share a row stride")
    if state.dtype != torch.float32 or not state.is_contiguous():
        raise TypeError("the recurrent state is contiguous fp32")
    if decay.dtype != torch.float32 or decay.numel() != H or not decay.is_contiguous():
        raise ValueError("decay is contiguous fp32 [H]")
    _check_seqs(seqs)
    o = torch.empty((n, H, dv), dtype=torch.float32, device=q.device)
    if plan is None and split_scan_takes(2, max_count, n, seqs.shape[0], H, dk, dv, q.dtype) and _split_scan(
            2, o, q, k, v, stride, (None, 0), (None, 0), None, None, decay, False, state, seqs, H, 0.0, k_scale, max_count):
        return o
    lib, dt, st = _lib_(), DTYPE_ID[q.dtype], _stream()

    def scan(into: torch.Tensor, table: torch.Tensor) -> None:
        rc = lib.b200_retention_scan(o.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), stride, decay.data_ptr(),
                                     float(k_scale), into.data_ptr(), table.data_ptr(), table.shape[0], H, dk, dv, dt, st)
        _lib.check_mixers(rc, "b200_retention_scan")

    if plan is None:
        scan(state, seqs)
        return o
    if plan.direct is not None:
        scan(state, plan.direct)
    seg_state = torch.empty((plan.segs.shape[0], H, dk, dv), dtype=torch.float32, device=q.device)
    scan(seg_state, plan.segs)
    rc = lib.b200_retention_carry(state.data_ptr(), seg_state.data_ptr(), plan.parents.data_ptr(), plan.parents.shape[0],
                                  plan.segs.data_ptr(), decay.data_ptr(), H, dk, dv, st)
    _lib.check_mixers(rc, "b200_retention_carry")
    rc = lib.b200_retention_apply_carry(o.data_ptr(), q.data_ptr(), stride, seg_state.data_ptr(), plan.segs.data_ptr(),
                                        plan.segs.shape[0], decay.data_ptr(), H, dk, dv, dt, st)
    _lib.check_mixers(rc, "b200_retention_apply_carry")
    return o


@_timed
def head_norm_act_gate(x: torch.Tensor, weight: Optional[torch.Tensor], gate: Optional[torch.Tensor], eps: float,
                       dtype: torch.dtype, gate_act: str = "silu", out_scale: float = 1.0,
                       out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """fp32 ``[n, H, dv]`` -> ``x * rsqrt(mean(x^2) + eps) [* weight] * act(gate) * out_scale`` as ``[n, H*dv]`` in
    ``dtype``; ``gate [n, H*dv]`` holds pre-activations, ``gate_act`` is ``"sigmoid"`` or ``"silu"``; ``out`` may be a
    column slice of a wider buffer."""
    _need_cuda(x)
    n, H, dv = x.shape
    if x.dtype != torch.float32 or not x.is_contiguous():
        raise ValueError("x must be contiguous fp32 [n, H, dv]")
    if weight is not None and (weight.numel() != dv or weight.dtype != dtype):
        raise ValueError("weight must be [dv] in the output dtype")
    if gate is not None and (tuple(gate.shape) != (n, H * dv) or gate.dtype != dtype):
        raise ValueError("gate must be [n, H*dv] in the output dtype")
    if out is None:
        out = torch.empty((n, H * dv), dtype=dtype, device=x.device)
    elif tuple(out.shape) != (n, H * dv) or out.dtype != dtype:
        raise ValueError("out must be [n, H*dv] in the output dtype")
    rc = _lib_().b200_head_norm_act_gate(out.data_ptr(), _rows2(out), x.data_ptr(), _ptr(weight), _ptr(gate),
                                         _rows2(gate) if gate is not None else 0, {"sigmoid": 0, "silu": 1}[gate_act],
                                         float(out_scale), float(eps), n, H, dv, DTYPE_ID[dtype], _stream())
    _lib.check_mixers(rc, "b200_head_norm_act_gate")
    return out


@_timed
def branch_postnorm_residual(x: torch.Tensor, a: torch.Tensor, sa: float, b: Optional[torch.Tensor], sb: float,
                             w_norm: torch.Tensor, layer_scale: Optional[torch.Tensor], eps: float,
                             want_copy: bool = True) -> Optional[torch.Tensor]:
    """In place ``x += layer_scale * w_norm * y * rsqrt(mean(y^2) + eps)`` with ``y = sa a + sb b`` on the fp32 residual;
    ``a`` is fp32 or of the weights' dtype, ``b`` (optional) of the weights' dtype.  With ``want_copy`` returns the new
    ``x`` in the weights' dtype (what sublayers that read the residual itself take as GEMM input)."""
    _need_cuda(x, a, w_norm)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or a.shape != x.shape:
        raise ValueError("x must be contiguous fp32 [rows, width] and the branches of the same shape")
    T = w_norm.dtype
    if a.dtype not in (T, torch.float32) or (b is not None and (b.dtype != T or b.shape != x.shape)):
        raise TypeError("a is fp32 or of the weights' dtype, b of the weights' dtype")
    if layer_scale is not None and (layer_scale.dtype != T or layer_scale.numel() != x.shape[1]):
        raise ValueError("layer_scale must be [width] in the weights' dtype")
    out = torch.empty(x.shape, dtype=T, device=x.device) if want_copy else None
    rc = _lib_().b200_branch_postnorm_residual(x.data_ptr(), a.data_ptr(), _rows2(a), int(a.dtype == torch.float32 and
                                               T != torch.float32), float(sa), _ptr(b), _rows2(b) if b is not None else 0,
                                               float(sb), w_norm.data_ptr(), _ptr(layer_scale), _ptr(out), float(eps),
                                               x.shape[0], x.shape[1], DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_branch_postnorm_residual")
    return out


@_timed
def cast_rows(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """Contiguous fp32 tensor -> the same numbers in ``dtype``."""
    _need_cuda(x)
    if x.dtype != torch.float32 or not x.is_contiguous():
        raise ValueError("x must be contiguous fp32")
    out = torch.empty(x.shape, dtype=dtype, device=x.device)
    rc = _lib_().b200_cast_rows(out.data_ptr(), x.data_ptr(), x.numel(), DTYPE_ID[dtype], _stream())
    _lib.check_mixers(rc, "b200_cast_rows")
    return out


@_timed
def softmax_group_topk(logits: torch.Tensor, correction: Optional[torch.Tensor], top: int, groups: int = 1,
                       keep: int = 1, sum_floor: float = 0.0):
    """fp32 ``[n, E]`` router logits -> ``(ids int32 [n, top], weights fp32 [n, top])``: softmax scores, the choice by
    score + ``correction`` inside the ``keep`` best of ``groups`` expert groups, weights = chosen scores over (their
    sum + ``sum_floor``)."""
    _need_cuda(logits)
    if logits.dtype != torch.float32 or not logits.is_contiguous() or logits.dim() != 2:
        raise ValueError("router logits are contiguous fp32 [n, E]")
    n, E = logits.shape
    if correction is not None and (correction.dtype != torch.float32 or correction.numel() != E
                                   or not correction.is_contiguous()):
        raise ValueError("correction is contiguous fp32 [E]")
    ids = torch.empty((n, top), dtype=torch.int32, device=logits.device)
    w = torch.empty((n, top), dtype=torch.float32, device=logits.device)
    rc = _lib_().b200_softmax_group_topk(ids.data_ptr(), w.data_ptr(), logits.data_ptr(), _ptr(correction),
                                         float(sum_floor), n, E, int(top), int(groups), int(keep), _stream())
    _lib.check_mixers(rc, "b200_softmax_group_topk")
    return ids, w


@_timed
def gather_rows(h: torch.Tensor, src: torch.Tensor, top: int) -> torch.Tensor:
    """``xs[r] = h[src[r] // top]``: rows in expert order."""
    _need_cuda(h, src)
    if not h.is_contiguous() or src.dtype != torch.int64:
        raise ValueError("h contiguous, src int64")
    xs = torch.empty((src.numel(), h.shape[1]), dtype=h.dtype, device=h.device)
    rc = _lib_().b200_gather_rows(xs.data_ptr(), h.data_ptr(), src.data_ptr(), src.numel(), int(top), h.shape[1],
                                  DTYPE_ID[h.dtype], _stream())
    _lib.check_mixers(rc, "b200_gather_rows")
    return xs


@_timed
def weighted_expert_combine(ys: torch.Tensor, where: torch.Tensor, ids: torch.Tensor, weights: torch.Tensor,
                            x_self: torch.Tensor, shared: Optional[torch.Tensor], n_real: int) -> torch.Tensor:
    """fp32 ``[n, width]``: ``sum_k weights[n, k] * (ys[where[n*top + k]] if ids[n, k] < n_real else x_self[n])`` plus
    ``shared[n]`` when given.  ``x_self`` is the fp32 row an identity expert returns."""
    _need_cuda(ys, where, ids, weights, x_self)
    n, top = ids.shape
    width = x_self.shape[1]
    if not ys.is_contiguous() or ys.shape[1] != width or where.dtype != torch.int64 or where.numel() != n * top:
        raise ValueError("ys contiguous [rows, width], where int64 [n * top]")
    if ids.dtype != torch.int32 or weights.dtype != torch.float32 or not ids.is_contiguous() or not weights.is_contiguous():
        raise ValueError("ids int32 and weights fp32, contiguous [n, top]")
    if x_self.dtype != torch.float32 or not x_self.is_contiguous() or x_self.shape[0] != n:
        raise ValueError("x_self is contiguous fp32 [n, width]")
    if shared is not None and (shared.shape != x_self.shape or shared.dtype != ys.dtype or not shared.is_contiguous()):
        raise ValueError("shared rows are contiguous [n, width] in the experts' dtype")
    out = torch.empty((n, width), dtype=torch.float32, device=ys.device)
    rc = _lib_().b200_weighted_expert_combine(out.data_ptr(), ys.data_ptr(), where.data_ptr(), ids.data_ptr(),
                                              weights.data_ptr(), x_self.data_ptr(), _ptr(shared), n, top, int(n_real),
                                              width, DTYPE_ID[ys.dtype], _stream())
    _lib.check_mixers(rc, "b200_weighted_expert_combine")
    return out


# ---- token shift, sigmoid-gated post-norm sublayers, a decoupled rotated key part (csrc/b200_gated_ops.cu) -----------
@_timed
def token_shift(x: torch.Tensor, mu: torch.Tensor, state: torch.Tensor, seqs: torch.Tensor, max_count: int,
                want_cast: bool = False):
    """``out[t] = x[t] + (x[t - 1] - x[t]) * mu`` per channel over each sequence's tokens, in ``mu``'s dtype; the row before
    a portion comes from ``state`` fp32 ``[slots, width]`` (zero for a fresh sequence), which then receives the portion's
    last row.  Returns ``(out, x rounded to that dtype or None)``."""
    _need_cuda(x, mu, state, seqs)
    _check_seqs(seqs)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2:
        raise ValueError("x must be contiguous fp32 [rows, width]")
    n, W = x.shape
    if mu.numel() != W or not mu.is_contiguous():
        raise ValueError("mu is contiguous [width]")
    if state.dtype != torch.float32 or state.dim() != 2 or state.shape[1] != W or not state.is_contiguous():
        raise ValueError("state is contiguous fp32 [slots, width]")
    T = mu.dtype
    out = torch.empty((n, W), dtype=T, device=x.device)
    cast = torch.empty((n, W), dtype=T, device=x.device) if want_cast else None
    rc = _lib_().b200_token_shift(out.data_ptr(), W, _ptr(cast), x.data_ptr(), mu.data_ptr(), state.data_ptr(),
                                  seqs.data_ptr(), seqs.shape[0], int(max_count), W, DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_token_shift")
    return out, cast


@_timed
def latent_rotary_append(q_rot: torch.Tensor, q_out: torch.Tensor, dkv: torch.Tensor, c_norm: torch.Tensor, eps: float,
                         freqs: Optional[torch.Tensor], gain: float, pool: torch.Tensor, slot_mapping: torch.Tensor,
                         tok_pos: torch.Tensor, interleaved: bool = True) -> None:
    """``dkv [n, rank + dr]``: its first ``rank = len(c_norm)`` columns RMS-normed with ``c_norm`` and its last ``dr``
    turned by the position go to one row of the one-head ``pool [blocks, 1, bs, rank + dr]``; ``q_out[n, h, :] =
    turn(q_rot[n, h, :])`` for 3-D views ``[n, H, dr]`` with contiguous last dimensions that do not overlap.  Pairs
    ``(2i, 2i + 1)`` (``interleaved``) or ``(i, i + len(freqs))``, ``i < len(freqs)``, are turned by ``pos * freqs[i]`` with
    cos and sin times ``gain``."""
    _need_cuda(q_rot, q_out, dkv, c_norm, pool, slot_mapping, tok_pos)
    n, H, dr = q_rot.shape
    rank = c_norm.numel()
    if q_out.shape != q_rot.shape or q_rot.stride(2) != 1 or q_out.stride(2) != 1:
        raise ValueError("q_rot and q_out are [n, H, dr] views with contiguous last dimensions")
    if dkv.shape != (n, rank + dr) or pool.dim() != 4 or pool.shape[1] != 1 or pool.shape[3] != rank + dr \
            or not pool.is_contiguous():
        raise ValueError("dkv is [n, rank + dr] and the pool [blocks, 1, block size, rank + dr]")
    T = pool.dtype
    if any(t.dtype != T for t in (q_rot, q_out, dkv, c_norm)):
        raise TypeError("activations, norm weight and pool share one dtype")
    if slot_mapping.dtype != torch.int64 or tok_pos.dtype != torch.int32:
        raise TypeError("slot_mapping is int64, tok_pos int32")
    rot_dims = 0
    if freqs is not None:
        if freqs.dtype != torch.float64 or not freqs.is_contiguous() or not freqs.is_cuda:
            raise ValueError("freqs is a contiguous float64 tensor on the device")
        rot_dims = 2 * freqs.numel()
    rc = _lib_().b200_latent_rotary_append_ext(q_rot.data_ptr(), q_rot.stride(0), q_rot.stride(1), q_out.data_ptr(),
                                               q_out.stride(0), q_out.stride(1), dkv.data_ptr(), _rows2(dkv),
                                               c_norm.data_ptr(), float(eps), _ptr(freqs), float(gain), rot_dims,
                                               int(interleaved), pool.data_ptr(), slot_mapping.data_ptr(),
                                               tok_pos.data_ptr(), n, H, dr, rank, DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_latent_rotary_append")


def heads_by_token(a: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """``a [H, n, r] @ w [H, r, dv]`` per head -> ``[n, H * dv]``, a token's heads side by side: the GEMMs write them there (a
    copy behind them took 16 us at 3900 tokens of 16 heads of 128), except for one token, whose heads lie so already, and where
    ``out=`` does not go: gradients, forward-mode tangents, functorch's transforms, and autocast, which does not see it."""
    (H, n, _), dv = a.shape, w.shape[2]
    if n > 1 and not (torch.is_grad_enabled() and (a.requires_grad or w.requires_grad)) and not torch.is_autocast_enabled(a.device.type):
        o = torch.empty((n, H, dv), dtype=a.dtype, device=a.device)
        try:
            torch.bmm(a, w, out=o.transpose(0, 1))
            return o.view(n, H * dv)
        except RuntimeError:      # a tangent or a transform: refused before anything ran (looking for them first takes 4 us of the host)
            pass
    return torch.bmm(a, w).transpose(0, 1).reshape(n, H * dv)


@_timed
def head_diff_norm(a: torch.Tensor, lam: float, out_scale: float, eps: float, rep: int, dtype: Optional[torch.dtype] = None,
                   out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``a [n, 2H, dv]`` (a view with a contiguous last dimension; fp32 or the storage dtype) holds two score maps'
    outputs per head, map 1 of head ``h`` at ``(h // rep) * 2 rep + h % rep`` and map 2 ``rep`` heads further: returns
    ``[n, H * dv]`` = ``unit_rms(a1 - lam a2) * out_scale`` per head in ``dtype`` (default: ``a``'s)."""
    _need_cuda(a)
    dtype = dtype or (out.dtype if out is not None else a.dtype)
    if a.dtype not in (dtype, torch.float32):
        raise TypeError("a is fp32 or of the output's dtype")
    n, H2, dv = a.shape
    if a.stride(2) != 1 or H2 % (2 * rep):
        raise ValueError("a is [n, 2H, dv] with a contiguous last dimension, H a multiple of rep")
    H = H2 // 2
    if out is None:
        out = torch.empty((n, H * dv), dtype=dtype, device=a.device)
    rc = _lib_().b200_head_diff_norm(out.data_ptr(), _rows2(out), a.data_ptr(), a.stride(0), a.stride(1),
                                     int(a.dtype == torch.float32 and dtype != torch.float32), float(lam), float(out_scale),
                                     float(eps), n, H, int(rep), dv, DTYPE_ID[dtype], _stream())
    _lib.check_mixers(rc, "b200_head_diff_norm")
    return out


@_timed
def gated_postnorm_residual(x: torch.Tensor, a: torch.Tensor, gate: Optional[torch.Tensor], w_norm: torch.Tensor,
                            weight_offset: float, eps: float, want_copy: bool = True) -> Optional[torch.Tensor]:
    """In place ``x += (weight_offset + w_norm) * y * rsqrt(mean(y^2) + eps)`` with ``y = a * sigmoid(gate)`` on the fp32
    residual; ``a`` is fp32 or of the weights' dtype, ``gate`` (logits, optional) of the weights' dtype.  With
    ``want_copy`` returns the new ``x`` in the weights' dtype."""
    _need_cuda(x, a, w_norm)
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or a.shape != x.shape:
        raise ValueError("x must be contiguous fp32 [rows, width] and the branch of the same shape")
    T = w_norm.dtype
    if a.dtype not in (T, torch.float32) or (gate is not None and (gate.dtype != T or gate.shape != x.shape)):
        raise TypeError("a is fp32 or of the weights' dtype, the gate of the weights' dtype")
    out = torch.empty(x.shape, dtype=T, device=x.device) if want_copy else None
    rc = _lib_().b200_gated_postnorm_residual(x.data_ptr(), a.data_ptr(), _rows2(a),
                                              int(a.dtype == torch.float32 and T != torch.float32), _ptr(gate),
                                              _rows2(gate) if gate is not None else 0, w_norm.data_ptr(),
                                              float(weight_offset), _ptr(out), float(eps), x.shape[0], x.shape[1],
                                              DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_gated_postnorm_residual")
    return out


@_timed
def relu_squared(z: torch.Tensor) -> torch.Tensor:
    """``max(z, 0)^2`` of 2-D rows (a column slice is fine), contiguous out."""
    _need_cuda(z)
    out = torch.empty(z.shape, dtype=z.dtype, device=z.device)
    if z.shape[0]:
        rc = _lib_().b200_relu_squared(out.data_ptr(), z.data_ptr(), _rows2(z), z.shape[0], z.shape[1], DTYPE_ID[z.dtype],
                                       _stream())
        _lib.check_mixers(rc, "b200_relu_squared")
    return out


@_timed
def gated_table_rows(z: torch.Tensor, table: torch.Tensor, col0: int, tokens: torch.Tensor) -> torch.Tensor:
    """``gelu_tanh(z[n, c]) * table[tokens[n], col0 + c]``: ``z [n, d]``, ``table [rows, >= col0 + d]`` of the same dtype,
    ``tokens`` int64 ``[n]``."""
    _need_cuda(z, table, tokens)
    n, d = z.shape
    if table.dtype != z.dtype or table.dim() != 2 or table.stride(1) != 1 or col0 + d > table.shape[1]:
        raise ValueError("the table is 2-D in z's dtype with at least col0 + d columns")
    if tokens.dtype != torch.int64 or tokens.numel() != n or not tokens.is_contiguous():
        raise ValueError("tokens is contiguous int64 [n]")
    out = torch.empty((n, d), dtype=z.dtype, device=z.device)
    rc = _lib_().b200_gated_table_rows(out.data_ptr(), z.data_ptr(), _rows2(z), table.data_ptr(), table.stride(0), int(col0),
                                       tokens.data_ptr(), n, d, DTYPE_ID[z.dtype], _stream())
    _lib.check_mixers(rc, "b200_gated_table_rows")
    return out


@_timed
def router_logits(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x [n, width] @ w [E, width].T + bias`` in fp32: a router's logits, every sum in an order fixed by the width (a
    token's choice of experts does not depend on the rest of the step).  ``x`` may be of any storage dtype."""
    _need_cuda(x, w)
    if w.dtype != torch.float32 or x.dim() != 2 or w.dim() != 2 or x.shape[1] != w.shape[1] \
            or not x.is_contiguous() or not w.is_contiguous():
        raise ValueError("x [n, width] is contiguous and w [E, width] contiguous fp32")
    if bias is not None and (bias.dtype != torch.float32 or bias.numel() != w.shape[0] or not bias.is_contiguous()):
        raise ValueError("bias is contiguous fp32 [E]")
    out = torch.empty((x.shape[0], w.shape[0]), dtype=torch.float32, device=x.device)
    rc = _lib_().b200_router_logits_ext(out.data_ptr(), x.data_ptr(), w.data_ptr(), _ptr(bias), x.shape[0], w.shape[0],
                                        x.shape[1], DTYPE_ID[x.dtype], _stream())
    _lib.check_mixers(rc, "b200_router_logits")
    return out


def router_sigmoid_topk(x: torch.Tensor, w: torch.Tensor, top: int):
    """``sigmoid_topk(router_logits(x, w), top)``; up to eight experts in one launch, the logits not written."""
    if w.shape[0] > 8 or top > w.shape[0]:
        return sigmoid_topk(router_logits(x, w), top)
    return _router_sigmoid_topk(x, w, top)


@_timed
def _router_sigmoid_topk(x: torch.Tensor, w: torch.Tensor, top: int):
    E = w.shape[0]
    _need_cuda(x, w)
    if w.dtype != torch.float32 or x.dim() != 2 or w.dim() != 2 or x.shape[1] != w.shape[1] \
            or not x.is_contiguous() or not w.is_contiguous():
        raise ValueError("x [n, width] is contiguous and w [E, width] contiguous fp32")
    n = x.shape[0]
    ids = torch.empty((n, top), dtype=torch.int32, device=x.device)
    weights = torch.empty((n, top), dtype=torch.float32, device=x.device)
    rc = _lib_().b200_router_sigmoid_topk(ids.data_ptr(), weights.data_ptr(), x.data_ptr(), w.data_ptr(), n, E, x.shape[1], int(top),
                                          DTYPE_ID[x.dtype], _stream())
    _lib.check_mixers(rc, "b200_router_sigmoid_topk")
    return ids, weights


# ---- recurrences decayed by one number per token and head, dynamic tanh norms (csrc/b200_recurrent_ops.cu) ------------
@_timed
def sigmoid_group_topk(logits: torch.Tensor, correction: Optional[torch.Tensor], n_experts: int, top: int, groups: int = 1,
                       keep: int = 1, scale: float = 1.0):
    """fp32 logits rows (their first ``n_experts`` columns) -> ``(ids int32 [n, top], weights fp32 [n, top])``: sigmoid
    scores, the choice by score + ``correction`` inside the ``keep`` of ``groups`` expert groups whose two largest choice
    scores have the largest sum, weights = ``scale`` times the chosen scores."""
    _need_cuda(logits)
    n, E = logits.shape[0], int(n_experts)
    if logits.dtype != torch.float32 or logits.dim() != 2 or logits.shape[1] < E:
        raise ValueError("router logits are fp32 [n, >= n_experts]")
    if correction is not None and (correction.dtype != torch.float32 or correction.numel() != E
                                   or not correction.is_contiguous()):
        raise ValueError("correction is contiguous fp32 [n_experts]")
    ids = torch.empty((n, top), dtype=torch.int32, device=logits.device)
    w = torch.empty((n, top), dtype=torch.float32, device=logits.device)
    rc = _lib_().b200_group_topk(ids.data_ptr(), w.data_ptr(), logits.data_ptr(), _rows2(logits), _ptr(correction), 1, 2, 0,
                                 0.0, float(scale), n, E, int(top), int(groups), int(keep), _stream())
    _lib.check_mixers(rc, "b200_group_topk")
    return ids, w


def _check_dyn_tanh(x: torch.Tensor, w: Optional[torch.Tensor], b: Optional[torch.Tensor], T: torch.dtype) -> None:
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2:
        raise ValueError("the residual stream is a contiguous fp32 [rows, width] tensor")
    for t in (w, b):
        if t is not None and (t.dtype != T or t.numel() != x.shape[1] or not t.is_contiguous()):
            raise ValueError("norm weight and bias are contiguous [width] in one dtype")


@_timed
def residual_dyn_tanh(x: torch.Tensor, y: Optional[torch.Tensor], norm=None) -> Optional[torch.Tensor]:
    """In place ``x += y`` on the fp32 residual (``y`` fp32 or of the norm's dtype; None: no update); with ``norm = (weight,
    bias, alpha)`` returns ``tanh(alpha x) * weight + bias`` of the new residual in the weight's dtype."""
    _need_cuda(x)
    w, b, alpha = norm if norm is not None else (None, None, 0.0)
    T = w.dtype if w is not None else (y.dtype if y is not None else torch.float32)
    _check_dyn_tanh(x, w, b, T)
    if y is not None and (y.shape != x.shape or y.dtype not in (T, torch.float32)):
        raise ValueError("y has the residual's shape and is fp32 or of the norm's dtype")
    out = torch.empty(x.shape, dtype=T, device=x.device) if w is not None else None
    rc = _lib_().b200_residual_dyn_tanh(x.data_ptr(), _ptr(y), _rows2(y) if y is not None else 0,
                                        int(y is not None and y.dtype == torch.float32 and T != torch.float32), _ptr(w),
                                        _ptr(b), float(alpha), _ptr(out), x.shape[0], x.shape[1], DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_residual_dyn_tanh")
    return out


@_timed
def expert_combine_dyn_tanh(x: torch.Tensor, ys: torch.Tensor, where: torch.Tensor, weights: torch.Tensor,
                            shared: Optional[torch.Tensor], shared_gate: Optional[torch.Tensor], norm=None
                            ) -> Optional[torch.Tensor]:
    """In place ``x[n] += sum_k weights[n, k] * ys[where[n*top + k]] + sigmoid(shared_gate[n]) * shared[n]`` on the fp32
    residual; ``shared_gate`` is a 1-D fp32 view of logits (any stride, None: factor 1).  ``norm`` as in
    ``residual_dyn_tanh``."""
    _need_cuda(x, ys, where, weights)
    w, b, alpha = norm if norm is not None else (None, None, 0.0)
    T = ys.dtype
    _check_dyn_tanh(x, w, b, T)
    n, top = weights.shape
    if not ys.is_contiguous() or ys.shape[1] != x.shape[1] or where.dtype != torch.int64 or where.numel() != n * top:
        raise ValueError("ys contiguous [rows, width], where int64 [n * top]")
    if weights.dtype != torch.float32 or not weights.is_contiguous() or n != x.shape[0]:
        raise ValueError("weights contiguous fp32 [n, top]")
    if shared is not None and (shared.shape != x.shape or shared.dtype != T or not shared.is_contiguous()):
        raise ValueError("shared rows are contiguous [n, width] in the experts' dtype")
    if shared_gate is not None and (shared_gate.dtype != torch.float32 or shared_gate.dim() != 1 or shared_gate.numel() != n):
        raise ValueError("shared_gate is fp32 [n]")
    out = torch.empty(x.shape, dtype=T, device=x.device) if w is not None else None
    rc = _lib_().b200_expert_combine_dyn_tanh(x.data_ptr(), ys.data_ptr(), where.data_ptr(), weights.data_ptr(), top,
                                              _ptr(shared), _ptr(shared_gate),
                                              shared_gate.stride(0) if shared_gate is not None else 0, _ptr(w), _ptr(b),
                                              float(alpha), _ptr(out), n, x.shape[1], DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_expert_combine_dyn_tanh")
    return out


@_timed
def silu_glu(gu: torch.Tensor) -> torch.Tensor:
    """``silu(g) * u`` of contiguous rows ``g | u``."""
    _need_cuda(gu)
    if not gu.is_contiguous() or gu.dim() != 2 or gu.shape[1] % 2:
        raise ValueError("gu must be contiguous [rows, 2*ff]")
    ff = gu.shape[1] // 2
    y = torch.empty((gu.shape[0], ff), dtype=gu.dtype, device=gu.device)
    rc = _lib_().b200_silu_glu(y.data_ptr(), gu.data_ptr(), gu.shape[0], ff, DTYPE_ID[gu.dtype], _stream())
    _lib.check_mixers(rc, "b200_silu_glu")
    return y


def _f32_heads(*tensors: torch.Tensor, H: int) -> None:
    for t in tensors:
        if t is not None and (t.dtype != torch.float32 or t.numel() != H or not t.is_contiguous()):
            raise ValueError("per-head constants are contiguous fp32 [H]")


@_timed
def capped_gates(zi: torch.Tensor, zf: torch.Tensor, bias_i: torch.Tensor, bias_f: torch.Tensor, cap: float,
                 m_state: torch.Tensor, seqs: torch.Tensor):
    """Exponential gates with a soft cap and a running maximum: ``(log decay, coef, m)``, fp32 ``[n, H]`` each (see
    ``b200_capped_gates``).  ``zi / zf [n, H]`` are column slices of one projection; ``m_state`` fp32 ``[slots, H]`` carries
    the maximum and is updated."""
    _need_cuda(zi, zf, m_state, seqs)
    _check_seqs(seqs)
    n, H = zi.shape
    _f32_heads(bias_i, bias_f, H=H)
    if zf.shape != zi.shape or zf.dtype != zi.dtype or (n > 1 and zf.stride(0) != zi.stride(0)):
        raise ValueError("zi and zf are [n, H] slices with one row stride")
    if m_state.dtype != torch.float32 or m_state.shape[1:] != (H,) or not m_state.is_contiguous():
        raise ValueError("m_state is contiguous fp32 [slots, H]")
    log_decay, coef, m = torch.empty((3, n, H), dtype=torch.float32, device=zi.device).unbind(0)
    rc = _lib_().b200_capped_gates(log_decay.data_ptr(), coef.data_ptr(), m.data_ptr(), zi.data_ptr(), zf.data_ptr(), _rows2(zi),
                                   bias_i.data_ptr(), bias_f.data_ptr(), float(cap), m_state.data_ptr(), seqs.data_ptr(),
                                   seqs.shape[0], H, DTYPE_ID[zi.dtype], _stream())
    _lib.check_mixers(rc, "b200_capped_gates")
    return log_decay, coef, m


@_timed
def step_sizes(z: torch.Tensor, bias: torch.Tensor, a_log: torch.Tensor):
    """``dt = softplus(z + bias)``: ``(log decay = -exp(a_log) dt, dt)``, fp32 ``[n, H]``."""
    _need_cuda(z)
    n, H = z.shape
    _f32_heads(bias, a_log, H=H)
    log_decay, coef = torch.empty((2, n, H), dtype=torch.float32, device=z.device).unbind(0)
    rc = _lib_().b200_step_sizes(log_decay.data_ptr(), coef.data_ptr(), z.data_ptr(), _rows2(z), bias.data_ptr(), a_log.data_ptr(),
                                 n, H, DTYPE_ID[z.dtype], _stream())
    _lib.check_mixers(rc, "b200_step_sizes")
    return log_decay, coef


def _check_decay_inputs(q, k, v, state, nstate, seqs, G: int):
    _need_cuda(q, k, v, state, seqs)
    _check_seqs(seqs)
    n = q.shape[0]
    _, H, dk, dv = state.shape
    if H % G or q.shape[1] != G * dk or k.shape != q.shape or v.shape != (n, H * dv):
        raise ValueError("projections do not match the state's shape")
    if k.dtype != q.dtype or v.dtype != q.dtype:
        raise TypeError("q, k and v share one dtype")
    if state.dtype != torch.float32 or not state.is_contiguous():
        raise TypeError("the recurrent state is contiguous fp32")
    if nstate is not None and (nstate.dtype != torch.float32 or nstate.shape[1:] != (H, dk) or not nstate.is_contiguous()):
        raise ValueError("nstate is contiguous fp32 [slots, H, dk]")
    return n, H, dk, dv


CHUNK_SCAN_FROM = 16     # tokens of a step's longest portion from which the chunked tensor-core scan serves the step


@_timed
def decay_scan(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, log_decay: torch.Tensor, coef: torch.Tensor,
               state: torch.Tensor, seqs: torch.Tensor, G: int, q_scale: float = 1.0, skip: Optional[torch.Tensor] = None,
               nstate: Optional[torch.Tensor] = None, max_count: int = 0):
    """``S <- e^log_decay S + coef k v^T``, ``o = S^T (q_scale q) + skip v`` over each sequence's tokens, and with ``nstate``
    the vector recurrence ``n <- e^log_decay n + coef k`` and ``n . (q_scale q)``.  ``q / k [n, G*dk]``, ``v [n, H*dv]``,
    ``log_decay / coef`` fp32 ``[n, H]``, ``state`` fp32 ``[slots, H, dk, dv]``.  Returns ``(o fp32 [n, H, dv], nq fp32 [n, H]
    or None)``.  ``max_count``: the largest token count in ``seqs`` (picks the kernel: bf16 steps with a portion of
    ``CHUNK_SCAN_FROM`` tokens or more run chunks on the tensor cores, others token by token)."""
    n, H, dk, dv = _check_decay_inputs(q, k, v, state, nstate, seqs, G)
    _f32_heads(skip, H=H)
    for t in (log_decay, coef):
        if t.dtype != torch.float32 or tuple(t.shape) != (n, H) or not t.is_contiguous():
            raise ValueError("log_decay and coef are contiguous fp32 [n, H]")
    o = torch.empty((n, H, dv), dtype=torch.float32, device=q.device)
    nq = torch.empty((n, H), dtype=torch.float32, device=q.device) if nstate is not None else None
    lib, dt = _lib_(), DTYPE_ID[q.dtype]
    chunks = max_count >= CHUNK_SCAN_FROM and lib.b200_decay_chunk_scan_supported(dk, dv, dt)
    fn = lib.b200_decay_chunk_scan if chunks else lib.b200_decay_scan
    rc = fn(o.data_ptr(), _ptr(nq), q.data_ptr(), _rows2(q), k.data_ptr(), _rows2(k), v.data_ptr(), _rows2(v),
            log_decay.data_ptr(), coef.data_ptr(), _ptr(skip), float(q_scale), state.data_ptr(), _ptr(nstate), seqs.data_ptr(),
            seqs.shape[0], H, G, dk, dv, dt, _stream())
    _lib.check_mixers(rc, "b200_decay_chunk_scan" if chunks else "b200_decay_scan")
    return o, nq


@_timed
def decay_step(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, gates, state: torch.Tensor, seqs: torch.Tensor, G: int,
               q_scale: float = 1.0, skip: Optional[torch.Tensor] = None, nstate: Optional[torch.Tensor] = None,
               m_state: Optional[torch.Tensor] = None):
    """``decay_scan`` for steps of one token per sequence, the gates formed on the way.  ``gates``: ``("capped", zi, zf,
    bias_i, bias_f, cap)`` with ``m_state`` (only read), or ``("step", z, bias, a_log)``.  Returns ``(o, nq, m)``."""
    n, H, dk, dv = _check_decay_inputs(q, k, v, state, nstate, seqs, G)
    if seqs.shape[0] != n:
        raise ValueError("decay_step serves one token per sequence")
    _f32_heads(skip, H=H)
    capped = gates[0] == "capped"
    if capped:
        _, za, zb, p0, p1, cap = gates
        if zb.shape != za.shape or (n > 1 and zb.stride(0) != za.stride(0)) or m_state is None \
                or m_state.dtype != torch.float32 or m_state.shape[1:] != (H,) or not m_state.is_contiguous():
            raise ValueError("zi and zf are [n, H] slices with one row stride; m_state is fp32 [slots, H]")
    else:
        (_, za, p0, p1), zb, cap = gates, None, 1.0
    if tuple(za.shape) != (n, H) or za.dtype != q.dtype:
        raise ValueError("gate logits are [n, H] in the activations' dtype")
    _f32_heads(p0, p1, H=H)
    o = torch.empty((n, H, dv), dtype=torch.float32, device=q.device)
    nq = torch.empty((n, H), dtype=torch.float32, device=q.device) if nstate is not None else None
    m = torch.empty((n, H), dtype=torch.float32, device=q.device) if capped else None
    rc = _lib_().b200_decay_step(o.data_ptr(), _ptr(nq), _ptr(m), q.data_ptr(), _rows2(q), k.data_ptr(), _rows2(k),
                                 v.data_ptr(), _rows2(v), 0 if capped else 1, za.data_ptr(), _ptr(zb), _rows2(za),
                                 p0.data_ptr(), p1.data_ptr(), float(cap), _ptr(skip), float(q_scale), state.data_ptr(),
                                 _ptr(nstate), _ptr(m_state), seqs.data_ptr(), n, H, G, dk, dv, DTYPE_ID[q.dtype], _stream())
    _lib.check_mixers(rc, "b200_decay_step")
    return o, nq, m


@_timed
def normalized_head_out(o: torch.Tensor, nq: torch.Tensor, m: torch.Tensor, floor: float, weight: torch.Tensor,
                        gate: torch.Tensor, eps: float, m_state: Optional[torch.Tensor] = None,
                        seqs: Optional[torch.Tensor] = None) -> torch.Tensor:
    """fp32 ``o [n, H, dv]`` over ``max(|nq|, exp(-m)) + floor`` per head, made unit-RMS per head, times ``weight [H*dv]``,
    times ``sigmoid(gate [n, H*dv])``: ``[n, H*dv]`` in the weight's dtype.  With ``m_state`` (steps of one token per
    sequence) the running maxima ``m`` are stored at the sequences' slots."""
    _need_cuda(o, nq, m, weight, gate)
    n, H, dv = o.shape
    if any(t.dtype != torch.float32 or not t.is_contiguous() for t in (o, nq, m)) or nq.shape != (n, H) or m.shape != (n, H):
        raise ValueError("o [n, H, dv], nq and m [n, H] are contiguous fp32")
    if weight.numel() != H * dv or not weight.is_contiguous() or tuple(gate.shape) != (n, H * dv) or gate.dtype != weight.dtype:
        raise ValueError("weight [H*dv] and gate [n, H*dv] share one dtype")
    if m_state is not None:
        _check_seqs(seqs)
        if seqs.shape[0] != n or m_state.dtype != torch.float32 or m_state.shape[1:] != (H,) or not m_state.is_contiguous():
            raise ValueError("m_state is contiguous fp32 [slots, H], one sequence per row")
    out = torch.empty((n, H * dv), dtype=weight.dtype, device=o.device)
    rc = _lib_().b200_normalized_head_out(out.data_ptr(), H * dv, o.data_ptr(), nq.data_ptr(), m.data_ptr(), float(floor),
                                          weight.data_ptr(), gate.data_ptr(), _rows2(gate), float(eps), _ptr(m_state),
                                          _ptr(seqs), n, H, dv, DTYPE_ID[weight.dtype], _stream())
    _lib.check_mixers(rc, "b200_normalized_head_out")
    return out


@_timed
def gated_part_norm(y: torch.Tensor, z: torch.Tensor, weight: torch.Tensor, eps: float, parts: int) -> torch.Tensor:
    """``y * silu(z)`` with each of ``parts`` equal parts of the row divided by its own RMS, times ``weight``: fp32 ``y [n,
    inner]``, ``z`` and the result in the weight's dtype."""
    _need_cuda(y, z, weight)
    n, inner = z.shape
    if y.dtype != torch.float32 or not y.is_contiguous() or y.numel() != n * inner:
        raise ValueError("y is contiguous fp32 [n, inner]")
    if weight.numel() != inner or not weight.is_contiguous() or z.dtype != weight.dtype or inner % parts:
        raise ValueError("weight is [inner] in z's dtype and the parts divide the row")
    out = torch.empty((n, inner), dtype=weight.dtype, device=y.device)
    rc = _lib_().b200_gated_part_norm(out.data_ptr(), y.data_ptr(), z.data_ptr(), _rows2(z), weight.data_ptr(), float(eps), n,
                                      inner, int(parts), DTYPE_ID[weight.dtype], _stream())
    _lib.check_mixers(rc, "b200_gated_part_norm")
    return out


# ---- per-channel selective state spaces, sublayers normed on both sides (csrc/b200_selective_ops.cu) --------------------
@_timed
def selective_scan(x: torch.Tensor, dt: torch.Tensor, B: torch.Tensor, C: torch.Tensor, z: torch.Tensor, dt_bias: torch.Tensor,
                   rates: torch.Tensor, skip: torch.Tensor, state: torch.Tensor, seqs: torch.Tensor, gain: float = 1.0,
                   out: Optional[torch.Tensor] = None, max_count: int = 0) -> torch.Tensor:
    """Per channel ``c`` and state ``n``, with ``dt = softplus(dt + dt_bias)``: ``S <- e^(rate dt) S + dt x B``, ``y = S.C +
    skip x``; returns ``gain * y * silu(z)`` ``[n, inner]`` in the activations' dtype (``out`` may be a column slice of a wider
    buffer).  ``x / dt / z [n, inner]`` and ``B / C [n, N]`` (one row stride) may be column slices; ``dt_bias``, ``skip`` fp32
    ``[inner]``, ``rates`` (negative) fp32 ``[inner, N]``, ``state`` fp32 ``[slots, inner, N]``.  ``max_count``: the largest token count in
    ``seqs``; steps of single tokens take a launch of their own."""
    _need_cuda(x, dt, B, C, z, state, seqs)
    _check_seqs(seqs)
    n, inner = x.shape
    N = B.shape[1]
    if dt.shape != x.shape or z.shape != x.shape or B.shape != (n, N) or C.shape != B.shape:
        raise ValueError("x, dt, z are [n, inner], B and C [n, N]")
    if n > 1 and B.stride(0) != C.stride(0):
        raise ValueError("B and C must share a row stride")
    if any(t.dtype != x.dtype for t in (dt, B, C, z)):
        raise TypeError("activations share one dtype")
    for t, shape in ((dt_bias, (inner,)), (skip, (inner,)), (rates, (inner, N)), (state, (state.shape[0], inner, N))):
        if t.dtype != torch.float32 or tuple(t.shape) != shape or not t.is_contiguous():
            raise ValueError("constants and state are contiguous fp32")
    if out is None:
        out = torch.empty((n, inner), dtype=x.dtype, device=x.device)
    elif out.shape != x.shape or out.dtype != x.dtype:
        raise ValueError("out must be [n, inner] in the activations' dtype")
    step = max_count == 1 and seqs.shape[0] == n
    fn = _lib_().b200_selective_step if step else _lib_().b200_selective_scan
    rc = fn(out.data_ptr(), _rows2(out), x.data_ptr(), _rows2(x), dt.data_ptr(), _rows2(dt), dt_bias.data_ptr(), rates.data_ptr(),
            B.data_ptr(), C.data_ptr(), _rows2(B), skip.data_ptr(), z.data_ptr(), _rows2(z), float(gain), state.data_ptr(),
            seqs.data_ptr(), seqs.shape[0], inner, N, DTYPE_ID[x.dtype], _stream())
    _lib.check_mixers(rc, "b200_selective_step" if step else "b200_selective_scan")
    return out


@_timed
def sandwich_residual(x: torch.Tensor, y: torch.Tensor, w_norm: torch.Tensor, layer_scale: Optional[torch.Tensor], eps: float,
                      w_next: Optional[torch.Tensor] = None, eps_next: float = 0.0, sign: float = 1.0) -> Optional[torch.Tensor]:
    """In place ``x += sign * layer_scale * w_norm * y * rsqrt(mean(y^2) + eps)`` on the fp32 residual (``y`` fp32 or of the
    weights' dtype); with ``w_next`` returns ``w_next * x * rsqrt(mean(x^2) + eps_next)`` of the new residual in that dtype."""
    _need_cuda(x, y, w_norm)
    T = w_norm.dtype
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or y.shape != x.shape:
        raise ValueError("x must be contiguous fp32 [rows, width] and y of the same shape")
    if y.dtype not in (T, torch.float32):
        raise TypeError("y is fp32 or of the weights' dtype")
    for w in (w_norm, layer_scale, w_next):
        if w is not None and (w.dtype != T or w.numel() != x.shape[1] or not w.is_contiguous()):
            raise ValueError("weights are contiguous [width] in one dtype")
    out = torch.empty(x.shape, dtype=T, device=x.device) if w_next is not None else None
    rc = _lib_().b200_sandwich_residual(x.data_ptr(), y.data_ptr(), _rows2(y), int(y.dtype == torch.float32 and T != torch.float32),
                                        float(sign), w_norm.data_ptr(), _ptr(layer_scale), float(eps), _ptr(w_next),
                                        float(eps_next), _ptr(out), x.shape[0], x.shape[1], DTYPE_ID[T], _stream())
    _lib.check_mixers(rc, "b200_sandwich_residual")
    return out


@_timed
def gelu_glu(gu: torch.Tensor) -> torch.Tensor:
    """``gelu_tanh(g) * u`` of contiguous rows ``g | u``."""
    _need_cuda(gu)
    if not gu.is_contiguous() or gu.dim() != 2 or gu.shape[1] % 2:
        raise ValueError("gu must be contiguous [rows, 2*ff]")
    ff = gu.shape[1] // 2
    y = torch.empty((gu.shape[0], ff), dtype=gu.dtype, device=gu.device)
    rc = _lib_().b200_gelu_glu(y.data_ptr(), gu.data_ptr(), gu.shape[0], ff, DTYPE_ID[gu.dtype], _stream())
    _lib.check_mixers(rc, "b200_gelu_glu")
    return y
