"""Packed variable-length attention (training / log-prob / prefill path).

``qkv`` is one packed buffer ``[T, (Hq + 2*Hkv) * D]`` (q heads | k heads | v heads per token), sequences are
consecutive row ranges described by :class:`SeqInfo`.  CUDA tensors use the tcgen05 kernels of
``csrc/fmha_fwd.cu`` / ``csrc/fmha_bwd.cu``; CPU tensors use the eager statement in ``reference``."""
from __future__ import annotations

import ctypes
import math
from typing import List, Optional, Sequence

import torch

from . import lib as _lib
from . import reference as ref




class SeqInfo:
    """Sequence boundaries of a packed batch plus the tile lists the attention kernels need."""

    def __init__(self, seqlens: Sequence[int], device=None):
        self.seqlens: List[int] = [int(x) for x in seqlens]
        cu = [0]
        for n in self.seqlens:
            cu.append(cu[-1] + n)
        self.cu_seqlens_cpu = cu
        self.total = cu[-1]
        self.max_seqlen = max(self.seqlens) if self.seqlens else 0
        self.device = device
        self._tiles = {}
        self._cu_dev = None
        self._pos = None

    @property
    def cu_seqlens(self) -> torch.Tensor:
        if self._cu_dev is None:
            self._cu_dev = torch.tensor(self.cu_seqlens_cpu, dtype=torch.int32, device=self.device)
        return self._cu_dev

    @property
    def positions(self) -> torch.Tensor:
        """Position of every packed token inside its sequence, int32 ``[T]``."""
        if self._pos is None:
            pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in self.seqlens]) if self.seqlens else \
                torch.zeros(0, dtype=torch.int32)
            self._pos = pos.to(self.device) if self.device is not None else pos
        return self._pos

    def tiles(self, hq: int, d: int, q_start: Optional[Sequence[int]] = None):
        """(seq_start, seq_len, offset) int32 device tensors, one entry per tile of query rows, their number and the rows
        of a tile for ``hq`` heads of width ``d``; longest sequences' last tiles first so the heaviest causal tiles start
        early.  ``q_start[i]`` leaves out the rows of sequence i below ``q_start[i] // 128 * 128``: chunked prefill
        computes only the new rows."""
        first = [int(q) // 128 * 128 for q in q_start] if q_start is not None else [0] * len(self.seqlens)
        rows = fwd_tile_rows(len(first), self.total - sum(first), hq, d)
        if q_start is None and rows in self._tiles:
            return self._tiles[rows]
        entries = [(self.cu_seqlens_cpu[i], n, t0) for i, n in enumerate(self.seqlens) for t0 in range(first[i], n, rows)]
        tiles = self._device_tiles(sorted(entries, key=lambda e: -e[2])) + (rows,)
        if q_start is None:
            self._tiles[rows] = tiles
        return tiles

    def kv_tiles(self):
        """The same for the 128-row K/V tiles of the backward kernel: a causal tile meets the query rows from its own
        on, so the tiles with most rows behind them come first."""
        if "kv" not in self._tiles:
            entries = [(self.cu_seqlens_cpu[i], n, t0) for i, n in enumerate(self.seqlens) for t0 in range(0, n, 128)]
            self._tiles["kv"] = self._device_tiles(sorted(entries, key=lambda e: e[2] - e[1]))
        return self._tiles["kv"]

    def _device_tiles(self, entries):
        mk = lambda k: torch.tensor([e[k] for e in entries], dtype=torch.int32, device=self.device)  # noqa: E731
        return (mk(0), mk(1), mk(2), len(entries))


def fwd_tile_rows(sequences: int, query_rows: int, hq: int, d: int) -> int:
    """Query rows of one block of the forward kernel: 256, or 128 where a second tile of 128 would mostly stand idle.  A block
    of 128 rows takes half an SM (d = 128) or a third, so short sequences hide each other's latencies; a longer one fetches
    its keys twice as often.  256 / 128 rows, us, causal: d = 128, 28 / 4 heads: 256 x 64 tokens 301 / 128, 128 x 128:
    188 / 119, 64 x 200: 149 / 123, 40 x 384: 192 / 147, 32 x 512: 192 / 176 but 216 / 237 not causal, and 4 x 384 with
    16 heads, one block an SM, 12 / 14; d = 64, 14 / 2: 256 x 64: 50 / 37, 128 x 128: 43 / 35, 64 x 160 30 / 31."""
    if query_rows <= 128 * sequences:
        return 128
    if d == 128 and query_rows <= 384 * sequences and -(-query_rows // 256) * hq > _lib.NUM_SMS:
        return 128
    return 256


def bwd_head_splits(seqlens: Sequence[int], hq: int, hkv: int, causal: bool) -> int:
    """Blocks over which the backward kernel divides the q heads of a kv head: more of them shorten the longest block, but
    each costs some five steps of its own (loading K and V, writing dK and dV), and another where a share's dK and dV go
    through a buffer.  In steps of one 128 x 128 tile of one head the pass takes the longest block, or the SMs' average and
    a tail that shrinks with the blocks an SM gets.  Forward and backward, us, for 1, 2, 3, 4, 7 blocks, causal: 28 / 4
    heads, d = 128: 32 x 64: 90, 108, 116, 126, 157; 16 x 128: 79, 75, 89, 88, 113; 4 x 512: 150, 116, 108, 113, 126;
    1 x 1024: 231, 154, 128, 103, 93; 4 x 2048: 841, 720, 738, 762, 836; 14 / 2 heads, d = 64: 1 x 9000: 1300, 874, 846,
    825, 845; 16 x 1000: 326, 301, 311, 326, 371."""
    rep = hq // hkv
    tiles = [(n + 127) // 128 for n in seqlens]
    average = sum(t * (t + 1) // 2 if causal else t * t for t in tiles) * hq / _lib.NUM_SMS
    longest, blocks = max(tiles, default=0), sum(tiles) * hkv

    def steps(splits):
        block, per_sm = -(-rep // splits) * longest, blocks * splits / _lib.NUM_SMS
        own = 5 * math.ceil(per_sm) + (per_sm if splits > 1 else 0)
        return max(block, average + block / max(1.0, per_sm) ** 2) + own
    return min(range(1, rep + 1), key=steps)


def bwd_ordered(max_seqlen: int, d: int, causal: bool) -> bool:
    """Whether the backward kernel adds the parts of dQ in a fixed order, so that equal inputs give equal gradients: causal
    sequences of up to 4096 rows (d = 64) or 8192 (d = 128), and all under ``torch.use_deterministic_algorithms``.  It
    costs up to 12 % of the pass at 1024 rows, a quarter at 2048, a third and more from 4096 on (csrc/fmha_bwd.cu)."""
    return torch.are_deterministic_algorithms_enabled() or causal and max_seqlen <= 64 * d


def fmha_bwd(qkv, out, lse, dout, info: SeqInfo, hq: int, hkv: int, d: int, causal: bool, scale: float) -> torch.Tensor:
    """Gradient of the packed ``qkv`` from the forward kernel's outputs."""
    L = _lib.get_lib()
    T = qkv.shape[0]
    dqkv = torch.empty_like(qkv)
    delta = torch.empty(hq, T, dtype=torch.float32, device=qkv.device)
    dq_acc = torch.empty(T, hq * d, dtype=torch.float32, device=qkv.device)
    splits = bwd_head_splits(info.seqlens, hq, hkv, causal)
    dkv_acc = torch.empty(splits, T, 2 * hkv * d, dtype=torch.float32, device=qkv.device) if splits > 1 else None
    turn = None
    if bwd_ordered(info.max_seqlen, d, causal):
        turn = torch.empty(hq * (T + 1), dtype=torch.int32, device=qkv.device)
        if info.total < T:
            dq_acc[info.total:].zero_()     # rows of no sequence
    ts, tl, t0, n = info.kv_tiles()
    rc = L.sb_fmha_bwd(_lib.ptr(qkv), _lib.ptr(out), _lib.ptr(dout), _lib.ptr(lse), _lib.ptr(delta), _lib.ptr(dq_acc),
                       _lib.ptr(dkv_acc), _lib.ptr(turn), _lib.ptr(dqkv), _lib.ptr(ts), _lib.ptr(tl), _lib.ptr(t0), n, T,
                       hq, hkv, d, int(causal), splits, ctypes.c_float(scale), _lib.ptr(_lib.status_word(qkv.device)), _lib.stream())
    _lib.check(rc, "sb_fmha_bwd")
    _lib.add_launches(int(splits > 1))
    return dqkv


class _AttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, info: SeqInfo, hq, hkv, d, causal, scale, q_start=None):
        L = _lib.get_lib()
        T = qkv.shape[0]
        out = torch.empty(T, hq * d, dtype=qkv.dtype, device=qkv.device)
        lse = torch.empty(hq, T, dtype=torch.float32, device=qkv.device)
        ts, tl, t0, n, rows = info.tiles(hq, d, q_start)
        rc = L.sb_fmha_fwd(_lib.ptr(qkv), _lib.ptr(out), _lib.ptr(lse), _lib.ptr(ts), _lib.ptr(tl), _lib.ptr(t0), n, rows,
                           T, hq, hkv, d, int(causal), ctypes.c_float(scale), _lib.ptr(_lib.status_word(qkv.device)),
                           _lib.stream())
        _lib.check(rc, "sb_fmha_fwd")
        ctx.save_for_backward(qkv, out, lse)
        ctx.meta = (info, hq, hkv, d, causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        qkv, out, lse = ctx.saved_tensors
        info, hq, hkv, d, causal, scale = ctx.meta
        dqkv = fmha_bwd(qkv, out, lse, dout.contiguous(), info, hq, hkv, d, causal, scale)
        return dqkv, None, None, None, None, None, None, None


def _pad_heads(qkv: torch.Tensor, n_heads_total: int, d: int, d_pad: int) -> torch.Tensor:
    T = qkv.shape[0]
    x = qkv.reshape(T, n_heads_total, d)
    return torch.nn.functional.pad(x, (0, d_pad - d)).reshape(T, n_heads_total * d_pad)


def attention_packed(qkv: torch.Tensor, info: SeqInfo, n_heads: int, n_kv_heads: int, head_dim: int,
                     causal: bool = True, scale: Optional[float] = None,
                     q_start: Optional[Sequence[int]] = None) -> torch.Tensor:
    """Attention over a packed batch; returns ``[T, n_heads * head_dim]``.  ``q_start`` (inference only): rows of
    sequence i below ``q_start[i] // 128 * 128`` are not computed (their output rows are undefined)."""
    scale = scale if scale is not None else 1.0 / math.sqrt(head_dim)
    T = qkv.shape[0]
    if not qkv.is_cuda:
        q, k, v = qkv.split([n_heads * head_dim, n_kv_heads * head_dim, n_kv_heads * head_dim], dim=-1)
        out = ref.attention_varlen(q.reshape(T, n_heads, head_dim), k.reshape(T, n_kv_heads, head_dim),
                                   v.reshape(T, n_kv_heads, head_dim), torch.tensor(info.cu_seqlens_cpu),
                                   causal=causal, scale=scale)
        return out.reshape(T, n_heads * head_dim)
    _lib.use_native(qkv)
    if q_start is not None:
        assert not (torch.is_grad_enabled() and qkv.requires_grad), "q_start is an inference-only option"
    if head_dim in (64, 128):
        return _AttnFn.apply(qkv.contiguous(), info, n_heads, n_kv_heads, head_dim, causal, scale, q_start)
    d_pad = 64 if head_dim < 64 else 128
    assert head_dim <= 128, "head_dim > 128 is not supported"
    padded = _pad_heads(qkv, n_heads + 2 * n_kv_heads, head_dim, d_pad)
    out = _AttnFn.apply(padded, info, n_heads, n_kv_heads, d_pad, causal, scale, q_start)
    return out.reshape(T, n_heads, d_pad)[..., :head_dim].reshape(T, n_heads * head_dim)


def attention_wide_heads(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, info: SeqInfo, causal: bool = True,
                         scale: Optional[float] = None) -> torch.Tensor:
    """Attention with query/key width and value width outside the tcgen05 kernels' set (multi-head latent attention:
    192 / 128).  ``q, k [T, nh, dq]``, ``v [T, nh, dv]`` packed -> ``[T, nh, dv]``.  On GPUs this is a library call
    (the flash-attn variable-length kernel with the values zero-padded to ``dq``, as the reference does in
    siirl/models/transformers/kimi_vl.py:172-221; PyTorch's fused attention per sequence when flash-attn is absent);
    on CPU the eager statement."""
    T, nh, dq = q.shape
    dv = v.shape[-1]
    scale = scale if scale is not None else 1.0 / math.sqrt(dq)
    if not q.is_cuda:
        return ref.attention_varlen(q, k, v, torch.tensor(info.cu_seqlens_cpu), causal=causal, scale=scale).to(q.dtype)
    import torch.nn.functional as F
    vp = F.pad(v, (0, dq - dv)) if dv < dq else v
    try:
        from flash_attn import flash_attn_varlen_func
        cu = torch.tensor(info.cu_seqlens_cpu, dtype=torch.int32, device=q.device)
        mx = max(info.seqlens) if len(info.seqlens) else 0
        out = flash_attn_varlen_func(q, k, vp, cu, cu, mx, mx, softmax_scale=scale, causal=causal)
    except ImportError:
        outs, at = [], 0
        for n in info.seqlens:
            o = F.scaled_dot_product_attention(q[at:at + n].transpose(0, 1)[None], k[at:at + n].transpose(0, 1)[None],
                                               vp[at:at + n].transpose(0, 1)[None], is_causal=causal, scale=scale)
            outs.append(o[0].transpose(0, 1))
            at += n
        out = torch.cat(outs) if outs else q.new_zeros(0, nh, dq)
    return out[..., :dv]
