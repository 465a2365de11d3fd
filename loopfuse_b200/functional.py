"""Tensor-level entry points: torch CUDA tensors in, kernels of liblf_sm100.so out.

These are what the compiled callable produced by ``loopfuse_backend`` calls; they can also be
used directly. PyTorch only supplies device memory and the current stream here - all arithmetic
happens in the library. Nothing in this module computes attention on the CPU or with torch ops.
The argument checks, the output allocation and the launch are in the native host path
(csrc/lf_host.cpp): in Python they took longer than a small kernel runs.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence

import torch

from . import _native
from .spec import MASK_NONE, ScoreMod

_DEV_TIMEOUT = 1
_DEV_BAD_PAGE = 2


def _require_cuda(*tensors: torch.Tensor) -> torch.device:
    dev = tensors[0].device
    for t in tensors:
        if not t.is_cuda:
            raise RuntimeError(
                "loopfuse_b200 kernels need CUDA tensors on an sm_100 GPU; there is no CPU path")
        if t.device != dev:
            raise ValueError("all tensors must live on the same device")
    return dev


def _check_bf16_lastdim(t: torch.Tensor, name: str) -> None:
    if t.dtype != torch.bfloat16:
        raise TypeError(f"{name} must be bfloat16, got {t.dtype}")
    if t.stride(-1) != 1:
        raise ValueError(f"{name} must have a contiguous last dim")


def _stream_ptr(dev: torch.device) -> int:
    return torch.cuda.current_stream(dev).cuda_stream


def new_status(device) -> torch.Tensor:
    """A zeroed device word the kernels report device-side problems into."""
    return torch.zeros(1, dtype=torch.int32, device=device)


def check_status(status: torch.Tensor, what: str = "kernel") -> None:
    """Synchronising read of a status word; raises if a kernel recorded a problem."""
    code = int(status.item())
    if code == 0:
        return
    if (code & 0xFF) == _DEV_TIMEOUT:
        raise RuntimeError(f"{what}: a bounded device-side wait ran out (site {code >> 8})")
    if (code & 0xFF) == _DEV_BAD_PAGE:
        raise RuntimeError(f"{what}: block_table holds a page id outside the pool")
    raise RuntimeError(f"{what}: device status {code}")


def prefill_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float = 1.0,
                      mods: Sequence[ScoreMod] = (), mask_kind: int = MASK_NONE,
                      window: int = 0, causal_offset: int = 0,
                      out: Optional[torch.Tensor] = None,
                      status: Optional[torch.Tensor] = None,
                      dbg_ranges: Optional[torch.Tensor] = None,
                      kv_tile: int = 0, sm_margin: int = 0,
                      k_block_table: Optional[torch.Tensor] = None,
                      v_block_table: Optional[torch.Tensor] = None,
                      seq_len: Optional[int] = None,
                      score_bias: Optional[torch.Tensor] = None,
                      bias_pos: Optional[int] = None,
                      q_pe: Optional[torch.Tensor] = None,
                      k_pe: Optional[torch.Tensor] = None,
                      q_bias: Optional[torch.Tensor] = None,
                      out_bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """softmax(mask(mods(scale * q k^T))) v for q [B,Hq,Sq,D], k/v [B,Hkv,Skv,D] (bf16).

    ``score_bias`` (bf16 ``[B, Hq, Sq, Skv]``) is added to the scores after the first
    ``bias_pos`` ops of ``mods`` (default: after all of them) and before the mask; the kernel
    reads it tile by tile (dense k / v only).

    ``q_pe`` ``[B, Hq, Sq, D_pe]`` and ``k_pe`` ``[B, Hkv, Skv, D_pe]`` (bf16, D_pe a multiple of
    8 up to 64) add a second product to the scores: ``scale * (q k^T + q_pe k_pe^T)``, the
    two-matmul (MLA-style) form; ``mods`` may then hold constant multipliers only.

    ``q_bias`` and ``out_bias`` (bf16, the shape of ``q``) are added to ``q`` before the scores and to
    the output, each with one rounding to bf16: in the same launch where a ``score_bias`` with only
    multipliers in front of it is given, else by ``add_bf16`` (the same bits).

    With ``k_block_table`` (``v_block_table``), ``k`` (``v``) is a paged pool
    ``[pages, page_size, Hkv, D]`` (or ``[pages, Hkv, D]``, one token per page) read through that
    int32 table ``[B, blocks]``; the gather is fused into the kernel's tile loads. ``seq_len``
    bounds the keys when the table covers more.

    ``kv_tile`` pins the KV tile of the kernel (64 or 128 keys; 0 lets the library choose);
    ``sm_margin`` leaves that many SMs free of the persistent kernels' CTAs (for a collective
    that runs at the same time on another stream)."""
    return _native.host().prefill(q, k, v, out, status, dbg_ranges, k_block_table, v_block_table,
                                  score_bias, q_pe, k_pe, scale, mods, mask_kind, window,
                                  causal_offset, kv_tile, sm_margin, seq_len, bias_pos, q_bias,
                                  out_bias)


def add_bf16(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """out = a + b for bf16 [B, H, S, D] tensors of one shape (any strides with innermost 1);
    ``out`` may be ``a`` or ``b``. The query-bias and output-bias steps of a biased attention."""
    return _native.host().add(a, b, out)


class PreparedPrefill:
    """A prefill call bound once to its tensors and parameters, for loops that launch the same
    problem again and again (a serving step, a benchmark): the argument record of the C ABI is
    filled and validated a single time, ``run()`` only launches. This is the per-call host work
    the reference's generated launcher repeats on every call (loopfuse/codegen.py:215-298:
    output allocation, stride extraction, grid computation). The tensors are kept alive by the
    object; new data written into the same buffers is picked up by the next ``run()``."""

    def __init__(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float = 1.0,
                 mods: Sequence[ScoreMod] = (), mask_kind: int = MASK_NONE, window: int = 0,
                 causal_offset: int = 0, out: Optional[torch.Tensor] = None,
                 status: Optional[torch.Tensor] = None, kv_tile: int = 0,
                 sm_margin: int = 0) -> None:
        self._args, self.out = _prefill_record(q, k, v, scale, mods, mask_kind, window,
                                               causal_offset, out, status, kv_tile, sm_margin)
        self._keep = (q, k, v, status)
        self._dev = q.device
        self._fn = _native.load().lf_prefill_bf16
        self._ref = C.byref(self._args)
        self._dev_index = self._dev.index if self._dev.index is not None else \
            torch.cuda.current_device()

    def run(self, out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Launch on the current stream of the tensors' device (which must be the current
        device); ``out`` replaces the output buffer (same shape and strides) for this and later
        runs."""
        if out is not None:
            if out.shape != self.out.shape or out.stride() != self.out.stride():
                raise ValueError("out must match the prepared output's shape and strides")
            self.out = out
            self._args.out = out.data_ptr()
        rc = self._fn(self._ref, torch.cuda.current_stream(self._dev_index).cuda_stream)
        if rc:
            _native.check(rc, "lf_prefill_bf16")
        return self.out


def prefill_kv_tile(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float = 1.0,
                    mods: Sequence[ScoreMod] = (), mask_kind: int = MASK_NONE, window: int = 0,
                    causal_offset: int = 0, kv_tile: int = 0) -> int:
    """KV tile size (64 or 128 keys) of the kernel ``prefill_attention`` runs for these
    arguments; skip ranges and ``dbg_ranges`` are in units of it."""
    a, _ = _prefill_record(q, k, v, scale, mods, mask_kind, window, causal_offset, q, None,
                           kv_tile, 0)
    rc = _native.load().lf_prefill_kv_tile(C.byref(a))
    if rc < 0:
        _native.check(rc, "lf_prefill_kv_tile")
    return rc


def prefill_q_tile(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float = 1.0,
                   mods: Sequence[ScoreMod] = (), mask_kind: int = MASK_NONE, window: int = 0,
                   causal_offset: int = 0, kv_tile: int = 0) -> int:
    """Query rows per head that one tile of the kernel ``prefill_attention`` runs for these
    arguments covers (128, or 32 in the packed grouped-query layout); ``dbg_ranges`` holds one
    (lo, hi) per (batch, head, tile of that many rows)."""
    a, _ = _prefill_record(q, k, v, scale, mods, mask_kind, window, causal_offset, q, None,
                           kv_tile, 0)
    rc = _native.load().lf_prefill_q_tile(C.byref(a))
    if rc < 0:
        _native.check(rc, "lf_prefill_q_tile")
    return rc


PREFILL_FORMS = ("pairs", "split", "narrow")


def prefill_form(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float = 1.0,
                 mods: Sequence[ScoreMod] = (), mask_kind: int = MASK_NONE, window: int = 0,
                 causal_offset: int = 0, kv_tile: int = 0, sm_margin: int = 0,
                 k_block_table: Optional[torch.Tensor] = None,
                 v_block_table: Optional[torch.Tensor] = None, seq_len: Optional[int] = None,
                 score_bias: Optional[torch.Tensor] = None, bias_pos: Optional[int] = None,
                 q_pe: Optional[torch.Tensor] = None,
                 k_pe: Optional[torch.Tensor] = None) -> str:
    """How the kernel that ``prefill_attention`` runs for these arguments deals the query tiles
    out: ``"pairs"`` (a CTA of two tiles per SM), ``"split"`` (one tile on a CTA's two slots) or
    ``"narrow"`` (two CTAs of one tile per SM). (Row biases do not change it.)"""
    rec, _, _ = _native.host().prefill_record(
        q, k, v, q, None, None, k_block_table, v_block_table, score_bias, q_pe, k_pe, scale, mods,
        mask_kind, window, causal_offset, kv_tile, sm_margin, seq_len, bias_pos)
    a = _native.LfPrefillArgs.from_buffer_copy(rec)
    rc = _native.load().lf_prefill_form(C.byref(a), 0)
    if rc < 0:
        _native.check(rc, "lf_prefill_form")
    return PREFILL_FORMS[rc]


def _prefill_record(q, k, v, scale, mods, mask_kind, window, causal_offset, out, status, kv_tile,
                    sm_margin):
    """(LfPrefillArgs, out) of a dense prefill, checked and filled but not launched."""
    rec, out, _ = _native.host().prefill_record(
        q, k, v, out, status, None, None, None, None, None, None, scale, mods, mask_kind, window,
        causal_offset, kv_tile, sm_margin, None, None)
    return _native.LfPrefillArgs.from_buffer_copy(rec), out


class DecodeWorkspace:
    """Caller-owned scratch for split-KV partials, grown on demand and reused by the calls that it is
    passed to. It belongs to one thread at a time. A call on another stream than the last one's
    gets a new buffer, so work in flight keeps the old one. (A call without a workspace allocates its
    partials from PyTorch's caching allocator.)"""

    def __init__(self) -> None:
        self._buf: Optional[torch.Tensor] = None
        self._stream: Optional[int] = None

    def get(self, nbytes: int, device) -> Optional[torch.Tensor]:
        if nbytes == 0:
            return None
        stream = torch.cuda.current_stream(device).cuda_stream
        if (self._buf is None or self._buf.numel() < nbytes or self._buf.device != device
                or self._stream != stream):
            self._buf = torch.empty(nbytes, dtype=torch.uint8, device=device)
            self._stream = stream
        return self._buf


def decode_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float = 1.0,
                     mods: Sequence[ScoreMod] = (), splits: int = 0,
                     out: Optional[torch.Tensor] = None,
                     workspace: Optional[DecodeWorkspace] = None,
                     status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Unmasked attention of G query rows per kv head: q [B,Hkv,G,D], k/v [B,Hkv,Skv,D]."""
    return _native.host().decode(q, k, v, out, workspace, status, scale, mods, splits)


def _pool_view(pool: torch.Tensor, name: str) -> torch.Tensor:
    _check_bf16_lastdim(pool, name)
    if pool.dim() == 3:  # [pages, Hkv, D]: one token per page
        pool = pool.unsqueeze(1)
    if pool.dim() != 4:
        raise ValueError(f"{name} must be [pages, page_size, Hkv, D] or [pages, Hkv, D]")
    return pool


def _table_i32(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        raise ValueError("block_table must be [batch, blocks]")
    if t.dtype != torch.int32:
        t = t.to(torch.int32)
    if t.stride(1) != 1:
        t = t.contiguous()
    return t


def paged_decode_attention(q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor,
                           block_table: torch.Tensor, *, seq_len: Optional[int] = None,
                           block_table_v: Optional[torch.Tensor] = None, scale: float = 1.0,
                           mods: Sequence[ScoreMod] = (), splits: int = 0,
                           out: Optional[torch.Tensor] = None,
                           workspace: Optional[DecodeWorkspace] = None,
                           status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Decode attention over a paged KV cache: q [B,Hkv,G,D]; pools [pages, page_size, Hkv, D]
    (or [pages, Hkv, D] for one-token pages); block_table int32 [B, blocks]. Token t of sequence
    b lives at pool[block_table[b, t // page_size], t % page_size]."""
    return _native.host().paged_decode(q, k_pool, v_pool, block_table, block_table_v, out,
                                       workspace, status, seq_len, scale, mods, splits)


def paged_gather(pool: torch.Tensor, block_table: torch.Tensor, *, seq_len: Optional[int] = None,
                 status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Materialise [B, Hkv, S, D] from a paged pool (page-index check and paged prefill input)."""
    dev = _require_cuda(pool, block_table)
    pool = _pool_view(pool, "pool")
    bt = _table_i32(block_table)
    n_pages, page_size, Hkv, D = pool.shape
    B = bt.shape[0]
    S = seq_len if seq_len is not None else bt.shape[1] * page_size
    out = torch.empty((B, Hkv, S, D), dtype=torch.bfloat16, device=dev)
    strides = (C.c_int64 * 3)(pool.stride(0), pool.stride(1), pool.stride(2))
    with torch.cuda.device(dev):
        rc = _native.load().lf_paged_gather_bf16(
            pool.data_ptr(), bt.data_ptr(), out.data_ptr(), B, Hkv, S, D, page_size, n_pages,
            strides, bt.stride(0), status.data_ptr() if status is not None else None,
            _stream_ptr(dev))
    _native.check(rc, "lf_paged_gather_bf16")
    return out


def kv_append(k_new: torch.Tensor, v_new: torch.Tensor, k_pool: torch.Tensor,
              v_pool: torch.Tensor, block_table: torch.Tensor, *,
              seq_pos: Optional[torch.Tensor] = None, start_pos: int = 0,
              block_table_v: Optional[torch.Tensor] = None,
              status: Optional[torch.Tensor] = None) -> None:
    """Write new K/V rows ``[B, Hkv, T, D]`` into the pages of a paged cache, in place: token i
    of sequence b goes to ``pool[block_table[b, pos // page_size], pos % page_size]`` with
    ``pos = seq_pos[b] + i`` (or ``start_pos + i``). The device-side producer of the cache that
    ``paged_decode_attention`` reads."""
    _native.host().kv_append(k_new, v_new, k_pool, v_pool, block_table, block_table_v, seq_pos,
                             start_pos, status)
