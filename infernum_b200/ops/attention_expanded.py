"""Prompt attention through a latent with the keys and values made
(``attention_expanded.cu``), one compiled module per (unrotated, rotated, value) size
of a head, built when a model first needs it.

``plan`` says whether a step runs this way: each cached vector the step's rows see is
turned into every head's key and value once (``2 kv_rank (dim + vdim)`` multiply-adds a
head), after which a query and a key cost ``dim + rot + vdim`` multiply-adds a head instead of
``2 kv_rank + rot`` over the latents themselves.
"""

from __future__ import annotations

import ctypes
from typing import Dict, Optional, Tuple

import torch

from ..csrc.build import load_module
from ..errors import KernelError
from . import core

_c_int, _c_float, _c_void_p = ctypes.c_int, ctypes.c_float, ctypes.c_void_p
_libs: Dict[Tuple[int, int, int], ctypes.CDLL] = {}
KEY_TILE = 128
# Rows an entry from which the made keys pay.  By the arithmetic (1.2 PFLOP/s for the product that makes them, 130 TFLOP/s
# over the latents against some 900 over made keys) some 28; below this the product and two more launches are not hidden.
MIN_ROWS_PER_ENTRY = 64
MAX_KEY_BYTES = 1 << 30


def supported(dim: int, rot_dim: int, vdim: int) -> bool:
    return dim in (64, 128) and rot_dim == 64 and vdim in (64, 128)


def lib_for(dim: int, rot_dim: int, vdim: int) -> ctypes.CDLL:
    lib = _libs.get((dim, rot_dim, vdim))
    if lib is None:
        lib = load_module(f"attn_expanded_d{dim}_r{rot_dim}_v{vdim}", ["attention_expanded.cu"],
                          [f"-DEX_D={dim}", f"-DEX_R={rot_dim}", f"-DEX_V={vdim}"])
        lib.ib_gather_latents.argtypes = [_c_void_p, _c_void_p, _c_void_p, _c_void_p, _c_void_p, _c_int, _c_int, _c_int, _c_int,
                                          _c_int, _c_int, _c_int, _c_void_p, _c_void_p]
        lib.ib_attention_expanded.argtypes = [
            _c_void_p, _c_int, _c_void_p, _c_void_p, _c_int, _c_int, _c_void_p, _c_int, _c_int, _c_int, _c_void_p, _c_int,
            _c_void_p, _c_void_p, _c_int, _c_int, _c_int, _c_int, _c_int, _c_float, _c_void_p, _c_void_p, _c_int, _c_void_p,
            _c_void_p]
        for fn in (lib.ib_gather_latents, lib.ib_attention_expanded, lib.ib_attention_expanded_sizes):
            fn.restype = _c_int
        if lib.ib_attention_expanded_sizes() != dim * 1000000 + rot_dim * 1000 + vdim:
            raise KernelError(f"attention module for sizes ({dim}, {rot_dim}, {vdim}) was built for others")
        _libs[(dim, rot_dim, vdim)] = lib
    return lib


def plan(ctx, n_rows: int, window: int, bytes_per_key: int) -> int:
    """Rows of the buffers that hold the step's keys (at least as many as there are: a recorded step knows bounds only), or
    0 when the step runs over the latents.  Every entry has to bring rows enough on average, and the keys made must not
    be many times the rows that read them (portions far behind in long contexts, recordings with room for many).
    Behind a window an entry's keys begin at the last multiple of ``KEY_TILE`` that its first row sees, at most
    ``window + KEY_TILE - 2`` before that row."""
    if n_rows < MIN_ROWS_PER_ENTRY * ctx.n_entries:
        return 0
    lens, reach = list(getattr(ctx, "host_kv_len", None) or ()), window + KEY_TILE - 2
    if len(lens) == ctx.n_entries:
        most, cu = 16 * n_rows, ctx.host_cu_rows
        keys = sum(min(n, cu[i + 1] - cu[i] + reach) if window > 0 else n for i, n in enumerate(lens))
    else:
        # a recording: lengths up to the bound, the rows among the entries in any way (``host_cu_rows`` does not say);
        # its buffers stay with it
        most, keys = 8 * n_rows, ctx.n_entries * ctx.max_kv_len
        if window > 0:
            keys = min(keys, n_rows + ctx.n_entries * reach)
    if keys > most or keys * bytes_per_key > MAX_KEY_BYTES:
        return 0
    return keys


def run(q: torch.Tensor, qr: torch.Tensor, pool: torch.Tensor, w_kv, out: torch.Tensor, kv_rank: int, dim: int, vdim: int,
        keys: int, ctx, tables: torch.Tensor, scale: float, window: int, rt, sink: Optional[torch.Tensor] = None,
        gate: Optional[torch.Tensor] = None) -> None:
    """``q`` [N, heads * (dim + rot)] with its rotated parts, rotated, in ``qr`` [N, heads, rot]; ``pool`` [pages, 1,
    page_size, kv_rank + rot]; ``w_kv`` the ``Linear`` of all heads' ``W_uk`` rows, then all heads' ``W_uv`` rows; ``out`` [N,
    heads * vdim].  ``sink`` and ``gate`` as in ``attention.latent_attention``."""
    num_pages, _one, page_size, width = pool.shape
    N, heads, rot = qr.shape
    core.require_cuda(q, qr, pool, out, tables, sink, gate)
    core.check_sink_and_gate(sink, gate, qr, "attention_expanded")
    if q.dtype != torch.bfloat16 or pool.dtype != q.dtype or out.dtype != q.dtype or not qr.is_contiguous() \
            or q.stride(1) != 1 or out.stride(1) != 1 or not pool.is_contiguous() or width != kv_rank + rot:
        raise KernelError("attention_expanded: q, qr, pool and out must be bfloat16 rows that fit together")
    lib = lib_for(dim, rot, vdim)
    c = torch.empty((keys, width), dtype=q.dtype, device=q.device)
    core.check(lib.ib_gather_latents(pool.data_ptr(), c.data_ptr(), ctx.cu_rows.data_ptr(), ctx.q_start.data_ptr(),
                                     tables.data_ptr(), tables.shape[1], ctx.n_entries, page_size, num_pages, int(window),
                                     width, keys, rt.err.data_ptr(), core.stream_ptr(q)), "gather_latents")
    kv = w_kv(c[:, :kv_rank])
    core.check(lib.ib_attention_expanded(
        q.data_ptr(), q.stride(0), qr.data_ptr(), c.data_ptr(), width, kv_rank, kv.data_ptr(), kv.stride(0), heads * dim,
        keys, out.data_ptr(), out.stride(0), ctx.cu_rows.data_ptr(), ctx.q_start.data_ptr(), ctx.n_entries, N,
        ctx.max_rows_per_entry, heads, int(window), float(scale), sink.data_ptr() if sink is not None else None,
        gate.data_ptr() if gate is not None else None, gate.stride(0) if gate is not None else 0, rt.err.data_ptr(),
        core.stream_ptr(q)), "attention_expanded")
