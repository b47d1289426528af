"""Launcher of the float32 attention kernel (csrc/attention_f32.cu) and the choice between it and the plain one."""

from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p

import torch

from . import build
from . import lib as K
from .sources import ATTENTION_F32_HEAD_DIMS

FEW_ROWS = 8        # packed rows (tokens x query heads of a key head) a request may bring to have its keys shared out
_libs = {}


def _lib(head_dim: int):
    l = _libs.get(head_dim)
    if l is None:
        l = build.load_library("attention_f32.cu", (f"-DHEAD_DIM={head_dim}",))
        P, I, L, F = c_void_p, c_int, c_longlong, c_float
        l.llm_attention_f32.argtypes = [P, P, P, P, P, L, I, I, I, I, P, P, P, I, I, I, I, F, I, P]
        l.llm_attention_f32.restype = c_int
        _libs[head_dim] = l
    return l


def takes(q: torch.Tensor, out: torch.Tensor, cache: K.CacheView) -> bool:
    """All float32, a head size the kernel is built for, and everything on 16-byte boundaries."""
    return (q.dtype == out.dtype == cache.dtype == torch.float32 and cache.head_dim in ATTENTION_F32_HEAD_DIMS
            and cache.v_dim == cache.head_dim and cache.kv_heads <= 65535 and cache.page_stride % 4 == 0 and q.is_contiguous() and out.is_contiguous()
            and (q.data_ptr() | out.data_ptr() | cache.k_ptr | cache.v_ptr) % 16 == 0)


def run(ctx, q: torch.Tensor, out: torch.Tensor, cache: K.CacheView, heads: int, scale: float, window: int) -> None:
    """Causal softmax attention of the step's rows (`window` 0: every key).  Which kernel runs hangs on types, sizes
    and alignment of the model's own buffers only, not on how a step is cut, so neither does a result's last bit."""
    if not takes(q, out, cache):
        K.attention_plain(q, out, cache, ctx.positions, ctx.row_seq, heads, ctx.n_tokens, scale, window, ctx.stream)
        return
    group = heads // cache.kv_heads
    few = any(n * group <= FEW_ROWS for n in ctx.host_q_len)
    K._check(_lib(cache.head_dim).llm_attention_f32(
        q.data_ptr(), out.data_ptr(), cache.k_ptr, cache.v_ptr, cache.block_table.data_ptr(), cache.page_stride,
        cache.table_stride, cache.page_tokens, cache.kv_heads, cache.head_dim, ctx.seq_q_start.data_ptr(),
        ctx.seq_q_len.data_ptr(), ctx.seq_kv_len.data_ptr(), ctx.n_seqs, ctx.max_q_len, 1 if few else 0, heads, scale,
        window, ctx.stream), "attention_f32")
