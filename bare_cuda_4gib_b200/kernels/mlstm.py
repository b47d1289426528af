"""Launchers of `csrc/mlstm.cu`: the gates and running maximum of an mLSTM head, the float32
operands for the state scan, and the quotient, unit norm and gate after it."""

from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import build
from .lib import _check, _dev, _ptr, dtype_code, sm_count

_lib = None


def lib():
    global _lib
    if _lib is None:
        l = build.load_library("mlstm.cu")
        P, I, L, F = c_void_p, c_int, c_longlong, c_float
        l.llm_mlstm_gates.argtypes = [P, L, I, I, P, P, I, F, P, P, P, P, P, P, P, I, I, P]
        l.llm_mlstm_operands.argtypes = [P, I, L, I, I, I, P, P, P, P, P, I, I, I, I, I, P]
        l.llm_mlstm_finish.argtypes = [P, P, P, P, L, P, L, I, I, I, I, I, F, P]
        l.llm_mlstm_step.argtypes = [P, I, L, I, I, I, I, P, L, I, I, P, P, F, P, P, P, P, L, P, P, P, I, I, I, I, I, F, F, P]
        for name in ("llm_mlstm_gates", "llm_mlstm_operands", "llm_mlstm_finish", "llm_mlstm_step"):
            getattr(l, name).restype = c_int
        _lib = l
    return _lib


def gates(ctx, z: torch.Tensor, i_col: int, f_col: int, i_bias: torch.Tensor, f_bias: torch.Tensor, cap: float,
          m_state: torch.Tensor, coef: torch.Tensor, heads: int, log_decay: Optional[torch.Tensor] = None,
          weight: Optional[torch.Tensor] = None) -> None:
    """z [rows, columns] float32 holds the gates' projections (input gate of head h at column
    i_col + h, forget gate at f_col + h); coef [rows, heads, 4] float32 receives (decay, input
    weight, exp(-m), m) per new token; m_state [slots + 1, heads] carries m between steps.  `log_decay` and `weight` [rows,
    heads] float32 (both or neither) receive the decay's logarithm and the input weight for `chunked`."""
    _dev(z, i_bias, f_bias, m_state, coef)
    if z.dtype != torch.float32 or m_state.dtype != torch.float32 or coef.dtype != torch.float32:
        raise TypeError("mlstm gates: projections, state and coefficients must be float32")
    _check(lib().llm_mlstm_gates(z.data_ptr(), z.stride(0), i_col, f_col, i_bias.data_ptr(), f_bias.data_ptr(),
                                 dtype_code(i_bias.dtype), float(cap), m_state.data_ptr(), coef.data_ptr(), _ptr(log_decay), _ptr(weight),
                                 ctx.seq_slot.data_ptr(), ctx.seq_q_start.data_ptr(), ctx.seq_q_len.data_ptr(),
                                 ctx.n_seqs, heads, ctx.stream), "mlstm_gates")


def operands(ctx, u: torch.Tensor, q_col: int, k_col: int, v_col: int, coef: torch.Tensor, qf, kf, decay, vf,
             heads: int, dk: int, dv: int, dvp: int) -> None:
    _dev(u, coef, qf, kf, decay, vf)
    _check(lib().llm_mlstm_operands(u.data_ptr(), dtype_code(u.dtype), u.stride(0), q_col, k_col, v_col, coef.data_ptr(),
                                    qf.data_ptr(), kf.data_ptr(), decay.data_ptr(), vf.data_ptr(), ctx.n_tokens, heads,
                                    dk, dv, dvp, ctx.stream), "mlstm_operands")


def finish(ctx, scanned: torch.Tensor, coef: torch.Tensor, norm_w: torch.Tensor, gate: torch.Tensor, out: torch.Tensor,
           heads: int, dv: int, dvp: int, eps: float) -> None:
    _dev(scanned, coef, norm_w, gate, out)
    _check(lib().llm_mlstm_finish(scanned.data_ptr(), coef.data_ptr(), norm_w.data_ptr(), gate.data_ptr(),
                                  gate.stride(0), out.data_ptr(), out.stride(0), dtype_code(out.dtype), ctx.n_tokens,
                                  heads, dv, dvp, float(eps), ctx.stream), "mlstm_finish")


def chunked_takes(dk: int, dv: int) -> bool:
    """Sizes the walk in chunks on the tensor cores is built for (csrc/mlstm_chunked.cu, a library per pair)."""
    return dk % 16 == 0 and 16 <= dk <= 256 and dv % 16 == 0 and 16 <= dv <= 1024


MAX_REQUESTS = 65535      # of the walk in chunks: they are a grid's third axis (the scan's first)


def chunks_pay(q_len, heads: int, dk: int, dv: int) -> bool:
    """Whether the walk in chunks takes less time than operands and scan for portions of these lengths (microseconds on one B200).

    A request's blocks (one per head and 16 value columns, and one more) take about 14 a chunk however few tokens it holds,
    a block an SM, so many short portions, and single tokens beside a portion, are better off with the scan, which takes
    about 0.145 a token at 16 heads of 128 x 128, 0.16 for every step of the longest chain and 1 a request.  Measured at that size,
    chunks / scan: one portion of 24 tokens 15.2 / 16.7, of 64 15.6 / 30.6, of 2,048 214 / 487; two of 32 29.7 / 21.5, two of 64
    29.9 / 35.0; eight of 32 114 / 51, of 64 115 / 90, of 128 118 / 167; 256 tokens beside four single ones 85 / 120, beside eight
    141 / 123, beside 24 365 / 141; 1,024 beside eight 220 / 295, beside 24 445 / 342."""
    if len(q_len) > MAX_REQUESTS:
        return False
    blocks, tokens = heads * (-(-dv // 16) + 1), 128 if dk <= 128 else 64
    chunks = [-(-n // tokens) for n in q_len]
    walk = 2.0 + 14.0 * max(max(chunks), -(-sum(chunks) * blocks // sm_count()))
    scan = 8.0 + 0.145 * sum(q_len) * (heads * dk * dv) / (16 * 128 * 128) + 0.16 * max(q_len) + 1.0 * len(q_len)
    return walk < 0.95 * scan


_chunked_libs = {}


def chunked_lib(dk: int, dv: int):
    l = _chunked_libs.get((dk, dv))
    if l is None:
        l = build.load_library("mlstm_chunked.cu", (f"-DML_DK={dk}", f"-DML_DV={dv}"))
        P, I, L, F = c_void_p, c_int, c_longlong, c_float
        l.llm_mlstm_chunked.argtypes = [P, P, P, L, P, P, P, P, F, P, P, P, I, I, I, I, P]
        l.llm_mlstm_chunked.restype = c_int
        _chunked_libs[(dk, dv)] = l
    return l


def chunked(ctx, u: torch.Tensor, q_col: int, k_col: int, v_col: int, log_decay: torch.Tensor, weight: torch.Tensor,
            state: torch.Tensor, out: torch.Tensor, heads: int, dk: int, dv: int, q_scale: float) -> None:
    """Every request's portion in chunks (of 128 tokens, 64 for keys of more than 128 entries): q, k and v are read from the
    bfloat16 projection u; [S | n] float32 [slots, heads, dk, dv + 4] is read and left as after the portion; out [rows, heads *
    (dv + 4)] float32 = [S^T q | n . q | 0] * q_scale."""
    _dev(u, log_decay, weight, state, out)
    if (u.dtype != torch.bfloat16 or state.dtype != torch.float32 or out.dtype != torch.float32 or not out.is_contiguous()
            or state.shape[-1] != dv + 4 or out.shape[-1] != heads * (dv + 4)):
        raise TypeError("mlstm chunked: element types or layout not as the kernel needs")
    base = u.data_ptr()
    _check(chunked_lib(dk, dv).llm_mlstm_chunked(
        base + 2 * q_col, base + 2 * k_col, base + 2 * v_col, u.stride(0), weight.data_ptr(), log_decay.data_ptr(),
        state.data_ptr(), out.data_ptr(), float(q_scale), ctx.seq_slot.data_ptr(), ctx.seq_q_start.data_ptr(),
        ctx.seq_q_len.data_ptr(), ctx.n_seqs, heads, dk, dv, ctx.stream), "mlstm_chunked")


STEP_MAX_VALUE_COLUMNS = 288      # vdim + pad the one-token kernel keeps per warp
STEP_MAX_SHARED = 48 * 1024


def step_takes(dk: int, dvp: int) -> bool:
    return dvp <= STEP_MAX_VALUE_COLUMNS and (2 * dk + 9 * dvp + 8) * 4 <= STEP_MAX_SHARED


def step(ctx, u: torch.Tensor, q_col: int, k_col: int, v_col: int, g_col: int, z: torch.Tensor, i_col: int, f_col: int,
         i_bias: torch.Tensor, f_bias: torch.Tensor, cap: float, state: torch.Tensor, m_state: torch.Tensor,
         norm_w: torch.Tensor, out: torch.Tensor, heads: int, dk: int, dv: int, dvp: int, q_scale: float, eps: float) -> None:
    """All of a head's work for a step of one token per request: gates, m, [S | n] updated in place,
    quotient, unit norm, weight and gate."""
    _dev(u, z, i_bias, f_bias, state, m_state, norm_w, out)
    if z.dtype != torch.float32 or state.dtype != torch.float32 or m_state.dtype != torch.float32:
        raise TypeError("mlstm step: gate projections and states must be float32")
    _check(lib().llm_mlstm_step(u.data_ptr(), dtype_code(u.dtype), u.stride(0), q_col, k_col, v_col, g_col, z.data_ptr(),
                                z.stride(0), i_col, f_col, i_bias.data_ptr(), f_bias.data_ptr(), float(cap),
                                state.data_ptr(), m_state.data_ptr(), norm_w.data_ptr(), out.data_ptr(), out.stride(0),
                                ctx.seq_slot.data_ptr(), ctx.seq_q_start.data_ptr(), ctx.seq_q_len.data_ptr(), ctx.n_seqs,
                                heads, dk, dv, dvp, float(q_scale), float(eps), ctx.stream), "mlstm_step")
