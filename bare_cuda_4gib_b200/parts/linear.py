"""A bias-free linear projection y = x W^T with W stored [out features, in features], as
cuongvng/bare-cuda-4gib keeps every matrix (engine/include/llm/kernels.h:48-57).

It is a building brick of mixers, feed-forwards and the head rather than a family of its own.
Which kernel runs is decided here from the element types: float32 anywhere, or a size the fast
kernel refuses, goes to the plain kernel; bfloat16 activations against bfloat16 weights go to the
tensor-core kernel (see `kernels.gemm`).
"""

from __future__ import annotations

from typing import Optional

import torch

from ..kernels import lib as K


class Linear:
    def __init__(self, weight: torch.Tensor, name: str):
        self.weight = weight.contiguous()
        self.name = name
        self.out_features, self.in_features = weight.shape
        self.fast = None  # set by prepare() when the tensor-core kernel takes this matrix
        self.few = False  # whether the few-token fused kernel takes this matrix

    def prepare(self, act_dtype: torch.dtype) -> None:
        if act_dtype == torch.bfloat16 and self.weight.dtype == torch.bfloat16 and self.weight.is_cuda:
            from ..kernels import gemm
            self.fast = gemm.plan_for(self.weight)
            from ..kernels import gemv
            self.few = gemv.supports(self.weight)

    def reserve(self, ctx, buffer: str) -> None:
        """For a product whose result is added into the residual stream: asks the workspace for what a step of a few rows will leave
        in `buffer`, so that the first such step does not have to allocate it."""
        if self.fast is not None and ctx.use_fast_gemm:
            from ..kernels import gemm, gemv
            gemm.reserve_partials(ctx.ws, self.fast, buffer, lambda rows: self.few and gemv.takes(rows, self.in_features))

    def forward(self, ctx, a, rows: int, out_dtype: torch.dtype, buffer: str,
                allow_partials: bool = False, swiglu: bool = False, epilogue=None,
                glu: Optional[str] = None) -> Optional[K.Partials]:
        """a[:rows] @ W^T into the workspace buffer `buffer`.  With `swiglu`, W is [gate; up] and
        the result is silu(gate) * up of half the width (fused where the kernel can).  `a` is a
        matrix or a `LazyNorm`.  `epilogue` (`AddTo`, `RotateAndCache`) names what the caller will
        do with the result next: a kernel that can do it itself does, and None comes back; from
        every other kernel the plain result comes back and the epilogue stays the caller's.
        `glu` names the activation of a gated product ("silu" is what `swiglu` asks for)."""
        activation = glu or "silu"
        swiglu = swiglu or glu is not None
        width = self.out_features // 2 if swiglu else self.out_features
        if self.few and ctx.use_fast_gemm:
            from ..kernels import gemv
            if gemv.takes(rows, self.in_features):
                return gemv.run(ctx, self.weight, a, rows, out_dtype, buffer, swiglu, epilogue, activation)
        if self.fast is not None and ctx.use_fast_gemm:
            from ..kernels import gemm
            kind = gemm.cluster_kind(self.fast, rows, out_dtype, swiglu, epilogue)
            if kind is not None:
                return gemm.run_cluster(ctx, self.fast, kind, a, rows, out_dtype, buffer, epilogue, activation)
            return gemm.run(ctx, self.fast, a, rows, out_dtype, buffer, allow_partials, swiglu, epilogue, activation)
        a = K.materialize(a)
        if swiglu:
            full = ctx.ws.get(buffer + ".gate_up", (rows, self.out_features), out_dtype)
            K.matmul_plain(a, self.weight, full, rows, ctx.stream)
            out = ctx.ws.get(buffer, (rows, width), out_dtype)
            K.glu(K.Partials(full), out, rows, activation, ctx.stream)
            return K.Partials(out)
        out = ctx.ws.get(buffer, (rows, width), out_dtype)
        K.matmul_plain(a, self.weight, out, rows, ctx.stream)
        return K.Partials(out)
