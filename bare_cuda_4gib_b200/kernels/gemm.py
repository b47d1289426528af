"""Launcher of the tcgen05 bfloat16 matrix product (csrc/gemm_tcgen05.cu): tensor maps, choice of
the token tile and of the K split, and the device error word that bounded waits report to."""

from __future__ import annotations

import ctypes
import functools
import os
from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Dict, Optional, Tuple

import torch

from ..errors import KernelLaunchError
from . import build
from .lib import DT_BF16, DT_F32, AddTo, glu_defines, LazyNorm, Partials, Prenormed, RotateAndCache, _check, _ptr, sm_count

BM, BK = 128, 64
SPLIT_MAX_ROWS = 256          # steps with more rows never split K
_libs = {}
_error_word: Optional[torch.Tensor] = None


def lib(activation: str = "silu"):
    """The library whose gated products (mode 1) apply `activation` to the gate."""
    _lib = _libs.get(activation)
    if _lib is None:
        l = build.load_library("gemm_tcgen05.cu", glu_defines(activation))      # the gate's activation is a library's own
        P, I, L, F = c_void_p, c_int, c_longlong, c_float
        l.llm_gemm_tensor_map.argtypes = [P, P, L, L, L, I]
        l.llm_gemm_tensor_map.restype = c_int
        l.llm_gemm_bf16.argtypes = [P, P, P, I, I, I, I, L, L, I, I, I, I, I, I, P, I, L, F, F, P, L, P, I, P, L, P, P]
        l.llm_gemm_bf16.restype = c_int
        l.llm_gemm_grouped_bf16.argtypes = [P, P, P, I, I, I, I, L, I, I, I, I, P, P, P, P, P, P]
        l.llm_gemm_grouped_bf16.restype = c_int
        l.llm_gemm_cluster.argtypes = [P, P, I, I, I, I, I, I, P, I, L, I, P, I, L, F, F, P, L, P, I, P, L, P, P, P, L, I, I, I, I,
                                       P, P, P, I, I, P, P]
        l.llm_gemm_cluster.restype = c_int
        l.llm_gemm_qkv.argtypes = [P, P, P, I, I, L, I, P, I, L, F, F, P, L, P, P, P, L, I, I, I, I, P, P, I, I, P, P]
        l.llm_gemm_qkv.restype = c_int
        l.llm_turn_table.argtypes = [P, P, P, L, I, I, P]
        l.llm_turn_table.restype = c_int
        _lib = _libs[activation] = l
    return _lib


def error_word(device) -> torch.Tensor:
    global _error_word
    if _error_word is None:
        _error_word = torch.zeros(1, dtype=torch.int32, device=device)
    return _error_word


def check_errors() -> None:
    """Reads the device error word (synchronises); raises if a kernel gave up on a wait."""
    if _error_word is not None:
        code = int(_error_word.item())
        if code:
            _error_word.zero_()
            role = {1: "gemm TMA producer", 2: "gemm MMA issuer", 3: "gemm epilogue", 11: "attention loader",
                    12: "attention MMA issuer", 13: "attention softmax",
                    14: "attention (shared memory not 1024-byte aligned)", 21: "few-token product, producer",
                    22: "few-token product, consumer", 4: "gemm cluster exchange", 31: "decode attention"}.get(code, f"code {code}")
            raise KernelLaunchError(f"a kernel gave up ({role}): a bounded wait ran out; the result is invalid")


def supports(weight: torch.Tensor) -> bool:
    n, k = weight.shape
    return (weight.dtype == torch.bfloat16 and weight.is_cuda and weight.is_contiguous()
            and k % 8 == 0 and weight.data_ptr() % 16 == 0)


def tensor_map(base_ptr: int, rows: int, cols: int, row_stride: int, box_rows: int) -> ctypes.Array:
    buf = (ctypes.c_ubyte * 128)()
    _check(lib().llm_gemm_tensor_map(ctypes.addressof(buf), base_ptr, rows, cols, row_stride, box_rows),
           "gemm tensor map")
    return buf


class GemmPlan:
    """A weight matrix ready for the kernel: its tensor map and the maps of the activation buffers
    it has been multiplied with."""

    def __init__(self, weight: torch.Tensor):
        self.weight = weight
        self.n, self.k = weight.shape
        self.weight_maps: Dict[int, ctypes.Array] = {}
        self.map_w = self.weight_map(BM)
        self.act_maps: Dict[Tuple[int, int, int], ctypes.Array] = {}

    def weight_map(self, box_rows: int) -> ctypes.Array:
        m = self.weight_maps.get(box_rows)
        if m is None:
            m = tensor_map(self.weight.data_ptr(), self.n, self.k, self.k, box_rows)
            self.weight_maps[box_rows] = m
        return m

    def act_map(self, a: torch.Tensor, bn: int) -> ctypes.Array:
        """`bn`: rows of the box (the token tile)."""
        key = (a.data_ptr(), bn, a.stride(0))
        m = self.act_maps.get(key)
        if m is None:
            esize = a.element_size()
            storage_left = a.untyped_storage().nbytes() - a.storage_offset() * esize
            # rows that lie wholly inside the storage (`a` may be a column view, whose last row ends early)
            capacity = max(a.shape[0], (storage_left // esize - self.k) // a.stride(0) + 1)
            m = tensor_map(a.data_ptr(), capacity, self.k, a.stride(0), bn)
            self.act_maps[key] = m
        return m


def plan_for(weight: torch.Tensor) -> Optional[GemmPlan]:
    if not supports(weight):
        return None
    return GemmPlan(weight)


def token_tile(rows: int) -> int:
    for bn in (16, 32, 64, 128):
        if rows <= bn:
            return bn
    # beyond 128 rows the tile follows the row count in steps of 16: a step of 129 to 160 rows ran a tenth
    # faster than with a tile of 256 tokens, most of which were padding
    return min(256, -(-rows // 16) * 16)


def choose_splits(rows: int, n: int, k: int, bn: int) -> int:
    """How many thread blocks share the K range of one output tile: enough to put about two
    blocks on every SM, at least four 64-wide K blocks each, and partial results (float32, written
    and read back through the L2 cache, not HBM) of at most about the weight's own bytes."""
    if rows > SPLIT_MAX_ROWS:
        return 1
    tiles = -(-n // BM) * -(-rows // bn)
    k_blocks = -(-k // BK)
    splits = min(k_blocks // 4, (2 * sm_count()) // tiles, max(1, k // (4 * rows)))
    splits = max(1, splits)
    per = -(-k_blocks // splits)
    return -(-k_blocks // per)


def max_splits(n: int, k: int) -> int:
    """The most blocks `choose_splits` ever puts on one output tile of an [n, k] weight, whatever
    the number of rows: the scratch for partial results is sized for it once, so that its address
    never changes under a captured graph."""
    return max(1, min(-(-k // BK) // 4, (2 * sm_count()) // -(-n // BM)))


TOKENS_ON_ROWS_ABOVE = 240    # steps with more rows put 128 tokens on the MMA rows (orientation 1); measured: a step of TinyLlama's sizes
                              # with 256 rows takes 1,657 us that way and 2,249 with the weights on the MMA rows, one of 240 rows 1,653
                              # that way and 1,349 with the cluster product
# The SwiGLU product changes over earlier: with the weights on the MMA rows a block holds only 64
# outputs, so from a few dozen tokens on the other orientation's wider tiles measured faster
# (TinyLlama's feed-forward at 64 / 96 / 128 / 256 tokens: 13.3 / 13.2 / 13.4 / 16.2 us that way against 16.8 / 20.2 / 23.2 / 27.7;
# 11,008 x 4,096 at 64 / 128: 35.7 / 36.4 against 42.5 / 53.0).  Up to here the cluster product takes it.
SWIGLU_TOKENS_ON_ROWS_ABOVE = 60


def tile_cost(rows: int, n_out: int, bn: int, swiglu: bool) -> float:
    """What a product in tiles of `bn` weight rows takes, in tiles of 256 (see `feature_tile`)."""
    tiles = -(-rows // BM) * -(-n_out // (bn // 2 if swiglu else bn))
    cost = -(-tiles // sm_count()) * (bn / 256.0 + 0.12)
    return cost * 0.88 if bn >= 192 and tiles > sm_count() else cost


def whole_heads_pay(rows: int, n_out: int, end: RotateAndCache) -> bool:
    """Whether turning heads in the product beats a kernel behind it: its tiles have to hold whole heads, which must not
    cost more than the best tile does."""
    d = end.cache.head_dim
    return tile_cost(rows, n_out, feature_tile(rows, n_out, False, d), False) <= tile_cost(rows, n_out, feature_tile(rows, n_out, False), False)


def feature_tile(rows: int, n_out: int, swiglu: bool, multiple: int = 0) -> int:
    """Orientation 1: how many weight rows a tile takes (a multiple of 16 up to 256; of 32 with
    SwiGLU, whose tile is half gate rows and half up rows).  Every SM works through
    ceil(tiles / SMs) tiles and a tile's time grows with its width, so the product of the two is
    minimised; a small fixed cost per tile breaks ties towards wider tiles.  Wide tiles (192 rows
    and more) of a product with more tiles than SMs run in the persistent kernel, whose tiles count an eighth
    less (no pipeline refill per tile, the epilogue off the critical path).  Of 32 sizes (eight layers of 2,048 to 12,288 outputs, 300 to
    2,048 rows) the tile this picks is within 8 % of the best one, but for 2,048 x 2,048 at 2,048 rows (256: 26.7 us, 128: 24.0).
    `multiple`: the tile has to be a multiple of this (whole heads)."""
    forced = os.environ.get("BARE_CUDA_B200_GEMM_BN")     # experiments only
    if forced and not multiple:
        return int(forced)
    return _feature_tile(rows, n_out, swiglu, multiple)


@functools.lru_cache(maxsize=4096)
def _feature_tile(rows: int, n_out: int, swiglu: bool, multiple: int) -> int:
    """The search itself, once for the same sizes: it takes 3.4 us on the host, and a layer of a step asks up to six times."""
    step = 32 if swiglu else 16
    best, best_cost = 256, None
    for bn in range(256, 63, -step):
        if multiple and bn % multiple:
            continue
        # between 160 and 256 a tile is too big for two blocks per SM with three stages each: only SwiGLU tiles (two stages) use
        # the range.  (2,048 rows, adding end, tiles of 128 / 192 / 256: 2,048 x 5,632 47.9 / 59.8 / 48.2 us, 4,096 x 4,096 74.4 / 69.8 /
        # 67.3; one of the measured products would gain: 12,288 x 4,096 254 / 170 / 187.)
        if not swiglu and 160 < bn < 256:
            continue
        cost = tile_cost(rows, n_out, bn, swiglu)
        if best_cost is None or cost < best_cost - 1e-9:
            best, best_cost = bn, cost
    return best


NO_EXTRA = (0, 0, 0, 0.0, 0.0, 0, 0, 0, 0, 0, 0)     # no row factor on the way in, nothing prepared on the way out


def takes_prenormed(rows: int, swiglu: bool) -> bool:
    """Whether a step of `rows` rows runs in the orientation whose epilogue can apply a norm's
    factor per row (tokens on the MMA rows), so that the product can take a `LazyNorm` that a
    product before it prepared."""
    return rows > (SWIGLU_TOKENS_ON_ROWS_ABOVE if swiglu else TOKENS_ON_ROWS_ABOVE)


def turns(end: RotateAndCache, n_out: int) -> bool:
    """Whether the many-token product's epilogue can turn the heads and write the cache: angles that the step's layers
    share, whole heads to a tile, 16-byte stores everywhere."""
    c, q = end.cache, end.q_out
    return ((end.inv_freq is None or end.angles is not None) and c.dtype == q.dtype == torch.bfloat16 and c.v_dim == c.head_dim and c.head_dim in (32, 64, 128, 256)
            and (end.q_heads + 2 * c.kv_heads) * c.head_dim == n_out and q.stride(0) % 8 == 0 and c.page_stride % 8 == 0
            and (q.data_ptr() | c.k_ptr | c.v_ptr) % 16 == 0)


def turn_table(ctx, l, end: RotateAndCache, rows: int) -> Tuple[int, int]:
    """The step's table of (cosine, sine) pairs for these angles (address, row stride), made by the first layer that asks
    for it."""
    if end.inv_freq is None:
        return 0, 0
    half = end.cache.head_dim // 2
    key = ("turn_table", end.angles, half)
    table = ctx.extras.get(key)
    if table is None:
        table = ctx.ws.get(f"turn_table {end.angles}", (half, 2 * ctx.ws.max_rows), torch.float32, max_rows=half)
        _check(l.llm_turn_table(end.positions.data_ptr(), end.inv_freq.data_ptr(), table.data_ptr(), ctx.ws.max_rows, rows, half,
                                ctx.stream), "turn_table")
        ctx.extras[key] = table
    return table.data_ptr(), ctx.ws.max_rows


def run(ctx, plan: GemmPlan, a, rows: int, out_dtype: torch.dtype, buffer: str,
        allow_partials: bool, swiglu: bool, epilogue=None, activation: str = "silu") -> Optional[Partials]:
    """`a`: a bfloat16 matrix, or a `LazyNorm` whose `prenormed` a product before this one left
    (`takes_prenormed` steps only).  `epilogue`: with an `AddTo` whose norm can be prepared, a
    many-token step adds the product into the float32 residual stream itself, leaves bfloat16(new
    residual * that norm's weight) and the rows' sums of squares for the product that reads the
    norm next (`ctx.prenormed`), and None comes back; otherwise the plain result comes back and the
    epilogue stays the caller's."""
    extra_in = NO_EXTRA[:5]
    if isinstance(a, LazyNorm):
        pre = a.prenormed
        if pre is None or a.row_index is not None or not takes_prenormed(rows, swiglu):
            a = a.materialize()
        else:
            extra_in = (pre.sq.data_ptr(), pre.items, pre.sq.stride(0), float(pre.x.shape[-1]), a.eps)
            a = pre.x
    ctx.prenormed = None
    if a.dtype != torch.bfloat16 or a.stride(-1) != 1 or a.shape[-1] != plan.k or a.data_ptr() % 16 or a.stride(0) % 8:
        raise KernelLaunchError(f"gemm_tcgen05: activations {tuple(a.shape)} {a.dtype} do not fit weight "
                                f"[{plan.n}, {plan.k}]")
    err = error_word(a.device)
    l = lib(activation if swiglu else "silu")
    code = DT_BF16 if out_dtype == torch.bfloat16 else DT_F32
    if takes_prenormed(rows, swiglu):
        n_out = plan.n // 2 if swiglu else plan.n
        if isinstance(epilogue, RotateAndCache) and not swiglu and turns(epilogue, n_out) and whole_heads_pay(rows, n_out, epilogue):
            c, q = epilogue.cache, epilogue.q_out
            bn = feature_tile(rows, n_out, False, c.head_dim)
            _check(l.llm_gemm_qkv(ctypes.addressof(plan.weight_map(bn)), ctypes.addressof(plan.act_map(a, BM)), q.data_ptr(), rows,
                                  plan.k, q.stride(0), bn, *extra_in, *turn_table(ctx, l, epilogue, rows), c.k_ptr, c.v_ptr,
                                  c.block_table.data_ptr(), c.page_stride, c.table_stride, c.page_tokens, c.kv_heads, c.head_dim,
                                  epilogue.positions.data_ptr(), epilogue.row_seq.data_ptr(), epilogue.q_heads,
                                  1 if epilogue.write_cache else 0, err.data_ptr(), ctx.stream), "gemm_tcgen05 (q, k, v)")
            return None
        bn = feature_tile(rows, n_out, swiglu)
        extra_out = NO_EXTRA[5:]
        out, then = None, None
        if (isinstance(epilogue, AddTo) and epilogue.then_norm is not None and not swiglu
                and epilogue.residual.dtype == torch.float32 and epilogue.residual.shape[-1] == n_out
                and epilogue.residual.stride(-1) == 1 and epilogue.residual.stride(0) % 4 == 0 and n_out % 4 == 0
                and epilogue.residual.data_ptr() % 16 == 0):
            then = epilogue.then_norm
            pre_w = then.tensors["weight"]
            if pre_w.is_cuda and pre_w.data_ptr() % 16 == 0 and pre_w.dtype in (torch.float32, torch.bfloat16):
                out = epilogue.residual
                f_tiles = -(-n_out // bn)
                pre_x = ctx.ws.get("prenormed.rows.x", (rows, n_out), torch.bfloat16)
                # one row of parts per feature tile (a tile is at least 64 wide), as long as the largest step
                most_tiles = -(-n_out // 64)
                pre_sq = ctx.ws.get("prenormed.rows.sq", (most_tiles, ctx.ws.max_rows), torch.float32, max_rows=most_tiles)
                extra_out = (pre_x.data_ptr(), pre_x.stride(0), pre_w.data_ptr(),
                             DT_BF16 if pre_w.dtype == torch.bfloat16 else DT_F32, pre_sq.data_ptr(), pre_sq.stride(0))
        fused = out is not None
        if not fused:
            out = ctx.ws.get(buffer, (rows, n_out), out_dtype)
        _check(l.llm_gemm_bf16(ctypes.addressof(plan.weight_map(bn // 2 if swiglu else bn)),
                               ctypes.addressof(plan.act_map(a, BM)), out.data_ptr(), DT_F32 if fused else code, rows,
                               n_out, plan.k, out.stride(0), 0, 1, bn, 1 if swiglu else 0, 1, n_out if swiglu else 0,
                               1 if fused else 0, *extra_in, *extra_out, err.data_ptr(), ctx.stream),
               "gemm_tcgen05 (tokens on rows)")
        if fused:
            ctx.prenormed = Prenormed(then, pre_x, pre_sq, f_tiles)
            return None
        return Partials(out)
    bn = token_tile(rows)
    if swiglu:
        inter = plan.n // 2
        out = ctx.ws.get(buffer, (rows, inter), out_dtype)
        if -(-inter // (BM // 2)) * -(-rows // bn) >= sm_count():
            # 64 gate rows and the matching 64 up rows share a block's 128 MMA rows: SwiGLU in the
            # epilogue and no partial results, when that alone gives every SM a block
            _check(l.llm_gemm_bf16(ctypes.addressof(plan.weight_map(BM // 2)), ctypes.addressof(plan.act_map(a, bn)),
                                   out.data_ptr(), code, rows, inter, plan.k, out.stride(0), 0, 1, bn, 1, 0, inter, 0,
                                   *NO_EXTRA, err.data_ptr(), ctx.stream), "gemm_tcgen05 (swiglu)")
            return Partials(out)
        # a narrow feed-forward: stream [gate; up] as one product split over K so that every SM takes
        # part, and add the partial results inside the SwiGLU kernel
        from . import lib as K
        full = run(ctx, plan, a, rows, torch.float32, buffer + ".gate_up", True, False)
        K.glu(full, out, rows, activation, ctx.stream)
        return Partials(out)
    splits = choose_splits(rows, plan.n, plan.k, bn) if (allow_partials and out_dtype == torch.float32) else 1
    if splits > 1:
        out = _partials(ctx.ws, plan, buffer, splits, rows)
        stride = out.stride(0)
    else:
        out = ctx.ws.get(buffer, (rows, plan.n), out_dtype)
        stride = 0
    _check(l.llm_gemm_bf16(ctypes.addressof(plan.map_w), ctypes.addressof(plan.act_map(a, bn)), out.data_ptr(),
                           DT_BF16 if out_dtype == torch.bfloat16 else DT_F32, rows, plan.n, plan.k,
                           out.stride(-2), stride, splits, bn, 0, 0, 0, 0, *NO_EXTRA, err.data_ptr(), ctx.stream),
           "gemm_tcgen05")
    return Partials(out, splits)


# ------------------------------------------------------------------ a few dozen tokens, ends fused in
CL_ADD, CL_SWIGLU, CL_ROPE = 1, 2, 3
# Measured, a whole step of TinyLlama's 22 layers, product + norm + rotation kernels against this: 30 rows 1,094 -> 881 us,
# 40 rows 1,189 -> 959, 64 rows 1,207 -> 950, 96 rows 1,341 -> 1,013, 130 rows 1,570 -> 1,206, 180 rows 1,783 -> 1,298, 240
# rows 2,037 -> 1,349; eight layers of the Llama-3-8B sizes: 30 rows 1,014 -> 936, 64 rows 1,121 -> 1,065, 112 rows 1,219 -> 1,135, 144 rows
# 1,396 -> 1,338, 180 rows 1,789 -> 1,508, 240 rows 1,845 -> 1,612; of the Llama-2-7B sizes: 30 rows 848 -> 802, 64 rows 918 -> 877, 112 rows
# 1,048 -> 1,003, 144 rows 1,167 -> 1,141, 180 rows 1,559 -> 1,250, 240 rows 1,642 -> 1,516.  Above, tokens are on the MMA rows.
CLUSTER_MAX_ROWS = TOKENS_ON_ROWS_ABOVE
# A tile of 96 or 128 tokens would fill an SM's shared memory with one block (96 rows 1,971 us, 128 rows 3,084).
CLUSTER_TILE_ROWS = 64
# A gated product has enough tiles; with more rows than a tile's it runs with tokens on the MMA rows (TinyLlama's: 13.4 us up to 128 rows).
CLUSTER_GATED_ROWS = 64
# With so few rows that the few-token product (gemv.py) takes the layer's other products, what comes here is a down
# projection whose input does not fit beside its ring.  A small one gains (12 rows x 2,048 x 5,632, 23 MB, with the norm: 10.1 -> 7.7 us);
# for a large one, bound by its weights, the split product's deeper ring streamed them faster when the line was drawn (8 rows x 4,096 x
# 14,336, 117 MB, with the norm: 22.3 against 23.5 us; with elected issuers it is 24.9 against 21.6, and the line stands where it stood).
CLUSTER_FEW_ROWS, CLUSTER_FEW_BYTES = 24, 64 << 20
# Layers of a smaller inner size keep the kernels they had.  The kernel takes them (every block of a cluster has two K blocks
# whatever the size), but a product that adds its result itself hands nothing on, and callers that run a tiny model's block by
# itself at 25 to 64 rows expect its contribution un-added.
CLUSTER_MIN_K = 8 * BK


CLUSTER_MAX_SIZE = 8


def cluster_size(n_tiles: int, k: int) -> int:
    """Blocks that share a tile's K range: as many (1, 2, 4, 8) as two blocks an SM and two 64-wide K blocks each allow."""
    c = CLUSTER_MAX_SIZE
    while c > 1 and (n_tiles * c > 2 * sm_count() or -(-k // BK) < 2 * c):
        c //= 2
    return c


@functools.lru_cache(maxsize=4096)
def cluster_tile(rows: int, n_tiles: int, k: int) -> int:
    """Tokens of a tile: the rows dealt out evenly over as few tiles as hold them, in steps of 16.  49 to 64 rows go in two
    tiles where the blocks of a cluster still walk through at most 12 K blocks each: the exchange at a tile's end lengthens with
    its tokens (64 rows, one tile / two: 2,048 x 2,048 7.0 / 6.2 us, 2,048 x 5,632 10.6 / 9.3).  With longer walks the larger cluster of one tile wins:
    4,096 x 4,096 (16 K blocks in two tiles) 11.5 / 12.0, 6,144 x 4,096 (32) 16.0 / 17.1, 4,096 x 11,008 (43) 20.7 / 22.7."""
    tiles = -(-rows // CLUSTER_TILE_ROWS)
    if 48 < rows <= 64 and cluster_walk(2 * n_tiles, k) <= 12:
        tiles = 2
    return -(-rows // (16 * tiles)) * 16


def cluster_walk(n_tiles: int, k: int) -> int:
    """The 64-wide K blocks that a block of a cluster goes through."""
    return -(--(-k // BK) // cluster_size(n_tiles, k))


CLUSTER_LONG_WALK = 48


@functools.lru_cache(maxsize=4096)
def cluster_pays(rows: int, n_tiles: int, k: int) -> bool:
    """Whether the cluster product beats the split product and the kernel behind it, for `n_tiles` tiles of weight rows.  It does while
    its blocks walk through K quickly.  With wide layers and several token tiles the clusters are small and the walks
    long, and then the other product, whose one tile holds all tokens, is faster, until that tile leaves its ring too few
    stages (more than 160 tokens).  Microseconds with the kernel behind it, cluster / other: 12,288 x 4,096 (32 K blocks a walk) 64
    rows 24.9 / 26.6, (64) 128 rows 35.7 / 36.2, 192 rows 36.0 / 56.2, (64, and more blocks than two to an SM) 240 rows 65.2 / 65.6;
    4,096 x 11,008 (43) 128 rows 26.2 / 30.3, (86) 144 rows 37.7 / 31.2, 192 rows 40.4 / 49.1; 4,096 x 14,336 (56) 96 rows 29.7 / 32.7,
    (112) 144 rows 47.3 / 36.6, 192 rows 49.8 / 54.4, 240 rows 49.9 / 61.0.  (Drawn before the products' issuers were elected, when walks of 56
    and 64 K blocks were slower in a cluster: those now gain 1 to 9 % there.)"""
    tiles = n_tiles * -(-rows // cluster_tile(rows, n_tiles, k))
    walk = cluster_walk(tiles, k)
    if tiles > 2 * sm_count():
        return walk <= CLUSTER_LONG_WALK // 2
    return walk <= CLUSTER_LONG_WALK or (rows > 160 and walk <= 2 * CLUSTER_LONG_WALK) or rows > 200


def cluster_pays_gated(rows: int, n_tiles: int, k: int) -> bool:
    """The same for a gated product of `n_tiles` tiles of 64 outputs, against tokens on the MMA rows (which run it from 61 rows on).
    With long walks a block an SM and a few SMs with two take as long as two everywhere: it has to fill two thirds of the places.  Eight
    layers, 64 rows, cluster / tokens on rows: 11,008 x 4,096 (172 of 296 places) 923 / 873 us, 14,336 x 4,096 (224) 1,065 / 1,084; all of
    TinyLlama's (5,632 x 2,048, 16 K blocks a walk) 952 / 936 (1,112 / 1,147 before the issuers were elected)."""
    tiles = n_tiles * -(-rows // cluster_tile(rows, n_tiles, k))
    return rows <= SWIGLU_TOKENS_ON_ROWS_ABOVE or cluster_walk(tiles, k) <= CLUSTER_LONG_WALK or 3 * tiles >= 4 * sm_count()


def reserve_partials(ws, plan: GemmPlan, buffer: str, taken) -> None:
    """Asks for the buffer of partial results that a step of a few rows will need of a product that more rows send to the cluster
    product: otherwise no step before the first decode step asks for it (36 MB for 4,096 x 14,336).  `taken(rows)`: whether the
    few-token product runs that many rows."""
    if plan.k < CLUSTER_MIN_K or plan.n % 8 or 2 * plan.n * plan.k <= CLUSTER_FEW_BYTES:
        return
    few = [rows for rows in (8, 16, CLUSTER_FEW_ROWS) if not taken(rows)]
    if any(choose_splits(rows, plan.n, plan.k, token_tile(rows)) > 1 for rows in few):
        _partials(ws, plan, buffer, 1, 1)


def _partials(ws, plan: GemmPlan, buffer: str, splits: int, rows: int) -> torch.Tensor:
    """The [splits, rows, features] buffer for a product that splits K."""
    return ws.get(buffer + ".partials", (splits, rows, plan.n), torch.float32, max_rows=SPLIT_MAX_ROWS,
                  max_lead=max_splits(plan.n, plan.k))


def cluster_kind(plan: GemmPlan, rows: int, out_dtype, swiglu: bool, epilogue) -> Optional[int]:
    """Which of the cluster product's ends a call asks for, None where the kernel does not take it."""
    if plan.k < CLUSTER_MIN_K or not 0 < rows <= CLUSTER_MAX_ROWS or plan.n % 8 or (rows <= CLUSTER_FEW_ROWS and 2 * plan.n * plan.k > CLUSTER_FEW_BYTES):
        return None
    if swiglu:
        # (more rows: tokens on the MMA rows, one tile for 128 of them)
        return CL_SWIGLU if rows <= CLUSTER_GATED_ROWS and cluster_pays_gated(rows, -(-plan.n // BM), plan.k) else None
    if isinstance(epilogue, AddTo):
        r = epilogue.residual
        fits = (r.dtype == torch.float32 and r.shape[-1] == plan.n and r.stride(-1) == 1 and r.stride(0) % 4 == 0
                and r.data_ptr() % 16 == 0 and cluster_pays(rows, -(-plan.n // BM), plan.k))
        return CL_ADD if fits else None
    if isinstance(epilogue, RotateAndCache):
        c, q = epilogue.cache, epilogue.q_out
        fits = (c.dtype == q.dtype == torch.bfloat16 and c.v_dim == c.head_dim and c.head_dim % 8 == 0 and 128 % c.head_dim == 0
                and (epilogue.q_heads + 2 * c.kv_heads) * c.head_dim == plan.n and q.stride(0) % 4 == 0 and q.data_ptr() % 16 == 0
                and (c.k_ptr | c.v_ptr) % 8 == 0 and c.page_stride % 4 == 0 and cluster_pays(rows, -(-plan.n // BM), plan.k))
        return CL_ROPE if fits else None
    return None


def run_cluster(ctx, plan: GemmPlan, kind: int, a, rows: int, out_dtype: torch.dtype, buffer: str, epilogue=None,
                activation: str = "silu") -> Optional[Partials]:
    """The product with the end that `cluster_kind` named; None comes back where the epilogue consumed the result."""
    extra_in = NO_EXTRA[:5]
    if isinstance(a, LazyNorm):
        pre = a.prenormed
        if pre is None or a.row_index is not None:
            a = a.materialize()
        else:
            extra_in = (pre.sq.data_ptr(), pre.items, pre.sq.stride(0), float(pre.x.shape[-1]), a.eps)
            a = pre.x
    ctx.prenormed = None
    if a.dtype != torch.bfloat16 or a.stride(-1) != 1 or a.shape[-1] != plan.k or a.data_ptr() % 16 or a.stride(0) % 8:
        raise KernelLaunchError(f"gemm_cluster: activations {tuple(a.shape)} {a.dtype} do not fit weight [{plan.n}, {plan.k}]")
    n_out = plan.n // 2 if kind == CL_SWIGLU else plan.n
    tiles = -(-n_out // (BM // 2 if kind == CL_SWIGLU else BM))
    bn = cluster_tile(rows, tiles, plan.k)
    cluster = cluster_size(tiles * -(-rows // bn), plan.k)
    pre = None
    extra_out, rope = (0, 0, 0, 0, 0, 0), (0, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0)
    if kind == CL_ADD:
        out = epilogue.residual
        then = epilogue.then_norm
        if then is not None and then.tensors["weight"].data_ptr() % 16 == 0 and then.tensors["weight"].dtype in (torch.float32, torch.bfloat16):
            w, slices = then.tensors["weight"], tiles * cluster
            pre_x = ctx.ws.get("prenormed.cluster.x", (rows, n_out), torch.bfloat16, max_rows=CLUSTER_MAX_ROWS)
            # one row of parts per slice; fewer rows are shared by larger clusters, so more slices
            pre_sq = ctx.ws.get("prenormed.cluster.sq", (slices, CLUSTER_MAX_ROWS), torch.float32, max_rows=tiles * CLUSTER_MAX_SIZE)
            extra_out = (pre_x.data_ptr(), pre_x.stride(0), w.data_ptr(), DT_BF16 if w.dtype == torch.bfloat16 else DT_F32,
                         pre_sq.data_ptr(), pre_sq.stride(0))
            pre = Prenormed(then, pre_x, pre_sq, slices)
    elif kind == CL_ROPE:
        c, out = epilogue.cache, epilogue.q_out
        rope = (c.k_ptr, c.v_ptr, c.block_table.data_ptr(), c.page_stride, c.table_stride, c.page_tokens, c.kv_heads, c.head_dim,
                epilogue.positions.data_ptr(), epilogue.row_seq.data_ptr(), _ptr(epilogue.inv_freq), epilogue.q_heads,
                1 if epilogue.write_cache else 0)
    else:
        out = ctx.ws.get(buffer, (rows, n_out), out_dtype)
    _check(lib(activation if kind == CL_SWIGLU else "silu").llm_gemm_cluster(
        ctypes.addressof(plan.weight_map(BM // 2 if kind == CL_SWIGLU else BM)), ctypes.addressof(plan.act_map(a, bn)), kind,
        cluster, bn, rows, n_out, plan.k, out.data_ptr(), DT_BF16 if out.dtype == torch.bfloat16 else DT_F32, out.stride(0),
        n_out if kind == CL_SWIGLU else 0, *extra_in, *extra_out, *rope, error_word(a.device).data_ptr(), ctx.stream),
        "gemm_cluster")
    ctx.prenormed = pre
    return None if kind in (CL_ADD, CL_ROPE) else Partials(out)
