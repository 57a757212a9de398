"""Host side of the TMA + tcgen05 matrix product: tensor maps, tile and split choice, launch.

A :class:`GemmPlan` is made once per weight and holds its TMA descriptor.  Descriptors of
activations are cached by (address, rows, width, tile), which is stable because activations
live in the engine's persistent workspace.
"""

from __future__ import annotations

import ctypes
from ctypes import c_int, c_uint, c_ulonglong, c_void_p
from functools import lru_cache

import torch

from mini_engine_b200.csrc import build, ops
from mini_engine_b200.csrc.build import load_library

NUM_SMS = 148
BLOCK_N = 128
BLOCK_K = 64
TOKEN_TILES = (16, 32, 64, 128, 256)
SPLIT_MAX_TOKENS = 1024  # products of more tokens have enough tiles without splitting
MIN_K_BLOCKS_PER_SPLIT = 4
PAIR_MIN_TOKENS = 128  # longer products run on CTA pairs (256 x 256 tiles), unsplit ones in the persistent kernel
# Products of 129 to 1,024 tokens whose reduction is split run on CTA pairs too (each split its own
# pairs) when a split is long: 48 k blocks and more (the down projection of Qwen3-8B: 256 tokens
# 33.1 -> 31.3 us, 512 tokens 48.9 -> 44.2 us); with 16 to 32 k blocks per split the lone CTAs are as
# fast or 2 % faster.
PAIR_SPLIT_MIN_K_BLOCKS = 48
# Up to this many tokens the stacked gated product cuts its reduction in two halves, one per CTA of a
# cluster of two: 384 CTAs of 72 KB, three to an SM, stream the weights at 6.5 TB/s where 192 CTAs
# with the whole reduction reach 5.9 (8 tokens, 12,288 gated features of 4,096: 34.3 us unsplit).
STACKED_HALVES_MAX_TOKENS = 16
# The persistent pair kernel numbers its tiles in groups of this many token tiles (all feature tiles
# of a group before the next group): the pairs that run together then share a block of tiles about
# as tall as it is wide, and a group's activations are read once for all features.  0: one group (the
# token tile fastest over the whole product).  Measured at Qwen3-8B's shapes: nothing changes up to
# 4,096 tokens; 8,192 tokens: q/k/v 317 -> 295 us, o 211 -> 193, down 606 -> 563, gate and up with
# SwiGLU 1,159 -> 1,119 (its groups 16 wide: with 8, 1,130); 16,384 tokens: 697 -> 574, 464 -> 384,
# 1,349 -> 1,125, 2,462 -> 2,247 us (1.43 to 1.47 PFLOP/s).
PAIR_GROUP_TOKEN_TILES = 8
PAIR_GROUP_TOKEN_TILES_GATED = 16
STACKED_MAX_TOKENS = 64  # gated products of up to this many tokens stack gate rows on up rows in one operand


def _ops_stream() -> c_void_p:
    return ops._stream()


_lib = None


def _library():
    global _lib
    if _lib is None:
        lib = load_library("gemm_tcgen05")
        lib.me_make_tensor_map.argtypes = [c_void_p, c_void_p, c_ulonglong, c_ulonglong, c_uint]
        lib.me_make_tensor_map.restype = c_int
        lib.me_gemm_tcgen05.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.me_gemm_tcgen05.restype = c_int
        lib.me_gemm_tcgen05_swiglu.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.me_gemm_tcgen05_swiglu.restype = c_int
        lib.me_gemm_tcgen05_pair_split.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]
        lib.me_gemm_tcgen05_pair_split.restype = c_int
        lib.me_gemm_tcgen05_persistent.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.me_gemm_tcgen05_persistent.restype = c_int
        lib.me_gemm_tcgen05_persistent_swiglu.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.me_gemm_tcgen05_persistent_swiglu.restype = c_int
        lib.me_gemm_tcgen05_stacked_swiglu.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p]
        lib.me_gemm_tcgen05_stacked_swiglu.restype = c_int
        lib.me_gemm_tcgen05_grouped.argtypes = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_int, c_int, c_int,
                                                ctypes.c_float, ctypes.c_float, ctypes.c_float, c_int, c_void_p]
        lib.me_gemm_tcgen05_grouped.restype = c_int
        lib.me_gemm_wait_probe.argtypes = [c_int, c_void_p, c_void_p]
        lib.me_gemm_wait_probe.restype = c_int
        lib.me_gemm_take_error.argtypes = [ctypes.POINTER(c_int)]
        lib.me_gemm_take_error.restype = c_int
        _lib = lib
    return _lib


def supports(outs: int, inner: int) -> bool:
    """TMA wants a 16-byte row pitch: ``inner`` a multiple of 8 bfloat16 values."""
    return inner % 8 == 0 and inner >= 8 and outs >= 1


def token_tile(tokens: int) -> int:
    for tile in TOKEN_TILES:
        if tokens <= tile:
            return tile
    return TOKEN_TILES[-1]


@lru_cache(maxsize=4096)
def choose_splits(tokens: int, outs: int, inner: int, max_splits: int = 8) -> int:
    """How many ranges the reduction axis is cut into.  It depends on the sizes only (for a
    given number of tokens the same split is always chosen), and no split is empty."""
    if tokens > SPLIT_MAX_TOKENS:
        return 1
    tile = token_tile(tokens)
    tiles = -(-outs // BLOCK_N) * -(-tokens // tile)
    k_blocks = -(-inner // BLOCK_K)
    slots = NUM_SMS * (3 if tile <= 16 else 2 if tile <= 64 else 1)  # CTAs of this tile size that fit an SM at once (72, 80, 96, 192 KB of shared memory)
    wanted = min(max_splits, max(1, slots // tiles), max(1, k_blocks // MIN_K_BLOCKS_PER_SPLIT))
    per_split = -(-k_blocks // wanted)
    return -(-k_blocks // per_split)


def _make_map(tensor: torch.Tensor, box_rows: int) -> ctypes.Array:
    """TMA descriptor of a contiguous bfloat16 matrix with boxes of ``box_rows`` x 64 elements."""
    if tensor.dtype != torch.bfloat16 or not tensor.is_contiguous() or tensor.dim() != 2:
        raise RuntimeError("TMA descriptors are made for contiguous 2-D bfloat16 tensors")
    rows, inner = tensor.shape
    holder = (ctypes.c_ubyte * 128)()
    code = _library().me_make_tensor_map(holder, tensor.data_ptr(), rows, inner, box_rows)
    if code != 0:
        raise RuntimeError(f"could not make a TMA descriptor for a {rows} x {inner} matrix (code {code})")
    return holder


class GemmPlan:
    def __init__(self, weight: torch.Tensor, dual_rows: int | None = None):
        if weight.dtype != torch.bfloat16 or not weight.is_contiguous() or not weight.is_cuda:
            raise RuntimeError("the tensor-core product takes a contiguous bfloat16 CUDA weight")
        self.weight = weight
        self.rows, self.inner = weight.shape
        self.dual_rows = dual_rows  # gate rows [0, dual_rows), up rows [dual_rows, 2 * dual_rows)
        self.map = _make_map(weight, BLOCK_N)
        # Boxes of 64 rows, for the few-token gated kernel that stacks gate rows on up rows.
        self.map_half = _make_map(weight, BLOCK_N // 2) if dual_rows is not None else None


_activation_maps: dict[tuple[int, int, int, int], ctypes.Array] = {}


def _activation_map(x: torch.Tensor, tile: int) -> ctypes.Array:
    key = (x.data_ptr(), x.shape[0], x.shape[1], tile)
    held = _activation_maps.get(key)
    if held is None:
        if len(_activation_maps) > 8192:
            _activation_maps.clear()
        held = _make_map(x, tile)
        _activation_maps[key] = held
    return held


def _check_x(plan: GemmPlan, x: torch.Tensor) -> None:
    if x.dtype != torch.bfloat16 or not x.is_contiguous() or x.dim() != 2 or x.shape[1] != plan.inner:
        raise RuntimeError(f"activation {tuple(x.shape)} {x.dtype} does not fit a weight of width {plan.inner}")
    if x.data_ptr() % 16:
        raise RuntimeError("activation must be 16-byte aligned for TMA")


def gemm(plan: GemmPlan, x: torch.Tensor, out: torch.Tensor, splits: int, group: int | None = None) -> None:
    """``out[s] = x @ weight^T`` restricted to the k range of split ``s``; float32
    ``[splits, T, rows]``.  ``group`` pins the width of the persistent kernel's tile groups (the
    kernel tests run several; the kernel bench times them)."""
    _check_x(plan, x)
    tokens = x.shape[0]
    if out.dtype != torch.float32 or tuple(out.shape) != (splits, tokens, plan.rows) or not out.is_contiguous():
        raise RuntimeError(f"output {tuple(out.shape)} does not fit [{splits}, {tokens}, {plan.rows}] float32")
    tile = token_tile(tokens)
    stream = _ops_stream()
    if tokens > PAIR_MIN_TOKENS and splits == 1:
        code = _library().me_gemm_tcgen05_persistent(
            plan.map, _activation_map(x, 128), out.data_ptr(), tokens, plan.rows, plan.inner,
            PAIR_GROUP_TOKEN_TILES if group is None else group, -1, stream,
        )  # fmt: skip
    elif tokens > PAIR_MIN_TOKENS and -(-plan.inner // BLOCK_K) >= PAIR_SPLIT_MIN_K_BLOCKS * splits:
        code = _library().me_gemm_tcgen05_pair_split(
            plan.map, _activation_map(x, 128), out.data_ptr(), tokens, plan.rows, plan.inner, splits, stream
        )
    else:
        code = _library().me_gemm_tcgen05(
            plan.map, _activation_map(x, tile), out.data_ptr(), tokens, plan.rows, plan.inner, tile, splits, stream
        )
    _count_launch()
    if code != 0:
        raise RuntimeError(f"tensor-core product failed to launch (code {code})")


def gemm_activated(plan: GemmPlan, x: torch.Tensor, act: torch.Tensor, activation: int) -> None:
    """``act = a(x @ weight^T)`` in bfloat16 with an activation of :data:`ops.PLAIN_ACTIVATIONS` in the epilogue, for
    products of more than ``PAIR_MIN_TOKENS`` tokens."""
    _check_x(plan, x)
    tokens = x.shape[0]
    if tokens <= PAIR_MIN_TOKENS:
        raise RuntimeError(f"the product with a plain activation takes more than {PAIR_MIN_TOKENS} tokens")
    if act.dtype != torch.bfloat16 or tuple(act.shape) != (tokens, plan.rows) or not act.is_contiguous():
        raise RuntimeError(f"activation output {tuple(act.shape)} does not fit [{tokens}, {plan.rows}] bfloat16")
    code = _library().me_gemm_tcgen05_persistent(
        plan.map, _activation_map(x, 128), act.data_ptr(), tokens, plan.rows, plan.inner, PAIR_GROUP_TOKEN_TILES, activation,
        _ops_stream(),
    )  # fmt: skip
    _count_launch()
    if code != 0:
        raise RuntimeError(f"activated tensor-core product failed to launch (code {code})")


def gemm_swiglu(
    plan: GemmPlan, x: torch.Tensor, act: torch.Tensor, halves: int | None = None, group: int | None = None, activation: str = "silu"
) -> None:
    """``act = silu(x @ gate^T) * (x @ up^T)`` in bfloat16, gate/up being the halves of the
    plan's weight; ``activation="gelu_tanh"`` gates with the tanh form of GELU instead.  ``halves`` (1 or 2) pins how many CTAs share a reduction of the few-token kernel
    instead of the rule's choice: the kernel tests run both forms, the kernel bench times them."""
    _check_x(plan, x)
    tokens = x.shape[0]
    if plan.dual_rows is None:
        raise RuntimeError("this plan was not made for a gated product")
    if act.dtype != torch.bfloat16 or tuple(act.shape) != (tokens, plan.dual_rows) or not act.is_contiguous():
        raise RuntimeError(f"activation output {tuple(act.shape)} does not fit [{tokens}, {plan.dual_rows}] bfloat16")
    if activation not in ("silu", "gelu_tanh"):
        raise RuntimeError(f"the gated product's epilogue knows 'silu' and 'gelu_tanh', got {activation!r}")
    gelu = 1 if activation == "gelu_tanh" else 0
    stream = _ops_stream()
    if tokens <= STACKED_MAX_TOKENS:
        tile = token_tile(tokens)
        if halves is None:
            halves = 2 if tokens <= STACKED_HALVES_MAX_TOKENS and plan.inner >= 2 * BLOCK_K else 1
        code = _library().me_gemm_tcgen05_stacked_swiglu(
            plan.map_half, _activation_map(x, tile), act.data_ptr(), tokens, plan.dual_rows, plan.inner, plan.dual_rows,
            tile, halves, gelu, stream,
        )  # fmt: skip
    elif tokens > PAIR_MIN_TOKENS:
        code = _library().me_gemm_tcgen05_persistent_swiglu(
            plan.map, _activation_map(x, 128), act.data_ptr(), tokens, plan.dual_rows, plan.inner, plan.dual_rows,
            PAIR_GROUP_TOKEN_TILES_GATED if group is None else group, gelu, stream,
        )  # fmt: skip
    else:
        tile = 128  # 65 to 128 tokens: lone CTAs with gate and up sums side by side in tensor memory
        code = _library().me_gemm_tcgen05_swiglu(
            plan.map, _activation_map(x, tile), act.data_ptr(), tokens, plan.dual_rows, plan.inner, plan.dual_rows,
            tile, gelu, stream,
        )
    _count_launch()
    if code != 0:
        raise RuntimeError(f"gated tensor-core product failed to launch (code {code})")


# ------------------------------------------------------------------------------ float32

# Tokens per CTA (with 16 two CTAs share an SM, else one), the us of a k block and of a round of CTAs beside its blocks.  Two CTAs on an SM have
# SPLIT_SHARED for a block; 64 and 128 tokens have their pieces made by a launch more, SPLIT_PIECES, of which nothing is left where launches overlap;
# a cluster's exchange costs SPLIT_EXCHANGE for each segment of 128 tokens.  Clusters of 1 to 8 CTAs that are resident at a time with one CTA to an
# SM (cudaOccupancyMaxActiveClusters on a B200; with two to an SM twice as many and two more).  The constants fit 478 shapes alone and 442 in chains
# of products (1 to 2,048 tokens, 64 to 32,768 outputs of 64 to 12,288 inputs) in all their forms: for 13 of them another form is more than 5 %
# faster.  us in a chain in plain stream order, 16 tokens to a CTA, 16 side by side | 64, 64 side by side, 128 side by side: 17 tokens x 2,048 x 2,048 29, 11 |
# 30, 20, 24; 40 x 576 x 2,048 29, 8.3 | 31, 11.8, 13.5; 128 of these 28, 16 | 31, 12, 15; 40 x 4,096 x 2,048 30, 26 | 31, 25.6, 31; 256 of these 78, 111 |
# 33, 62, 52; where launches overlap, 40 x 576 x 2,048 29, 8.3 | 28, 8.3, 10.5 and 40 x 4,096 x 2,048 34, 25 | 28, 22, 28.  With 64 and 128 alone, small
# products in plain stream order were up to 29 % behind what they took before pieces were made ahead.
SPLIT_TILES = {16: (0.84, 4.2), 64: (0.70, 5.8), 128: (1.15, 6.4)}
SPLIT_SHARED, SPLIT_EXCHANGE = 1.12, 0.30
SPLIT_PIECES = (3.4, 0.0)  # in plain stream order, and where a launch begins while the one before ends
# The same for runs of sorted rows, whose weights are each read once only, so that a CTA's block waits for memory more: one decoded token of Molotar's
# sizes 668 us with these constants and 684 with those above, 48 tokens 1,263 and 1,281.
SPLIT_GROUPED = {16: (1.0, 5.0), 64: (0.70, 5.0), 128: (1.25, 5.0)}
SPLIT_CLUSTERS = (NUM_SMS, 74, 45, 33, 26, 22, 15, 15)
SPLIT_PIECES_MIN_TILE = 64  # tokens per CTA from which on their pieces are made ahead, by a kernel of their own
# Bytes of pieces at a time: they come out of what the page pool leaves, so larger steps (from 7,281 tokens of 12,288 on) run in parts.  8,192 x 1,024 x
# 12,288 in one part and in two 1,390 to 1,480 | 1,530 to 1,640 us, 8,192 x 6,144 x 12,288 8.9 to 9.3 | 8.4 to 8.8 ms.
SPLIT_PIECES_BYTES = 512 << 20
SPLIT_MIN_K_BLOCKS = 4  # of a segment
# Shorter reductions stay on CUDA cores: a chain of fmaf over so few terms is about as exact as the short chain of the tensor
# core (relative error of normal operands at 64: 1.5e-7 against 0.7e-7), and nothing is to be gained.
SPLIT_MIN_INNER = 64
_split_lib = None


def _split_library():
    global _split_lib
    if _split_lib is None:
        lib = load_library("gemm_split")
        lib.me_make_tensor_map_f32.argtypes = [c_void_p, c_void_p, c_ulonglong, c_ulonglong, c_uint]
        lib.me_make_tensor_map_f32.restype = c_int
        lib.me_make_tensor_map_pieces.argtypes = [c_void_p, c_void_p, c_ulonglong, c_ulonglong, c_uint]
        lib.me_make_tensor_map_pieces.restype = c_int
        lib.me_gemm_split.argtypes = [c_void_p] * 5 + [c_int] * 4 + [c_void_p] + [c_int] * 2 + [c_void_p, c_int, c_int, c_void_p]
        lib.me_gemm_split.restype = c_int
        lib.me_gemm_split_take_error.argtypes = [ctypes.POINTER(c_int)]
        lib.me_gemm_split_take_error.restype = c_int
        _split_lib = lib
    return _split_lib


def split_supports(weight: torch.Tensor) -> bool:
    """TMA wants a 16-byte aligned start and row pitch: ``inner`` a multiple of 4 float32 values.  A property of the weight
    alone: every step of a model takes the same kernel (but for activations that do not start on 16 bytes, which
    :class:`parts.linear.Linear` sends to the CUDA cores; the workspace's always do)."""
    return (
        weight.dtype == torch.float32 and weight.is_cuda and weight.is_contiguous()
        and weight.shape[1] % 4 == 0 and weight.shape[1] >= SPLIT_MIN_INNER and weight.data_ptr() % 16 == 0
    )  # fmt: skip


def split_segments(outs: int, inner: int) -> int:
    """Ranges of k blocks that an output's sum is formed in.  From the weight's shape alone, never from the tokens: a row's
    bits must not depend on the batch.  About one CTA per SM when a single token tile runs with its segments side by side."""
    tiles, k_blocks = -(-outs // BLOCK_N), -(-inner // BLOCK_K)
    wanted = min(8, max(1, 160 // tiles), max(1, k_blocks // SPLIT_MIN_K_BLOCKS))
    per_segment = -(-k_blocks // wanted)
    return -(-k_blocks // per_segment)


@lru_cache(maxsize=4096)
def split_form(tokens: int, outs: int, inner: int, segments: int, tile: int | None = None, overlapped: bool = False) -> tuple[int, bool]:
    """Tokens per CTA (or the given ``tile``), and whether a tile's segments run in the CTAs of a cluster or one after the other in a
    CTA; the bits are the same in every form.  ``tile``: of a grouped product.  The form whose rounds of resident CTAs take least time, in plain stream order or
    (``overlapped``) as programmatic dependents."""
    blocks = -(-inner // BLOCK_K)
    per_segment = -(-blocks // segments)
    forms = []
    for rows, (block, start) in (SPLIT_TILES if tile is None else SPLIT_GROUPED).items():
        if (rows != tile) if tile is not None else (rows > 16 and tokens <= 16):
            continue
        per_sm = 2 if rows == 16 else 1
        pieces = SPLIT_PIECES[overlapped] if rows >= SPLIT_PIECES_MIN_TILE else 0.0
        ctas = -(-outs // BLOCK_N) * -(-tokens // rows)
        cost = lambda resident: SPLIT_SHARED if tile is None and rows == 16 and resident > NUM_SMS else block  # noqa: B023, E731
        if rows < 128 or segments == 1:
            forms.append((-(-ctas // (per_sm * NUM_SMS)) * (blocks * cost(ctas) + start) + pieces, rows, False))
        if segments > 1:
            rounds = -(-ctas // (per_sm * SPLIT_CLUSTERS[segments - 1] + (2 * (per_sm - 1) if tile is None else 0)))
            forms.append((rounds * (per_segment * cost(ctas * segments) + start + SPLIT_EXCHANGE * segments * rows / 128) + pieces, rows, True))
    return min(forms)[1:]


class SplitPlan:
    """A float32 weight for :func:`gemm_split`, or, with ``group_rows`` rows for each group, for :func:`gemm_split_grouped`."""

    def __init__(self, weight: torch.Tensor, group_rows: int | None = None):
        if not split_supports(weight):
            raise RuntimeError(f"the float32 tensor-core product takes a contiguous float32 CUDA weight whose width is a multiple of 4 and at least {SPLIT_MIN_INNER}")
        self.weight = weight
        self.rows, self.inner = weight.shape
        if group_rows is not None and (group_rows < 1 or self.rows % group_rows):
            raise RuntimeError(f"{self.rows} weight rows do not form groups of {group_rows}")
        self.group_rows = group_rows
        self.segments = split_segments(group_rows or self.rows, self.inner)
        self.map = _make_split_map(_split_library().me_make_tensor_map_f32, weight, self.rows, self.inner, BLOCK_N)


def _make_split_map(make, tensor: torch.Tensor, rows: int, inner: int, box_rows: int) -> ctypes.Array:
    holder = (ctypes.c_ubyte * 128)()
    code = make(holder, tensor.data_ptr(), rows, inner, box_rows)
    if code != 0:
        raise RuntimeError(f"could not make a TMA descriptor for a {rows} x {inner} float32 matrix (code {code})")
    return holder


_split_activation_maps: dict[tuple[int, int, int, int, bool], ctypes.Array] = {}


def _split_activation_map(x: torch.Tensor, tile: int, rows: int = 0, inner: int = 0) -> ctypes.Array:
    """Of a float32 matrix, or (``rows`` given) of the pieces of one of ``rows`` x ``inner`` values."""
    key = (x.data_ptr(), rows or x.shape[0], inner or x.shape[1], tile, rows > 0)
    held = _split_activation_maps.get(key)
    if held is None:
        if len(_split_activation_maps) > 8192:
            _split_activation_maps.clear()
        make = _split_library().me_make_tensor_map_pieces if rows else _split_library().me_make_tensor_map_f32
        held = _split_activation_maps[key] = _make_split_map(make, x, key[1], key[2], tile)
    return held


def gemm_split(plan: SplitPlan, x: torch.Tensor, out: torch.Tensor, form: tuple[int, bool] | None = None, workspace=None) -> None:
    """``out[T, rows] = x @ weight^T`` in float32 (three bfloat16 pieces of each operand, see gemm_split.cu).
    ``form`` pins the tokens per CTA and where a tile's segments run instead of the rule's choice: the kernel tests run all.
    The tokens' pieces, where they are made ahead, lie in a buffer of the ``workspace``."""
    tokens = x.shape[0]
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or x.shape[1] != plan.inner or x.data_ptr() % 16:
        raise RuntimeError(f"activation {tuple(x.shape)} {x.dtype} does not fit a float32 weight of width {plan.inner}")
    if out.dtype != torch.float32 or tuple(out.shape) != (tokens, plan.rows) or not out.is_contiguous():
        raise RuntimeError(f"output {tuple(out.shape)} does not fit [{tokens}, {plan.rows}] float32")
    if tokens == 0:
        return
    tile, side_by_side = form or split_form(tokens, plan.rows, plan.inner, plan.segments, None, build._programmatic_launch)
    _launch_split(plan, x, out, plan.rows, tile, side_by_side, None, workspace)


def _launch_split(
    plan: SplitPlan, x: torch.Tensor, out: torch.Tensor, outs: int, tile: int, side_by_side: bool, groups: torch.Tensor | None, workspace,
    withheld: bool = False,
) -> None:  # fmt: skip
    rows, inner = x.shape
    pieces = None
    if tile < SPLIT_PIECES_MIN_TILE:
        x_map = _split_activation_map(x, tile)
    else:
        width = 3 * (-(-inner // 8) * 8)
        if 2 * width * rows > SPLIT_PIECES_BYTES:  # as many rows at a time as their pieces have room, in parts of about the same size
            parts = -(-rows // max(tile, SPLIT_PIECES_BYTES // (2 * width) // tile * tile))
            at_once = -(-rows // (parts * tile)) * tile
            if at_once < rows:
                for first in range(0, rows, at_once):
                    part = slice(first, min(first + at_once, rows))
                    _launch_split(
                        plan, x[part], out[part], outs, tile, side_by_side, None if groups is None else groups[first // tile :], workspace, withheld
                    )  # fmt: skip
                return
        if workspace is None:
            held = torch.empty(width * rows, dtype=torch.bfloat16, device=x.device)
        else:
            held = workspace.growing("split.pieces", (width * rows,), torch.bfloat16)
        pieces, x_map = held.data_ptr(), _split_activation_map(held, tile, rows, inner)
        _count_launch()
    code = _split_library().me_gemm_split(
        plan.map, x_map, x.data_ptr(), plan.weight.data_ptr(), out.data_ptr(), rows, outs, inner, tile, pieces, plan.segments,
        1 if side_by_side else 0, None if groups is None else groups.data_ptr(), 0 if groups is None else outs, 1 if withheld else 0, _ops_stream(),
    )  # fmt: skip
    _count_launch()
    if code != 0:
        raise RuntimeError(f"float32 tensor-core product failed to launch (code {code})")


def gemm_split_grouped(
    plan: SplitPlan, x: torch.Tensor, out: torch.Tensor, group_of_block: torch.Tensor, pad: int, filled: int, side_by_side: bool | None = None,
    workspace=None,
) -> None:  # fmt: skip
    """A float32 product over rows that are sorted by group: the plan's weight holds ``plan.group_rows`` rows per group, run ``b``
    of ``pad`` rows of ``x`` (one of ``SPLIT_TILES``) belongs to group ``group_of_block[b]`` (int32 on the device; negative: no rows
    there), ``out[t] = x[t] @ weight_of_group^T``.  A row's bits depend on the row and its group's weight alone.  ``filled``:
    about how many runs hold rows, for the choice of the form."""
    rows, outs = x.shape[0], plan.group_rows
    if outs is None:
        raise RuntimeError("this plan was not made for a grouped product")
    if x.dtype != torch.float32 or not x.is_contiguous() or x.dim() != 2 or x.shape[1] != plan.inner or x.data_ptr() % 16:
        raise RuntimeError(f"activation {tuple(x.shape)} {x.dtype} does not fit a float32 weight of width {plan.inner}")
    if out.dtype != torch.float32 or tuple(out.shape) != (rows, outs) or not out.is_contiguous():
        raise RuntimeError(f"output {tuple(out.shape)} does not fit [{rows}, {outs}] float32")
    if pad not in SPLIT_TILES or rows % pad or group_of_block.dtype != torch.int32 or group_of_block.numel() < rows // pad:
        raise RuntimeError("the rows of a grouped product come in runs of a token tile with one int32 group each")
    if side_by_side is None:
        side_by_side = split_form(max(1, min(filled, rows // pad)) * pad, outs, plan.inner, plan.segments, pad, build._programmatic_launch)[1]
    _launch_split(plan, x, out, outs, pad, side_by_side, group_of_block, workspace)


GROUP_PAD = 128  # rows of a run of the sorted rows that belongs to one group: the token tile of the grouped product


def gemm_grouped(
    plan: GemmPlan, x: torch.Tensor, out: torch.Tensor, group_of_block: torch.Tensor, group_rows: int, outs: int,
    dual_rows: int = 0, slope: float = 1.0, limit: float | None = None, offset: float = 0.0, activation: int | None = None,
) -> None:  # fmt: skip
    """A product over rows that are sorted by group: the plan's weight holds ``group_rows`` rows per group, run
    ``b`` of ``GROUP_PAD`` rows of ``x`` belongs to group ``group_of_block[b]`` (int32 on the device; negative: no
    rows there).  ``out [rows, outs]`` float32 is ``x[t] . w[group * group_rows + n]``; with ``dual_rows`` it is
    bfloat16 and holds the gated unit of rows ``n`` and ``dual_rows + n`` of the row's group with the constants of
    :func:`ops.swiglu`; with ``activation`` (a number of :data:`ops.PLAIN_ACTIVATIONS`) it is bfloat16 and holds the
    activated sums."""
    _check_x(plan, x)
    rows = x.shape[0]
    want = torch.bfloat16 if dual_rows or activation is not None else torch.float32
    if out.dtype != want or tuple(out.shape) != (rows, outs) or not out.is_contiguous():
        raise RuntimeError(f"output {tuple(out.shape)} {out.dtype} does not fit [{rows}, {outs}] {want}")
    if rows % GROUP_PAD or group_of_block.dtype != torch.int32 or group_of_block.numel() < rows // GROUP_PAD:
        raise RuntimeError("the rows of a grouped product come in runs of GROUP_PAD with one int32 group each")
    code = _library().me_gemm_tcgen05_grouped(
        plan.map, _activation_map(x, GROUP_PAD), out.data_ptr(), rows, outs, plan.inner, group_of_block.data_ptr(),
        GROUP_PAD, group_rows, dual_rows, float(slope), float(limit or 0.0), float(offset),
        -1 if activation is None else activation, _ops_stream(),
    )  # fmt: skip
    _count_launch()
    if code != 0:
        raise RuntimeError(f"grouped tensor-core product failed to launch (code {code})")


def _count_launch() -> None:
    ops._Counter.launches += 1


def wait_probe(polls: int = 4096) -> bool:
    """Launch a CTA whose barrier waits run out after ``polls`` polls because nothing ever arrives
    at them (no fault, trap or endless loop): it records the failure as the product kernels do,
    gives its tensor memory back and returns.  True when it returned; :func:`take_error` then
    reports the recorded code.  Exists so that the give-up path can be tested."""
    lib = _library()
    returned = torch.zeros(1, dtype=torch.int32, device="cuda")
    code = lib.me_gemm_wait_probe(polls, returned.data_ptr(), _ops_stream())
    _count_launch()
    if code != 0:
        raise RuntimeError(f"the wait probe failed to launch (code {code})")
    return bool(returned.item())


def split_wait_probe(plan: SplitPlan, x: torch.Tensor, out: torch.Tensor, side_by_side: bool, tile: int = 16) -> None:
    """The float32 product in the form of ``tile`` tokens to a CTA with every weight tile withheld: all waits of its roles run out after a few
    polls, the kernel records that, gives its tensor memory back and returns without a result.  Exists so that the give-up path can be tested."""
    if x.shape[1] != plan.inner or tuple(out.shape) != (x.shape[0], plan.rows) or not (x.is_contiguous() and out.is_contiguous()):
        raise RuntimeError("the probe takes the arguments of a product")
    _launch_split(plan, x, out, plan.rows, tile, side_by_side, None, None, withheld=True)


def take_error() -> int:
    """The first failure that a tensor-core kernel recorded on the device since the last call
    (a wait that ran into its limit), or 0.  Synchronises the device."""
    first = 0
    for lib, name in ((_lib, "me_gemm_take_error"), (_split_lib, "me_gemm_split_take_error")):
        if lib is None:
            continue
        code = c_int(0)
        status = getattr(lib, name)(ctypes.byref(code))
        if status != 0:
            raise RuntimeError(f"could not read the kernels' error flag (CUDA error {status})")
        first = first or code.value
    return first
