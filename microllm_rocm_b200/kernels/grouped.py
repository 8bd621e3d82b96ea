"""Grouped matrix products: one product per group over that group's rows (`csrc/grouped_gemm.cu`).

Two uses: the experts of a routed feed-forward (groups = experts, rows = the tokens routed to each, known only on
the device) and the per-head products of latent attention (groups = heads, every group takes all rows).  fp32
operands run in true fp32 with a fixed summation order; bf16 operands accumulate in fp32.
"""
from __future__ import annotations

from ctypes import c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import build, ops
from .build import KernelError
from .device import sm_count
from .gemm_bf16 import device_error_flag

SOURCE = "grouped_gemm.cu"
ops.register_signatures(SOURCE, {
    "mlb_grouped_gemm": [c_void_p, c_longlong, c_longlong, c_void_p, c_longlong, c_longlong, c_void_p, c_longlong, c_longlong,
                         c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_longlong, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int,
                         c_int, c_void_p],
})


MMA_SOURCE = "grouped_mma.cu"
ops.register_signatures(MMA_SOURCE, {
    "mlb_grouped_mma": [c_void_p, c_longlong, c_longlong, c_void_p, c_longlong, c_longlong, c_void_p, c_longlong, c_longlong,
                        c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_longlong, c_longlong, c_int, c_int, c_int, c_int, c_int,
                        c_int, c_int, c_void_p, c_int, c_void_p],
})

# CTA pairs on the fifth-generation tensor cores: groups of many rows (csrc/grouped_tc2.cu)
PAIR_SOURCE = "grouped_tc2.cu"
ops.register_signatures(PAIR_SOURCE, {
    "mlb_grouped_pair": [c_void_p, c_longlong, c_void_p, c_void_p, c_longlong, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int,
                         c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p],
    "mlb_gather_rows": [c_void_p, c_longlong, c_void_p, c_int, c_void_p, c_int, c_void_p, c_int, c_int, c_void_p],
})

# None: pair_pays decides; tests set it to True or False to send listed products to the pair kernel, or not
USE_PAIRS = None

# Tests set it to False to send bf16 products to the CUDA-core kernel and compare.
USE_TENSOR_CORES = True


def sources():
    return [(SOURCE, {}), (MMA_SOURCE, {}), (PAIR_SOURCE, {})]


def mma_supported(a: torch.Tensor, weight: torch.Tensor, a_group_cols: int = 0) -> bool:
    """The tensor-core kernel moves 16-byte pieces: bf16 operands whose K, row pitches and column blocks are multiples
    of 8 elements."""
    return (USE_TENSOR_CORES and a.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and weight.shape[2] % 8 == 0
            and a.stride(0) % 8 == 0 and weight.stride(1) % 8 == 0 and weight.stride(0) % 8 == 0 and a_group_cols % 8 == 0
            and a.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0)


def pair_supported(a: torch.Tensor, weight: torch.Tensor) -> bool:
    """The pair kernel reads its operands by TMA out of whole matrices: what the tensor-core kernel takes, the weights of the
    groups one behind another."""
    G, N, K = weight.shape
    return mma_supported(a, weight) and G <= 1024 and weight.is_contiguous() and a.stride(1) == 1 and G * N < 1 << 31


def pair_pays(rows: int, groups: int, weight_rows: int, weight_bytes: int, sms: int, dual: bool = True) -> bool:
    """Whether a listed product goes to pairs of SMs with tiles of 256 weight rows (`weight_bytes` a group; `dual`: the gated form).  Against
    it stand the set-up of a pair (5 us, and 2 for the gathering), waves of tiles that a last one leaves half empty, and an epilogue that
    short sums do not hide.  Measured (148 SMs, us, mma.sync / pairs):
      * Groups of more than 16 rows, where mma.sync takes 64 rows a tile: every pair needs a tile.  32 of 768 rows, width 1,024: gate/up
        of 512 23 / 21, down 16 / 12; sums of 256 lose (64 groups of 48 rows 15.5 / 16.5).
      * From 96 rows on (128 a tile) few tiles are enough, but sums below 1,024 need work to amortize: gate/up from 0.8 GFLOP on, plain
        from 2.  600 rows, width 2,048: gate/up of 704 44 / 28, down 17.2 / 19.2; 8 groups of 192 rows, 512 x 1,024: 15.1 / 17.9;
        64 groups of 192 of 1,408, width 2,048: 617 / 186 and 379 / 108; sums of 256 lose (16 x 600 rows 25.6 / 29.0).
      * Up to 16 rows both stream the weights, 16 rows a tile on mma.sync: pairs where the weights in use are large and fill their
        waves of tiles.  48 rows for 64 groups of 1,408, width 2,048: 69 + 43 / 65 + 39; 12 rows for 32 of 1,408, width 4,096: gate/up 49 / 54; 512 rows for 64 of 704: 71 / 79 (384 tiles
        in six waves of 74); 48 rows for 16 groups of 1,408, width 4,096: 73 / 78 (176 tiles in three waves); 512 for 32 of 704, width 2,048:
        55 / 45."""
    if USE_PAIRS is not None:
        return USE_PAIRS
    active, pairs = min(groups, rows), sms // 2
    tiles, total = active * -(-weight_rows // 256), active * weight_bytes
    k = weight_bytes // (2 * weight_rows)
    if rows >= 96 * groups:
        return k >= 1024 or (k >= 512 and 2 * rows * weight_rows * k >= (0.8e9 if dual else 2e9))
    if rows > 16 * groups:
        return tiles >= pairs and k >= 512
    filled = active * weight_rows / (256 * pairs * max(1, -(-tiles // pairs)))
    return (total >= 150 << 20 and filled >= 0.75) if rows >= 16 * groups else (total >= (300 if dual else 250) << 20 and filled >= 0.85)


def _pair(a, weight, out, *, rows, outputs, group_offsets, a_rows, a_row_div, c_rows, dual, act, row_scale, row_tile, alloc, error_flag):
    G, w_rows, K = weight.shape
    if rows < 0 or a_row_div <= 0 or row_tile not in (16, 64, 128):      # (refused by the launchers of the other routes)
        raise KernelError(f"grouped product: bad sizes, {rows} rows, divisor {a_row_div}, row tile {row_tile}")
    out_bf16 = 1 if ops.dtype_tag(out) == ops.BF16 else 0                # (fp32 or bf16: other types are refused, as on the other routes)
    flag = error_flag if error_flag is not None else device_error_flag(a.device)
    L = ops.lib(PAIR_SOURCE)
    source = a
    if a_rows is not None:                               # the pair kernel reads rows as they lie: in the order of the list
        source = alloc((rows, K), a.dtype) if alloc is not None else torch.empty((rows, K), dtype=a.dtype, device=a.device)
        build.check(L, L.mlb_gather_rows(a.data_ptr(), a.stride(0), a_rows.data_ptr(), int(a_row_div), group_offsets.data_ptr(), G,
                                         source.data_ptr(), int(rows), K, ops._stream()))
    # the copies take whole boxes of rows, a tile's last ones with rows of the next group: up to the end of the matrix and no further
    rows = min(int(rows), source.shape[0])
    if rows == 0:
        return
    # one tile for most groups: the mean and a quarter more
    mean = rows / min(G, rows)
    cap = 32 if mean <= 16 else min(256, max(64, -(-int(1.25 * mean) // 64) * 64))
    sms = sm_count(a.device)
    build.check(L, L.mlb_grouped_pair(
        source.data_ptr(), source.stride(0), weight.data_ptr(), out.data_ptr(), out.stride(0), group_offsets.data_ptr(), ops._ptr(c_rows),
        ops._ptr(row_scale), ops._ptr(a_rows) if row_scale is not None else None, out_bf16, 1 if dual else 0,
        int(act), outputs if dual else 0, rows, outputs, K, G, w_rows, cap, sms - sms % 2, flag.data_ptr(), ops._stream()))


def row_tile_for(rows: int, groups: int, listed: bool, tensor_cores: bool) -> int:
    """Rows of a CTA's tile: 16 while a group holds few rows (decoding: a CTA should not multiply rows that do not
    exist), 128 on the tensor cores once the groups are large (twice the reuse of every weight tile), else 64."""
    per_group = rows / max(1, groups) if listed else rows
    if per_group <= 16:
        return 16
    return 128 if tensor_cores and per_group >= 96 else 64


def grouped_linear(a: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, *, rows: int, a_group_cols: int = 0,
                   c_group_cols: int = 0, group_offsets: Optional[torch.Tensor] = None, a_rows: Optional[torch.Tensor] = None,
                   c_rows: Optional[torch.Tensor] = None, a_row_div: int = 1, factor: Optional[torch.Tensor] = None,
                   row_scale: Optional[torch.Tensor] = None, row_tile: int = 64, error_flag: Optional[torch.Tensor] = None,
                   w_constant: bool = False) -> None:
    """weight [G, N, K]; a [*, lda] and out [*, ldc] are 2-D and row-major.

    group g multiplies the K columns of `a` that start at g * a_group_cols with weight[g] and writes N columns of
    `out` starting at g * c_group_cols.  With `group_offsets` ([G + 1] int32 on the device) group g owns the places
    offsets[g]..offsets[g+1]-1 of a sorted list of `rows` places; `a_rows[place] // a_row_div` is the row read and
    `c_rows[place]` the row written (None: the place itself).  Without it every group takes rows 0..rows-1.
    `factor` (fp32, the shape of `out`): the result is multiplied by it element by element.  `row_scale` (fp32, one number per
    entry that a_rows may name): a row's result is multiplied by row_scale[a_rows[place]] (not on the tensor cores).  `w_constant`: no kernel of the same step
    writes `weight`, which may then be read while the kernel in front still runs (without lists)."""
    ops._need(a, "a", dims=2); ops._need(weight, "weight", dims=3); ops._need(out, "out", dims=2)
    if a.dtype != weight.dtype:
        raise KernelError(f"grouped_linear: operands are {a.dtype} and {weight.dtype}")
    G, N, K = weight.shape
    if a_group_cols * (G - 1) + K > a.shape[1] or c_group_cols * (G - 1) + N > out.shape[1]:
        raise KernelError("grouped_linear: a group's columns run past its matrix")
    for name, t in (("group_offsets", group_offsets), ("a_rows", a_rows), ("c_rows", c_rows)):
        if t is not None:
            ops._need(t, name, torch.int32, 1)
    if group_offsets is not None and group_offsets.shape[0] != G + 1:
        raise KernelError("grouped_linear: group_offsets must have one entry per group and one more")
    if factor is not None:
        ops._need(factor, "factor", torch.float32, 2)
        if factor.shape[1] < out.shape[1]:
            raise KernelError("grouped_linear: the factor matrix is narrower than the output")
    if row_scale is not None:
        ops._need(row_scale, "row_scale", torch.float32)
    if (group_offsets is not None and a_rows is None and factor is None and row_scale is None and not a_group_cols and not c_group_cols
            and pair_supported(a, weight) and pair_pays(rows, G, N, weight.stride(0) * 2, sm_count(a.device), dual=False)):
        _pair(a, weight, out, rows=rows, outputs=N, group_offsets=group_offsets, a_rows=None, a_row_div=a_row_div, c_rows=c_rows, dual=False,
              act=0, row_scale=None, row_tile=row_tile, alloc=None, error_flag=error_flag)
        return
    tensor_cores = mma_supported(a, weight, a_group_cols) and row_scale is None
    if row_tile == 128 and not tensor_cores:
        row_tile = 64
    if tensor_cores:
        L = ops.lib(MMA_SOURCE)
        build.check(L, L.mlb_grouped_mma(
            a.data_ptr(), a.stride(0), a_group_cols, weight.data_ptr(), weight.stride(1), weight.stride(0), out.data_ptr(),
            out.stride(0), c_group_cols, ops._ptr(group_offsets), ops._ptr(a_rows), ops._ptr(c_rows), int(a_row_div),
            ops._ptr(factor), factor.stride(0) if factor is not None else 0, 0, int(rows), N, K, G, ops.dtype_tag(out),
            int(row_tile), 0, None, 1 if w_constant else 0, ops._stream()))
        return
    L = ops.lib(SOURCE)
    build.check(L, L.mlb_grouped_gemm(
        a.data_ptr(), a.stride(0), a_group_cols, weight.data_ptr(), weight.stride(1), weight.stride(0), out.data_ptr(),
        out.stride(0), c_group_cols, ops._ptr(group_offsets), ops._ptr(a_rows), ops._ptr(c_rows), int(a_row_div),
        ops._ptr(factor), factor.stride(0) if factor is not None else 0, ops._ptr(row_scale), int(rows), N, K, G, ops.dtype_tag(a),
        ops.dtype_tag(out), int(row_tile), ops._stream()))


def grouped_silu_mul(a: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, *, rows: int, group_offsets: torch.Tensor,
                     a_rows: Optional[torch.Tensor] = None, a_row_div: int = 1, row_tile: int = 64, alloc=None,
                     activation: str = "silu", limit: Optional[float] = None, row_scale: Optional[torch.Tensor] = None,
                     error_flag: Optional[torch.Tensor] = None) -> None:
    """weight [G, 2 * F, K]: per group F gate rows over F up rows; out[place] = silu(a gate^T) * (a up^T), [rows, F]; or,
    with `activation` "clamped_swish" and its `limit`, the clamped form (ops.activation_code).  `row_scale` (fp32, one number per
    entry that a_rows may name): both products are multiplied by row_scale[a_rows[place]] in front of the activation, which is a
    weight on the row that goes in.
    On the tensor cores both products and the activation are one kernel; otherwise the fused product leaves
    [rows, 2 * F] (from `alloc(shape, dtype)`) and the activation kernel follows."""
    ops._need(a, "a", dims=2); ops._need(weight, "weight", dims=3); ops._need(out, "out", dims=2)
    G, two_f, K = weight.shape
    F = two_f // 2
    if activation not in ("silu", ops.CLAMPED_ACTIVATION):
        raise KernelError(f"grouped_silu_mul: activation {activation!r}")
    if two_f % 2 or tuple(out.shape) != (rows, F):
        raise KernelError("grouped_silu_mul: the weight holds gate rows over up rows, the output one column per pair")
    if row_scale is not None:
        ops._need(row_scale, "row_scale", torch.float32)
    if mma_supported(a, weight):
        ops._need(group_offsets, "group_offsets", torch.int32, 1)
        if a_rows is not None:
            ops._need(a_rows, "a_rows", torch.int32, 1)
        if pair_supported(a, weight) and pair_pays(rows, G, two_f, weight.stride(0) * 2, sm_count(a.device)):
            _pair(a, weight, out, rows=rows, outputs=F, group_offsets=group_offsets, a_rows=a_rows, a_row_div=a_row_div, c_rows=None, dual=True,
                  act=ops.activation_code(activation, limit), row_scale=row_scale, row_tile=row_tile, alloc=alloc, error_flag=error_flag)
            return
        L = ops.lib(MMA_SOURCE)
        build.check(L, L.mlb_grouped_mma(
            a.data_ptr(), a.stride(0), 0, weight.data_ptr(), weight.stride(1), weight.stride(0), out.data_ptr(), out.stride(0), 0,
            group_offsets.data_ptr(), ops._ptr(a_rows), None, int(a_row_div), None, 0, F, int(rows), F, K, G,
            ops.dtype_tag(out), int(row_tile), ops.activation_code(activation, limit), ops._ptr(row_scale), 0, ops._stream()))
        return
    row_tile = min(row_tile, 64)
    gate_up = alloc((rows, two_f), a.dtype) if alloc is not None else torch.empty((rows, two_f), dtype=a.dtype, device=a.device)
    grouped_linear(a, weight, gate_up, rows=rows, group_offsets=group_offsets, a_rows=a_rows, a_row_div=a_row_div, row_tile=row_tile,
                   row_scale=row_scale)
    ops.gated_act_mul(gate_up, out, activation, limit)
