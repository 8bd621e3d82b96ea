"""Latent attention's own kernels (`csrc/latent.cu`): what follows the fused input projection (norm of the latent,
rotation, cache store, query split, gate activation) and the attention over the compressed cache."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import build, ops
from .build import KernelError

SOURCE = "latent.cu"
ops.register_signatures(SOURCE, {
    "mlb_latent_prepare": [c_void_p, c_longlong, c_int, c_longlong, c_longlong, c_longlong, c_longlong, c_void_p, c_float,
                           c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int, c_float, c_void_p, c_void_p, c_int, c_void_p, c_int,
                           c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p],
    "mlb_latent_compress": [c_void_p, c_longlong, c_int, c_longlong, c_longlong, c_int, c_void_p, c_void_p, c_int, c_longlong, c_void_p,
                            c_float, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int, c_float, c_void_p, c_int, c_int, c_int,
                            c_int, c_int, c_int, c_void_p, c_void_p],
    "mlb_latent_attention_plain": [c_void_p, c_int, c_void_p, c_int, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_void_p,
                                   c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_float, c_void_p, c_void_p],
})

MAX_RANK = 512
MAX_KEY_WIDTH = 640

MMA_SOURCE = "latent_mma.cu"
ops.register_signatures(MMA_SOURCE, {
    "mlb_latent_mma_widths": [c_int],
    "mlb_latent_attention_mma": [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p,
                                 c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_float, c_void_p, c_void_p],
})
TC_SOURCE = "latent_tc.cu"
ops.register_signatures(TC_SOURCE, {
    "mlb_latent_tc_rows_per_tile": [],
    "mlb_latent_attention_tc": [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                c_int, c_int, c_float, c_void_p, c_void_p],
})
TC_ROWS_PER_TILE = 128              # of which a CTA of the tcgen05 kernel owns half the output columns
ROWS_PER_TILE = 16                  # (token, head) rows of one sequence that a group of warps of the tensor-core kernel owns
KEYS_PER_TILE = 32
MIN_KEY_TILES_PER_SPLIT = 4         # a CTA that shares a work item's keys streams 128 of them at least
MAX_SPLITS = 64
GROUPS = None                       # 1 or 2: tests set the groups of rows a CTA holds (where the keys are not split); None: _plan decides
TCGEN05 = None                      # tests set which sequences go to the tcgen05 kernel: True all (where the keys are not split), False none; None: the rule
USE_TENSOR_CORES = True             # tests set it to False to run the plain kernel on the same inputs


def mma_supported(rank: int, rot_dim: int) -> bool:
    return rank % 32 == 0 and (rank + rot_dim) % 16 == 0 and rank <= MAX_RANK


def mma_sources(rank: int, rot_dim: int):
    return [(MMA_SOURCE, {"LAT_R": rank, "LAT_DR": rot_dim})] if mma_supported(rank, rot_dim) else []


def tc_supported(rank: int, rot_dim: int, page_size: int = KEYS_PER_TILE) -> bool:
    """The width that was measured and whose CTA has a multiprocessor to itself (csrc/latent_tc.cu says why it must)."""
    return rank == 512 and rot_dim == 64 and page_size % 8 == 0 and (KEYS_PER_TILE % page_size == 0 or page_size % KEYS_PER_TILE == 0)


def tc_sources(rank: int, rot_dim: int):
    return [(TC_SOURCE, {"LAT_R": rank, "LAT_DR": rot_dim})] if tc_supported(rank, rot_dim) else []


def key_splits(num_work: int, max_seq_len: int, sms: int) -> int:
    """How many CTAs share the keys of one work item: enough to give every multiprocessor two CTAs, while each still
    streams a few key tiles."""
    key_tiles = max(1, -(-max_seq_len // KEYS_PER_TILE))
    return max(1, min((2 * sms) // max(1, num_work), key_tiles // MIN_KEY_TILES_PER_SPLIT, MAX_SPLITS))


def two_groups_pay(tiles: int, mean_keys: float, most_keys: int, sms: int) -> bool:
    """Whether a CTA holds two groups of 16 rows, which share a ring of keys: from five tiles of 16 rows a multiprocessor on, and from four
    where the tiles see about as many keys.  The CTAs are half as many, and with four tiles a multiprocessor all of them run at
    once: the longest then sets the time.  Measured (512 + 64 wide, 148 SMs, us, one group / two): 16 heads, a prompt of 592 tokens
    (592 tiles) 59 / 71, 640 69 / 73, 704 84 / 81, 740 92 / 83, 2,048 577 / 434; 592 tokens behind 1,500 288 / 235, 20 times 32 behind
    2,000 471 / 382; 3 times 200 29 / 30; 4 heads, 2,500 tokens (625 tiles) 220 / 261, 3,000 334 / 315."""
    return tiles >= 5 * sms or (tiles >= 4 * sms and mean_keys >= 0.7 * most_keys)


def _plan(ctx, heads: int):
    """Work items of a step ((sequence, first row) per 16 rows of a sequence's new (token, head) rows, or 32; long causal
    ranges first), the key split and the groups of 16 rows a CTA holds (two_groups_pay; one where the keys are split), shared by every
    layer with this many heads."""
    from .device import sm_count
    key = ("latent_mma", heads)
    plan = ctx.extras.get(key)
    if plan is not None:
        return plan
    starts = ctx.seq_starts_host
    device = ctx.positions.device
    sms = sm_count(device)
    rows = [(starts[a + 1] - starts[a]) * heads for a in range(ctx.num_seqs)]
    tiles = sum(-(-n // ROWS_PER_TILE) for n in rows)
    splits = key_splits(tiles, ctx.max_seq_len, sms) if ctx.decode_only or tiles <= 32 else 1
    front = ctx.seq_pos0_host or [0] * ctx.num_seqs
    new = [starts[a + 1] - starts[a] for a in range(ctx.num_seqs)]
    mean = sum(n * (p + 0.5 * (n + 1)) for n, p in zip(new, front)) / max(1, sum(new))           # keys that a new token sees
    groups = 2 if splits == 1 and not ctx.decode_only and two_groups_pay(tiles, mean, max((n + p for n, p in zip(new, front)), default=0), sms) else 1
    if GROUPS is not None and splits == 1:
        groups = GROUPS
    work = []
    for a in range(ctx.num_seqs):
        work += [(front[a] + first // heads, a, first) for first in range(0, rows[a], groups * ROWS_PER_TILE)]
    if not ctx.decode_only:
        work.sort(key=lambda item: -item[0])
    work_dev = ops.upload([x for _, a, first in work for x in (a, first)], "int32", device)
    plan = ctx.extras[key] = (work_dev, len(work), splits, groups)
    return plan


def tc_pays(tiles: int, mean_keys: float) -> bool:
    """Whether a step's sequences of 128 (token, head) rows and more, `tiles` tiles of 128 rows whose tokens see `mean_keys` keys, go to the tcgen05
    kernel: a CTA takes 9 us before its first tile of keys and 1.8 for each, so many tiles want 64 keys and few tiles thousands.
    Measured (512 + 64 wide, 148 SMs, us, mma.sync / tcgen05): 16 heads, a prompt of 2,048 tokens 427 / 242, 1,024 118 / 78, 512 47 / 41, 256 26 / 25,
    128 13 / 18; 512 behind 2,000 356 / 152, 64 behind 2,000 130 / 120; 8 times 128 tokens 32.6 / 30.4, 45 13 / 15, 16 behind 1,000 80 / 66,
    8 behind 1,000 62 / 66; 40 times 40 35.0 / 36.3; 4 heads, 2,048 tokens 163 / 122, 512 36.8 / 38.3; 64 heads, 128 tokens 22 / 19."""
    return (tiles >= 32 and mean_keys >= 64) or tiles * mean_keys >= 12000


def _tc_plan(ctx, heads: int):
    """(work of the tcgen05 kernel, its length, work of the mma.sync kernel, its length, its groups) of a step whose keys are not split: items
    as in _plan, of 128 rows and of 16 or 32; None where the first would be empty."""
    from .device import sm_count
    key = ("latent_tc", heads)
    if key in ctx.extras:
        return ctx.extras[key]
    device = ctx.positions.device
    sms = sm_count(device)
    starts, front = ctx.seq_starts_host, ctx.seq_pos0_host or [0] * ctx.num_seqs
    new = [starts[a + 1] - starts[a] for a in range(ctx.num_seqs)]
    rows = [n * heads for n in new]
    takes = [n > 0 and (n >= TC_ROWS_PER_TILE if TCGEN05 is None else TCGEN05) for n in rows]
    tiles = sum(-(-n // TC_ROWS_PER_TILE) for n, t in zip(rows, takes) if t)
    mean = sum(n * (p + 0.5 * (n + 1)) for n, p, t in zip(new, front, takes) if t) / max(1, sum(n for n, t in zip(new, takes) if t))
    rest = [a for a in range(ctx.num_seqs) if not takes[a]]

    def upload(step, which):
        work = [(front[a] + min(rows[a], first + step) // heads, a, first) for a in which for first in range(0, rows[a], step)]
        work.sort(key=lambda item: -item[0])
        return ops.upload([x for _, a, first in work for x in (a, first)], "int32", device) if work else None, len(work)
    plan = None
    if 0 < tiles < 65536 and (TCGEN05 or tc_pays(tiles, mean)):
        # Two groups a CTA from five tiles a multiprocessor on and not from four, as two_groups_pay has it for tiles that see as many keys: beside the other
        # kernel the CTAs do not all run at once.  16 heads, beside a prompt of 700, us, one / two: 85 x 7 tokens behind 1,500 (595 tiles) 366 / 404, 90 x 7 behind
        # 500 165 / 169, 100 x 7 behind 1,000 (700) 288 / 294, 600 x 1 behind 300 119 / 151, but 160 x 4 behind 1,000 (640) 284 / 254; 110 x 7 behind 200
        # (770) 105 / 108, 130 x 7 behind 800 (910) 303 / 260, 400 x 2 behind 300 (800) 136 / 135.
        groups = 2 if sum(-(-rows[a] // ROWS_PER_TILE) for a in rest) >= 5 * sms else 1
        plan = (*upload(TC_ROWS_PER_TILE, [a for a in range(ctx.num_seqs) if takes[a]]), *upload(groups * ROWS_PER_TILE, rest), groups)
    ctx.extras[key] = plan
    return plan


def plan_stale(ctx, max_seq_len: int) -> bool:
    from .device import sm_count
    for key, plan in ctx.extras.items():
        if isinstance(key, tuple) and key and key[0] == "latent_mma":
            if key_splits(plan[1], max_seq_len, sm_count(ctx.positions.device)) != plan[2]:
                return True
    return False


def forget_plans(ctx) -> None:
    for key in [k for k in ctx.extras if isinstance(k, tuple) and k and k[0] == "latent_mma"]:
        del ctx.extras[key]


def attention(q: torch.Tensor, pages: torch.Tensor, out: torch.Tensor, sink: Optional[torch.Tensor], ctx,
              block_table: torch.Tensor, heads: int, rank: int, rot_dim: int, scale: float, window: Optional[int]) -> None:
    """The step's attention over the compressed cache: bf16 on the tensor cores when the widths suit them (sequences of many new rows on
    the tcgen05 kernel, which gives the same bits as the mma.sync one; the two write disjoint rows), else (and always in fp32) the plain
    kernel."""
    if not (USE_TENSOR_CORES and q.dtype == torch.bfloat16 and pages.dtype == torch.bfloat16 and out.dtype == torch.bfloat16
            and mma_supported(rank, rot_dim)):
        attention_plain(q, pages, out, sink, ctx.positions, ctx.token_seq, block_table, heads, rank, rot_dim, scale, window,
                        ctx.error_flag)
        return
    ops._need(q, "q", torch.bfloat16, 2); ops._need(pages, "pages", torch.bfloat16, 3); ops._need(out, "out", torch.bfloat16, 2)
    T = q.shape[0]
    num_pages, page_size, width = pages.shape
    if width != rank + rot_dim or q.shape[1] != heads * width or tuple(out.shape) != (T, heads * rank):
        raise KernelError("latent.attention: shapes do not agree")
    work, num_work, splits, groups = _plan(ctx, heads)
    tc_work = side = None
    if splits == 1 and not ctx.decode_only and GROUPS is None and TCGEN05 is not False and tc_supported(rank, rot_dim, page_size):
        plan = _tc_plan(ctx, heads)
        if plan is not None:
            tc_work, num_tc, work, num_work, groups = plan
    if tc_work is not None and num_work:     # other sequences, other rows: the two launches run side by side
        side = ops.side_stream()
        ops.fork(side)
    try:
        if tc_work is not None:
            L = ops.lib(TC_SOURCE, {"LAT_R": rank, "LAT_DR": rot_dim})
            build.check(L, L.mlb_latent_attention_tc(
                q.data_ptr(), pages.data_ptr(), out.data_ptr(), ops._ptr(sink), ctx.seq_starts.data_ptr(), ctx.seq_pos0.data_ptr(), block_table.data_ptr(),
                tc_work.data_ptr(), num_tc, block_table.shape[1], num_pages, page_size, heads, int(window or 0), T * heads, float(scale),
                ops._ptr(ctx.error_flag), ops._stream() if side is None else side))
            if num_work == 0:
                return
        part_o = part_ml = None
        if splits > 1:
            part_o = ctx.buffer("latent.part_o", (splits, T * heads, rank), torch.float32)
            part_ml = ctx.buffer("latent.part_ml", (splits, T * heads, 2), torch.float32)
        L = ops.lib(MMA_SOURCE, {"LAT_R": rank, "LAT_DR": rot_dim})
        build.check(L, L.mlb_latent_attention_mma(
            q.data_ptr(), pages.data_ptr(), out.data_ptr(), ops._ptr(sink), ctx.seq_starts.data_ptr(), ctx.seq_pos0.data_ptr(),
            block_table.data_ptr(), work.data_ptr(), num_work, ops._ptr(part_o), ops._ptr(part_ml), block_table.shape[1], num_pages,
            page_size, heads, int(window or 0), splits, groups, T * heads, float(scale), ops._ptr(ctx.error_flag), ops._stream()))
    finally:
        if side is not None:                 # (also where a launch is refused: whoever catches that lets go of the tensors, and may be capturing)
            ops.join(side)


def sources():
    return [(SOURCE, {})]


def check_sizes(rank: int, rot_dim: int) -> None:
    if rank <= 0 or rank > MAX_RANK or rank + rot_dim > MAX_KEY_WIDTH:
        raise KernelError(f"latent attention: a latent of {rank} and a rotated part of {rot_dim} exceed {MAX_RANK} / {MAX_KEY_WIDTH}")


def prepare(proj: torch.Tensor, *, q_col: int, kv_col: int, gate_col: int, norm_weight: torch.Tensor, eps: float,
            positions: torch.Tensor, token_seq: torch.Tensor, block_table: Optional[torch.Tensor], inv_freq: torch.Tensor,
            rot_dims: int, q_plain: torch.Tensor, q_full: torch.Tensor, pages: Optional[torch.Tensor],
            gate_out: Optional[torch.Tensor], heads: int, dim: int, rot_dim: int, rank: int,
            error_flag: Optional[torch.Tensor], interleaved: bool = False, magnitude: float = 1.0) -> None:
    """proj: the fused projection [T, N] fp32 or its [S, T, N] partial sums; see csrc/latent.cu for what goes where.
    pages [num_pages, page_size, rank + rot_dim]; None: a run that reads another run's cache stores nothing."""
    n_partials, stride = 1, 0
    first = proj
    if proj.dim() == 3:
        ops._need(proj, "proj", torch.float32, 3)
        n_partials, stride = proj.shape[0], proj.shape[1] * proj.shape[2]
        first = proj[0]
    ops._need(first, "proj", torch.float32, 2)
    T = first.shape[0]
    ops._need(q_plain, "q_plain", dims=2); ops._need(q_full, "q_full", q_plain.dtype, 2)
    ops._need(norm_weight, "norm_weight", torch.float32, 1); ops._need(inv_freq, "inv_freq", torch.float32, 1)
    ops._need(positions, "positions", torch.int32, 1); ops._need(token_seq, "token_seq", torch.int32, 1)
    if (tuple(q_plain.shape) != (T, heads * dim) or tuple(q_full.shape) != (T, heads * (rank + rot_dim))
            or norm_weight.shape[0] != rank or inv_freq.shape[0] * 2 != rot_dims or positions.shape[0] != T):
        raise KernelError("latent.prepare: shapes do not agree")
    gate_width = 0
    if gate_out is not None:
        ops._need(gate_out, "gate_out", torch.float32, 2)
        gate_width = gate_out.shape[1]
        if gate_out.shape[0] != T:
            raise KernelError("latent.prepare: one gate row per token")
    if max(q_col + heads * (dim + rot_dim), kv_col + rank + rot_dim if pages is not None else 0, gate_col + gate_width) > first.shape[1]:
        raise KernelError("latent.prepare: a column range runs past the projection")
    num_pages = page_size = max_blocks = 0
    if pages is not None:
        ops._need(pages, "pages", dims=3); ops._need(block_table, "block_table", torch.int32, 2)
        num_pages, page_size, width = pages.shape
        if width != rank + rot_dim:
            raise KernelError(f"latent.prepare: pages {tuple(pages.shape)} do not hold rows of {rank} + {rot_dim}")
        max_blocks = block_table.shape[1]
    L = ops.lib(SOURCE)
    build.check(L, L.mlb_latent_prepare(
        first.data_ptr(), first.stride(0), n_partials, stride, q_col, kv_col, gate_col, norm_weight.data_ptr(), float(eps),
        positions.data_ptr(), token_seq.data_ptr(), ops._ptr(block_table), max_blocks, inv_freq.data_ptr(), int(rot_dims),
        1 if interleaved else 0, float(magnitude), q_plain.data_ptr(), q_full.data_ptr(), ops.dtype_tag(q_plain), ops._ptr(pages),
        ops.dtype_tag(pages) if pages is not None else ops.F32, ops._ptr(gate_out), num_pages, page_size, T, heads, dim,
        rot_dim, rank, gate_width, ops._ptr(error_flag), ops._stream()))


def compress(proj: torch.Tensor, *, cq_col: int, cq_weight: torch.Tensor, cq_out: torch.Tensor, kv_col: int, norm_weight: torch.Tensor,
             eps: float, positions: torch.Tensor, token_seq: torch.Tensor, block_table: Optional[torch.Tensor], inv_freq: torch.Tensor,
             rot_dims: int, interleaved: bool, magnitude: float, pages: Optional[torch.Tensor], rot_dim: int, rank: int,
             error_flag: Optional[torch.Tensor]) -> None:
    """Out of one projection (fp32 rows or their partial sums): the token's cache row, as in `prepare`, and the queries' own latent
    cq_out [T, RQ] = columns cq_col.. / rms * cq_weight in cq_out's dtype.  pages None: a run that stores nothing."""
    n_partials, stride, first = 1, 0, proj
    if proj.dim() == 3:
        ops._need(proj, "proj", torch.float32, 3)
        n_partials, stride, first = proj.shape[0], proj.shape[1] * proj.shape[2], proj[0]
    ops._need(first, "proj", torch.float32, 2); ops._need(cq_out, "cq_out", dims=2)
    ops._need(cq_weight, "cq_weight", torch.float32, 1); ops._need(norm_weight, "norm_weight", torch.float32, 1)
    ops._need(inv_freq, "inv_freq", torch.float32, 1); ops._need(positions, "positions", torch.int32, 1)
    T, width = first.shape
    rq = cq_out.shape[1]
    if (cq_out.shape[0] != T or cq_weight.shape[0] != rq or norm_weight.shape[0] != rank or inv_freq.shape[0] * 2 != rot_dims
            or positions.shape[0] != T or max(cq_col + rq, kv_col + rank + rot_dim) > width):
        raise KernelError("latent.compress: shapes do not agree")
    num_pages = page_size = max_blocks = 0
    if pages is not None:
        ops._need(pages, "pages", dims=3); ops._need(block_table, "block_table", torch.int32, 2)
        num_pages, page_size, page_width = pages.shape
        if page_width != rank + rot_dim:
            raise KernelError(f"latent.compress: pages {tuple(pages.shape)} do not hold rows of {rank} + {rot_dim}")
        max_blocks = block_table.shape[1]
    L = ops.lib(SOURCE)
    build.check(L, L.mlb_latent_compress(
        first.data_ptr(), first.stride(0), n_partials, stride, cq_col, rq, cq_weight.data_ptr(), cq_out.data_ptr(), ops.dtype_tag(cq_out),
        kv_col, norm_weight.data_ptr(), float(eps), positions.data_ptr(), token_seq.data_ptr(), ops._ptr(block_table), max_blocks,
        inv_freq.data_ptr(), int(rot_dims), 1 if interleaved else 0, float(magnitude), ops._ptr(pages),
        ops.dtype_tag(pages) if pages is not None else ops.F32, num_pages, page_size, T, rot_dim, rank, ops._ptr(error_flag), ops._stream()))


def attention_plain(q: torch.Tensor, pages: torch.Tensor, out: torch.Tensor, sink: Optional[torch.Tensor],
                    positions: torch.Tensor, token_seq: torch.Tensor, block_table: torch.Tensor, heads: int, rank: int,
                    rot_dim: int, scale: float, window: Optional[int], error_flag: Optional[torch.Tensor]) -> None:
    """q [T, heads * (rank + rot_dim)], pages [num_pages, page_size, rank + rot_dim], out [T, heads * rank]."""
    ops._need(q, "q", dims=2); ops._need(pages, "pages", dims=3); ops._need(out, "out", dims=2)
    ops._need(block_table, "block_table", torch.int32, 2)
    T = q.shape[0]
    num_pages, page_size, width = pages.shape
    if width != rank + rot_dim or q.shape[1] != heads * width or tuple(out.shape) != (T, heads * rank) or positions.shape[0] != T:
        raise KernelError("latent.attention_plain: shapes do not agree")
    if sink is not None:
        ops._need(sink, "sink", torch.float32, 1)
        if sink.shape[0] != heads:
            raise KernelError("latent.attention_plain: one sink per head")
    L = ops.lib(SOURCE)
    build.check(L, L.mlb_latent_attention_plain(
        q.data_ptr(), ops.dtype_tag(q), pages.data_ptr(), ops.dtype_tag(pages), out.data_ptr(), ops.dtype_tag(out), ops._ptr(sink),
        positions.data_ptr(), token_seq.data_ptr(), block_table.data_ptr(), block_table.shape[1], num_pages, page_size, T,
        heads, rank, rot_dim, int(window or 0), float(scale), ops._ptr(error_flag), ops._stream()))
