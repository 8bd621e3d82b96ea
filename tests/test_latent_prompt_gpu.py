"""Latent attention of prompts on the tcgen05 kernel (csrc/latent_tc.cu): the bits of the mma.sync kernel, which has float64 as its judge elsewhere."""
import pytest
import torch

from microllm_rocm_b200.kernels import latent

DEV = "cuda"
RANK, ROT = 512, 64
pytestmark = pytest.mark.gpu

def step(seqs, heads, page, seed, window=None):
    """(context, queries, pages, table, cache rows of each sequence): the pool's other rows, and pages in front of the window, are not there."""
    from microllm_rocm_b200.parts.base import StepContext
    starts = [0]
    for n, _ in seqs:
        starts.append(starts[-1] + n)
    T, A, width = starts[-1], len(seqs), RANK + ROT
    on = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    positions = on([p + i for n, p in seqs for i in range(n)])
    ctx = StepContext(num_tokens=T, num_seqs=A, token_ids=positions, positions=positions, token_seq=on([a for a, (n, _) in enumerate(seqs) for _ in range(n)]),
                      seq_starts=on(starts), seq_pos0=on([p for _, p in seqs]), seq_lens=on([n + p for n, p in seqs]), block_tables={}, state_slots=None,
                      logit_rows=None, error_flag=torch.zeros(1, dtype=torch.int32, device=DEV), seq_starts_host=starts, seq_pos0_host=[p for _, p in seqs],
                      max_new_tokens=max(n for n, _ in seqs), max_seq_len=max(n + p for n, p in seqs))
    g = torch.Generator(DEV).manual_seed(seed)
    q = (torch.randn(T, heads * width, generator=g, device=DEV) * 0.4).bfloat16()
    blocks = [-(-(n + p) // page) for n, p in seqs]
    order = torch.randperm(sum(blocks) + 2, generator=torch.Generator().manual_seed(seed)).tolist()
    pages = torch.full((sum(blocks) + 2, page, width), float("nan"), dtype=torch.bfloat16, device=DEV)
    table, held = torch.full((A, max(blocks)), -1, dtype=torch.int32), []
    for a, (n, p) in enumerate(seqs):
        table[a, :blocks[a]] = torch.tensor(order[:blocks[a]])
        order = order[blocks[a]:]
        rows, at = torch.randn(n + p, width, generator=g, device=DEV).bfloat16(), torch.arange(n + p)
        pages[table[a].long()[at // page].to(DEV), (at % page).to(DEV)] = rows
        lost = max(0, p - window + 1) // page if window else 0                # pages in front of the window were given back
        if lost:
            pages[table[a, :lost].long().to(DEV)] = float("nan")
            table[a, :lost] = -1
        held.append(rows)
    return ctx, q, pages, table.to(DEV), held


def run(ctx, q, pages, table, sinks, heads, window, tc=True):
    ctx.extras.clear()
    latent.TCGEN05 = tc
    out = torch.full((q.shape[0], heads * RANK), float("nan"), dtype=torch.bfloat16, device=DEV)
    try:
        latent.attention(q, pages, out, sinks, ctx, table, heads, RANK, ROT, (RANK + ROT) ** -0.5, window)
    finally:
        latent.TCGEN05 = None
    assert (ctx.extras.get(("latent_tc", heads)) is not None) == tc
    assert int(ctx.error_flag.item()) == 0
    return out


@pytest.mark.parametrize("heads, seqs, page, window, sink", [
    (16, [(64, 0)], 64, None, False), (16, [(65, 63), (100, 64), (3, 9), (1, 200)], 16, None, True), (16, [(130, 700), (257, 0)], 8, 300, True),
    (16, [(200, 1500)], 32, 40, False), (5, [(333, 1), (210, 129)], 16, 128, True), (1, [(1030, 50)], 64, 7, True), (40, [(26, 0), (77, 65)], 16, None, False)])
def test_bits_of_the_mma_kernel(heads, seqs, page, window, sink):
    """Whole and partial tiles of 128 rows and of 32 keys, tokens that straddle tiles, one row, portions behind a cache, windows, sinks; the pool's other
    rows are not numbers."""
    ctx, q, pages, table, _ = step(seqs, heads, page, heads + seqs[0][0], window)
    sinks = torch.randn(heads, device=DEV) if sink else None
    got = run(ctx, q, pages, table, sinks, heads, window)
    pages = torch.nan_to_num(pages)              # (a row of the other kernel takes part in what its sixteen see)
    assert torch.equal(got, run(ctx, q, pages, table, sinks, heads, window, tc=False)) and bool(torch.isfinite(got.float()).all())


def test_the_rule_divides_a_step():
    """Sequences of many rows and of few in one step: two launches, all rows written, the same bits."""
    heads, seqs = 16, [(3, 40), (700, 0), (1, 900), (640, 64), (5, 0)]
    ctx, q, pages, table, _ = step(seqs, heads, 16, 5)
    out = torch.full((q.shape[0], heads * RANK), float("nan"), dtype=torch.bfloat16, device=DEV)
    latent.attention(q, pages, out, None, ctx, table, heads, RANK, ROT, (RANK + ROT) ** -0.5, None)
    work, num, rest, num_rest, groups = ctx.extras[("latent_tc", heads)]
    assert sorted(set(work.tolist()[::2])) == [1, 3] and sorted(set(rest.tolist()[::2])) == [0, 2, 4] and groups == 1
    assert torch.equal(out, run(ctx, q, torch.nan_to_num(pages), table, None, heads, None, tc=False))


@pytest.mark.parametrize("window", [None, 20])
def test_keys_that_a_row_does_not_see_do_not_reach_it(window):
    """Cache rows that are not finite, at the causal edge of a tile of eight tokens, at a window's start and in the middle."""
    heads, seqs, page = 16, [(70, 0), (90, 50)], 16
    ctx, q, pages, table, _ = step(seqs, heads, page, 3)
    clean = run(ctx, q, pages, table, None, heads, window)
    for a, position, value in ((0, 1, "nan"), (0, 32, "inf"), (0, 63, "nan"), (0, 69, "-inf"), (1, 51, "nan"), (1, 86, "nan"), (1, 31, "inf"), (1, 139, "nan")):
        spoiled = pages.clone()
        spoiled[int(table[a, position // page]), position % page] = float(value)
        got = run(ctx, q, spoiled, table, None, heads, window)
        start, (n, p) = ctx.seq_starts_host[a], seqs[a]
        other = slice(ctx.seq_starts_host[1 - a], ctx.seq_starts_host[2 - a])
        assert torch.equal(got[other], clean[other])
        for i in range(n):
            sees = p + i >= position and (window is None or p + i - window < position)
            assert bool((~torch.isfinite(got[start + i].float())).any()) == sees, (a, position, i)
            if not sees:
                assert torch.equal(got[start + i], clean[start + i])


@pytest.mark.parametrize("warp", [0, 1, 2, 5, 7])
def test_a_held_back_warp_changes_nothing(warp):
    from microllm_rocm_b200.kernels import ops
    heads, seqs = 16, [(150, 200), (64, 0)]
    ctx, q, pages, table, _ = step(seqs, heads, 16, 9)
    clean = run(ctx, q, pages, table, None, heads, None)
    ops.TEST_DEFINES["latent_tc.cu"] = {"MLB_LAG_WARP": warp}
    try:
        assert torch.equal(run(ctx, q, pages, table, None, heads, None), clean)
    finally:
        ops.TEST_DEFINES.pop("latent_tc.cu")


@pytest.mark.parametrize("polls", [0, 1, 4])
def test_a_wait_that_runs_out_is_reported_and_leaves_nothing_behind(polls):
    """Every wait gives up after a few polls: the error flag says so (or, where none ran out, the rows are right), the kernel ends, and the next launch is as ever."""
    from microllm_rocm_b200.kernels import ops
    heads, seqs = 16, [(150, 200), (64, 0), (40, 700)]
    ctx, q, pages, table, _ = step(seqs, heads, 16, 9)
    clean = run(ctx, q, pages, table, None, heads, None)
    ops.TEST_DEFINES["latent_tc.cu"] = {"MLB_SPIN_LIMIT": polls}
    latent.TCGEN05 = True
    try:
        for _ in range(3):
            ctx.error_flag.zero_()
            out = torch.empty_like(clean)
            latent.attention(q, pages, out, None, ctx, table, heads, RANK, ROT, (RANK + ROT) ** -0.5, None)
            code = int(ctx.error_flag.item())
            assert 61 <= code <= 73 if polls == 0 else code == 0 or 61 <= code <= 73
            assert code != 0 or torch.equal(out, clean)
    finally:
        latent.TCGEN05 = None
        ops.TEST_DEFINES.pop("latent_tc.cu")
    ctx.error_flag.zero_()
    assert torch.equal(run(ctx, q, pages, table, None, heads, None), clean)
