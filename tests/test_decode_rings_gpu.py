"""Decode attention whose keys come by way of each warp's own ring in shared memory (fa_decode_t_kernel in csrc/attention_mma.cu): the bits of the form
that loads them into registers."""
import pytest
import torch

DEV = "cuda"


def test_a_captured_step_is_planned_again_where_the_rings_begin_to_pay():
    from types import SimpleNamespace
    from microllm_rocm_b200.kernels import attention
    ctx = SimpleNamespace(extras={("attention_rings", 8, False, 1 << 30): False, ("attention_rings", 8, True, 1 << 30): False, ("attention_rings", 8, False, 1024): False})
    assert not attention.decode_plan_stale(ctx, 3199) and attention.decode_plan_stale(ctx, 3200)
    attention.forget_plans(ctx)
    assert not ctx.extras and not attention.decode_plan_stale(ctx, 3200)


# one sequence (eight warps a CTA), a few, many; fewer tiles than a ring
# holds, none, more; windows whose first pages were given back; the first keys kept; lists of a mixed step
@pytest.mark.gpu
@pytest.mark.parametrize("lens, nkv, group", [([1], 2, 6), ([700], 2, 6), ([5, 17, 1, 3000], 4, 7), ([1, 2, 16, 33, 95, 96, 97, 112, 113, 400, 1600] * 6, 2, 6), ([900] * 30, 4, 8)])
@pytest.mark.parametrize("window, keep, extra", [(None, 0, False), (100, 0, True), (48, 20, False)])
def test_bits_of_the_registers(lens, nkv, group, window, keep, extra):
    from microllm_rocm_b200.kernels import attention
    from microllm_rocm_b200.parts.base import StepContext
    d, page, A, nh = 128, 32, len(lens), nkv * group
    news = [3 if extra and a == 0 and n >= 3 else 1 for a, n in enumerate(lens)]       # a prompt portion beside decoded tokens: those are listed
    g = torch.Generator(DEV).manual_seed(A)
    on = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    blocks = [-(-n // page) for n in lens]
    order = torch.randperm(sum(blocks) + 2, generator=torch.Generator().manual_seed(A)).tolist()
    pages = torch.randn(sum(blocks) + 2, 2, nkv, page, d, generator=g, device=DEV).bfloat16()
    table = torch.full((A, max(blocks)), -1, dtype=torch.int32)
    for a, b in enumerate(blocks):
        table[a, :b] = torch.tensor(order[:b])
        order = order[b:]
        pages[table[a, b - 1].long(), :, :, (lens[a] - 1) % page + 1:] = float("nan")         # what no token has written yet
        if window and not keep:
            table[a, :max(0, lens[a] - news[a] + 1 - window) // page] = -1
    starts = [0]
    for n in news:
        starts.append(starts[-1] + n)
    pos0 = [n - k for n, k in zip(lens, news)]
    q = torch.randn(starts[-1], nh * d, generator=g, device=DEV).bfloat16()
    sink = torch.randn(nh, device=DEV) if keep else None

    def run(own):
        positions = on([p + i for p, n in zip(pos0, news) for i in range(n)])
        ctx = StepContext(num_tokens=starts[-1], num_seqs=A, token_ids=positions, positions=positions, token_seq=on([a for a, n in enumerate(news) for _ in range(n)]),
                          seq_starts=on(starts), seq_pos0=on(pos0), seq_lens=on(lens), block_tables={}, state_slots=None, logit_rows=None,
                          error_flag=torch.zeros(1, dtype=torch.int32, device=DEV), seq_starts_host=starts, seq_pos0_host=pos0, max_new_tokens=max(news),
                          max_seq_len=max(lens))
        out = torch.full_like(q, float("nan"))
        attention.OWN_RINGS, attention.DECODE_RING = own, False
        try:
            attention.paged_attention(q, pages, out, ctx, table.to(DEV), nh, nkv, d, d ** -0.5, window, sink=sink, keep_first=keep)
        finally:
            attention.OWN_RINGS = attention.DECODE_RING = None
        assert int(ctx.error_flag.item()) == 0
        return out
    got = run(True)
    assert torch.equal(got, run(False)) and bool(torch.isfinite(got.float()).all())
