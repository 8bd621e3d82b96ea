"""Which launches a call makes, and with what arguments, on the CPU: the launchers are stand-ins that note what they are called with, so a choice
that would race or overwrite on a device shows as an argument."""
import re
from types import SimpleNamespace

import pytest
import torch

from microllm_rocm_b200.kernels import build, ops


@pytest.fixture
def calls(monkeypatch):
    """[(launcher, {argument name: value})] of the calls made."""
    made = []

    class Library:
        def __init__(self, source):
            text = open(f"{build.CSRC}/{source}").read()
            self.names = {fn: [p.strip().split()[-1].lstrip("*") for p in params.split(",") if p.strip()]
                          for fn, params in re.findall(r"MLB_EXPORT\s+int\s+(\w+)\s*\(([^)]*)\)", text, re.S)}

        def __getattr__(self, fn):
            def launcher(*args):
                assert len(args) == len(self.names[fn])
                made.append((fn, dict(zip(self.names[fn], args))))
                return 0
            return launcher

    monkeypatch.setattr(ops, "lib", lambda source, defines=None: Library(source))
    monkeypatch.setattr(ops, "_need", lambda *args, **kwargs: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    return made


def lists(counts):
    """The lists of a step in which sequence a brings counts[a] tokens."""
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    on = lambda x: torch.tensor(x, dtype=torch.int32)
    return SimpleNamespace(num_tokens=starts[-1], num_seqs=len(counts), seq_starts=on(starts), seq_pos0=on([4] * len(counts)), error_flag=on([0]),
                           token_seq=on([a for a, n in enumerate(counts) for _ in range(n)]), max_new_tokens=max(counts), seq_starts_host=starts)


@pytest.mark.parametrize("counts, alone", [([1], True), ([1, 1, 1], True), ([2, 0], False), ([0, 2], False), ([3, 0, 0], False), ([2, 1, 0], False), ([2, 1], False)])
def test_only_steps_of_one_token_a_sequence_move_the_convolutions_state_in_its_launch(calls, monkeypatch, counts, alone):
    """As many tokens as sequences is not enough: a sequence of two tokens would have two threads on its state, and the second no sight of the first."""
    from microllm_rocm_b200.kernels import recurrent
    monkeypatch.setattr(recurrent, "_columns", lambda t, name: (None, t.shape[-1], 1, 0))
    T, C, taps, ctx = sum(counts), 12, 4, lists(counts)
    f = lambda *s: torch.zeros(*s)
    recurrent.short_conv(f(T, C), 0, f(C, taps), f(len(counts), taps - 1, C), ctx.token_seq, ctx, f(T, C), silu=False)
    assert [fn for fn, _ in calls] == ["mlb_short_conv"] + ([] if alone else ["mlb_short_conv_state"])
    assert calls[0][1]["move"] == (1 if alone else 0)


@pytest.mark.parametrize("captured", [False, True])
def test_library_products_on_second_streams_have_a_workspace_of_their_thread_or_captured_step(calls, monkeypatch, captured):
    """Every host thread has a second stream of its own, and nothing orders two of them: their products may not share a workspace, with each other or
    with the first stream's.  Those of one thread may, and theirs goes when the thread does; a captured step, which another thread may run again
    while the one that captured it goes on, has its own."""
    import gc
    import threading
    import weakref

    from microllm_rocm_b200.kernels import gemm_bf16
    from microllm_rocm_b200.parts.base import Mixer, StepContext
    from microllm_rocm_b200.parts.parallel import ParallelMixers
    monkeypatch.setattr(ops, "_stream", lambda: ops._launch_on.__dict__.get("side") or 1)
    monkeypatch.setattr(ops, "side_stream", lambda: 100 + threading.get_ident())
    monkeypatch.setattr(gemm_bf16, "_direct_library", lambda device: True)
    monkeypatch.setattr(gemm_bf16, "_workspaces", {})
    monkeypatch.setattr(gemm_bf16, "LIBRARY_WORKSPACE_BYTES", 64)

    class Main(Mixer):
        def forward(self, x, ctx, cache):
            on_device = SimpleNamespace(is_cuda=True, shape=x.shape, device=x.device, stride=x.stride, data_ptr=x.data_ptr)
            for role in ("in", "out"):
                y = gemm_bf16.library_linear(on_device, x, None, torch.float32, None, alloc=lambda shape, dtype: ctx.buffer(role, shape, dtype))
            return y

    class Aside(Main):
        beside_others = lambda self: True

    def context():
        ids = torch.zeros(8, dtype=torch.int32)
        return StepContext(num_tokens=8, num_seqs=1, token_ids=ids, positions=ids, token_seq=ids, seq_starts=ids, seq_pos0=ids, seq_lens=ids, block_tables={},
                           state_slots=ids, logit_rows=ids, error_flag=ids, captured=captured)
    mixer = ParallelMixers.__new__(ParallelMixers)
    mixer.branches = [("left", 1.0, "", Main()), ("right", 1.0, "", Aside())]
    contexts, used = [context(), context()], [None, None]
    lock, both, gone = threading.Lock(), threading.Barrier(2), []

    def work(i):
        with lock:
            calls.clear()
            for _ in range(2):                                # two layers of one step
                mixer.forward_terms(torch.zeros(8, 8), contexts[i], {})
            used[i] = [(a["stream"], a["workspace"]) for fn, a in calls if fn == "mlb_lt_matmul"]
            mixer.forward_terms(torch.zeros(8, 8), context(), {})          # another step of this thread
            used[i].append(next((a["stream"], a["workspace"]) for fn, a in calls[-4:] if fn == "mlb_lt_matmul" and a["stream"] != 1))
            gone.extend(weakref.ref(t) for t in list(contexts[i].extras.values()) + list(gemm_bf16._second_workspaces.__dict__.values()))
        both.wait(timeout=30)                                 # (until both have theirs)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    other = [u.pop()[1] for u in used]
    aside, first = [{w for s, w in u if s != 1} for u in used], [{w for s, w in u if s == 1} for u in used]
    assert [len(u) for u in used] == [8, 8] and all(len(s) == 1 for s in aside + first)
    assert aside[0] != aside[1] and first[0] == first[1] and not (aside[0] | aside[1]) & first[0]
    assert captured or other == [w for s in aside for w in s]             # (an eager step takes its thread's again)
    contexts.clear()
    gc.collect()
    assert gone and not any(r() is not None for r in gone)


@pytest.mark.parametrize("w_constant", [False, True])
def test_a_grouped_products_weights_are_read_ahead_only_on_the_callers_word(calls, monkeypatch, w_constant):
    """The kernel in front may be the one that writes them."""
    from microllm_rocm_b200.kernels import grouped
    a, w = torch.zeros(9, 3 * 64, dtype=torch.bfloat16), torch.zeros(3, 32, 64, dtype=torch.bfloat16)
    grouped.grouped_linear(a, w, torch.zeros(9, 96), rows=9, a_group_cols=64, c_group_cols=32, **({"w_constant": True} if w_constant else {}))
    assert calls[0][0] == "mlb_grouped_mma" and calls[0][1].get("w_constant", 1) == int(w_constant)


@pytest.mark.parametrize("refuses", ["mlb_latent_attention_tc", "mlb_latent_attention_mma", None])
def test_latent_attention_joins_the_second_stream_whichever_launch_refuses(calls, monkeypatch, refuses):
    """Whoever catches the error lets go of tensors that the other launch may still use, and may be capturing."""
    from microllm_rocm_b200.kernels import latent
    heads, seqs = 16, [(700, 0), (1, 900), (700, 0)]
    ctx = lists([n for n, _ in seqs])
    ctx.extras, ctx.seq_pos0_host, ctx.max_seq_len, ctx.positions, ctx.decode_only = {}, [p for _, p in seqs], 901, ctx.token_seq, False
    monkeypatch.setattr("microllm_rocm_b200.kernels.device.sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "upload", lambda values, dtype, device: torch.tensor(values, dtype=torch.int32))
    monkeypatch.setattr(ops, "side_stream", lambda: 200)
    monkeypatch.setattr(ops, "fork", lambda side: calls.append(("fork", side)))
    monkeypatch.setattr(ops, "join", lambda side: calls.append(("join", side)))

    def check(lib, status):
        if calls[-1][0] == refuses:
            raise build.KernelError("refused")
    monkeypatch.setattr(build, "check", check)
    T, bf16 = ctx.num_tokens, torch.bfloat16
    run = lambda: latent.attention(torch.zeros(T, heads * 576, dtype=bf16), torch.zeros(4, 16, 576, dtype=bf16), torch.zeros(T, heads * 512, dtype=bf16), None, ctx,
                                   torch.zeros(3, 64, dtype=torch.int32), heads, 512, 64, 0.1, None)
    if refuses is None:
        run()
    else:
        with pytest.raises(build.KernelError, match="refused"):
            run()
    names = [name for name, _ in calls]
    assert names[0] == "fork" and names[-1] == "join" and names.count("join") == 1
    assert [a["stream"] for name, a in calls if name == "mlb_latent_attention_tc"] == [200]


def paged_step(calls, monkeypatch, head_dim, nkv, group, lens, news=None):
    """The context behind one call of paged_attention over sequences of `lens` tokens, `news` of them new (one each)."""
    from microllm_rocm_b200.kernels import attention
    monkeypatch.setattr(attention, "sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "upload", lambda values, dtype, device: torch.tensor(values, dtype=torch.int32))
    monkeypatch.setattr(ops, "side_stream", lambda: 200)
    monkeypatch.setattr(ops, "fork", lambda side: None)
    monkeypatch.setattr(ops, "join", lambda side: None)
    news = news or [1] * len(lens)
    ctx = lists(news)
    ctx.extras, ctx.seq_pos0_host, ctx.max_seq_len, ctx.positions = {}, [n - k for n, k in zip(lens, news)], max(lens), ctx.token_seq
    ctx.mean_seq_len = sum(lens) / len(lens)
    q = torch.zeros(ctx.num_tokens, nkv * group * head_dim, dtype=torch.bfloat16)
    attention.paged_attention(q, torch.zeros(4, 2, nkv, 16, head_dim, dtype=torch.bfloat16), torch.zeros_like(q), ctx, torch.zeros(len(lens), 8, dtype=torch.int32),
                              nkv * group, nkv, head_dim, 0.1, None)
    return ctx


@pytest.mark.parametrize("head_dim, nkv, group, lens, later", [
    (128, 2, 6, [1000] * 4, 3200),                           # 8 CTAs share the keys: the rings take over at 400 keys each
    (64, 2, 6, [1000] * 4, None), (128, 2, 16, [1000] * 4, None),          # widths and groups that have no rings
    (128, 2, 6, [1100], None),                               # clusters of 16: none either
    (128, 4, 7, [9000] * 10, None)])                         # the TMA ring took the step
def test_a_captured_step_is_planned_again_only_where_another_kernel_would_run(calls, monkeypatch, head_dim, nkv, group, lens, later):
    from microllm_rocm_b200.kernels import attention
    ctx = paged_step(calls, monkeypatch, head_dim, nkv, group, lens)
    plan = next(v for k, v in ctx.extras.items() if k[0] == "attention_mma")
    assert plan[3] == (16 if len(lens) == 1 else plan[3]) and plan[9] == (len(lens) == 10)
    at = [n for n in range(max(lens), 20000, 100) if attention.decode_plan_stale(ctx, n, 148)]
    assert (at[0] if at else None) == later


@pytest.mark.parametrize("lens, news, rings", [
    ([3000, 200, 300, 250], [512, 1, 1, 1], False),          # a long prompt portion beside short decoded tokens
    ([3000, 2000, 3900, 200], [512, 1, 1, 1], True), ([3000, 700], [2, 300], False)])
def test_own_rings_go_by_the_tokens_that_take_them(calls, monkeypatch, lens, news, rings):
    """Keys a CTA of the listed sequences, not of the prompt portions beside them (which another kernel takes); none where nothing is listed."""
    from microllm_rocm_b200.kernels import attention
    ctx = paged_step(calls, monkeypatch, 128, 4, 7, lens, news)
    plan = next(v for k, v in ctx.extras.items() if k[0] == "attention_mma")
    decoded = [a for fn, a in calls if fn == "mlb_paged_attention_mma"]
    assert len(decoded) == (1 if 1 in news else 0) and all(bool(a["mode"] & 16) == rings for a in decoded)
    assert not decoded or attention.own_rings_pay(plan[8], max(n for n, k in zip(lens, news) if k == 1), False) == rings


def test_the_tcgen05_kernel_of_latent_prompts_takes_only_widths_that_fill_a_multiprocessor():
    """It asks for all of the tensor memory ahead of its wait for the kernel in front: where two CTAs fit one multiprocessor (128 and 256 wide), one of a launch
    behind could hold the memory that one of the launch in front still waits for, and wait for that launch."""
    from microllm_rocm_b200.kernels import latent
    assert latent.tc_supported(512, 64, 16) and latent.tc_sources(512, 64) == [(latent.TC_SOURCE, {"LAT_R": 512, "LAT_DR": 64})]
    for rank in (128, 256, 384):
        assert latent.mma_supported(rank, 64) and not latent.tc_supported(rank, 64, 16) and not latent.tc_sources(rank, 64)


def test_a_gated_few_row_product_on_the_second_stream_says_so(calls, monkeypatch):
    """There it starts early whatever its grid: its weights travel beside the first stream's kernels."""
    from microllm_rocm_b200.kernels import gemm_bf16
    monkeypatch.setattr(ops, "side_stream", lambda: 200)
    x, w, out = (torch.zeros(*s, dtype=torch.bfloat16) for s in ((4, 64), (64, 64), (4, 32)))
    gemm_bf16.gemv_silu_mul(x, w, out)
    with ops.on_side_stream():
        gemm_bf16.gemv_silu_mul(x, w, out)
    gemm_bf16.gemv_silu_mul(x, w, out)
    assert [a.get("beside") for fn, a in calls if fn == "mlb_gemv_gated"] == [0, 1, 0]


@pytest.mark.parametrize("nkv, group, lens, rings", [
    (4, 7, [4096], True), (4, 7, [4096] * 4, True), (8, 5, [4096] * 4, True), (4, 7, [4096] * 7, True), (4, 7, [3000] * 12, True), (2, 6, [4000] * 16, True),
    (4, 7, [4096] * 8, False), (4, 7, [4096, 600, 2000, 900, 4000, 300, 1500, 3000], True), (8, 5, [2400] * 8, True),      # eight of one length on clusters of eight
    (2, 6, [1700] * 24, False), (2, 6, [900] * 48, False), (2, 6, [900] * 72, False), (4, 7, [1000] * 20, False),             # many of one length
    (2, 6, [100 + 40 * i for i in range(41)] + [300] * 7, False), (2, 6, [300] * 40 + [1900], True), (2, 6, [80] * 30, False)])   # many, one or a few much longer
def test_own_rings_are_taken_where_they_were_the_faster_ones(calls, monkeypatch, nkv, group, lens, rings):
    """The same bits either way: sequences of one length that fill the device by their number were 1 to 3 % slower with them."""
    from microllm_rocm_b200.kernels import attention
    ctx = paged_step(calls, monkeypatch, 128, nkv, group, lens)
    plan = next(v for k, v in ctx.extras.items() if k[0] == "attention_mma")
    decoded = [a for fn, a in calls if fn == "mlb_paged_attention_mma"]
    assert not plan[9] and len(decoded) == 1 and bool(decoded[0]["mode"] & 16) == rings
