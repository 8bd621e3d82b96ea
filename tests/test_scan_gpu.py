"""The recurrences' scan kernel with one and with two columns a lane (scan_per_lane in csrc/delta_rule.cu), and the convolution whose one token a
sequence moves the state on itself: what a row's bits are depends on neither."""
import pytest
import torch

DEV = "cuda"


def step(counts, pos0):
    from microllm_rocm_b200.parts.base import StepContext
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    on = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    A, T = len(counts), starts[-1]
    ctx = StepContext(num_tokens=T, num_seqs=A, token_ids=on([0] * T), positions=on([p + i for n, p in zip(counts, pos0) for i in range(n)]),
                      token_seq=on([a for a, n in enumerate(counts) for _ in range(n)]), seq_starts=on(starts), seq_pos0=on(pos0),
                      seq_lens=on([n + p for n, p in zip(counts, pos0)]), block_tables={}, state_slots=on(list(range(A))), logit_rows=None,
                      error_flag=torch.zeros(1, dtype=torch.int32, device=DEV), seq_starts_host=starts, seq_pos0_host=list(pos0),
                      max_new_tokens=max(counts), max_seq_len=max(n + p for n, p in zip(counts, pos0)))
    return ctx, ctx.state_slots


@pytest.mark.gpu
@pytest.mark.parametrize("dk, dv", [(128, 128), (96, 52), (64, 64), (30, 37), (200, 40)])
@pytest.mark.parametrize("rule", ["delta", "decayed_sum", "bonus_read", "head", "head and vector"])
def test_many_sequences_have_the_bits_of_each_alone(rule, dk, dv):
    """Sequences together fill the device and take two columns a lane, one alone takes one; portions of one token, of part of a staged chunk and
    of several, some from a state and some from zero."""
    from microllm_rocm_b200.kernels import recurrent
    H, counts, pos0 = 16, [1, 3, 8, 37, 64, 5, 17, 2, 9, 33], [4, 0, 7, 0, 12, 1, 0, 3, 0, 2]
    A, T = len(counts), sum(counts)
    g = torch.Generator(DEV).manual_seed(dk)
    f = lambda *s: torch.randn(*s, generator=g, device=DEV)
    q, k, v = f(T, H * dk) * dk ** -0.5, torch.nn.functional.normalize(f(T, H, dk), dim=-1).reshape(T, -1), f(T, H * dv)
    decay, head_decay = torch.rand(T, H * dk, generator=g, device=DEV) * 0.3 + 0.7, torch.rand(T, H, generator=g, device=DEV) * 0.2 + 0.8
    beta, bonus, start, vector = torch.rand(T, H, generator=g, device=DEV), f(H, dk), f(A + 1, H, dk, dv), f(A + 1, H, dk)

    def run(which):
        starts = torch.cumsum(torch.tensor([0] + counts), 0).tolist()
        rows = torch.cat([torch.arange(starts[a], starts[a + 1]) for a in which]).to(DEV)
        ctx, slots = step([counts[a] for a in which], [pos0[a] for a in which])
        cut = lambda t: t[rows].contiguous()
        keep = torch.tensor(which, device=DEV)
        state, n_state = torch.cat([start[keep], start[-1:]]).contiguous(), torch.cat([vector[keep], vector[-1:]]).contiguous()
        o, den = torch.empty(len(rows), H * dv, device=DEV), torch.zeros(len(rows), H, device=DEV)
        if rule == "delta":
            recurrent.delta_scan(cut(q), cut(k), cut(decay), cut(beta), cut(v), o, state, slots, ctx, H, H, dk, dv)
        elif rule.startswith("head"):
            beside = dict(n_state=n_state, den=den) if rule != "head" else {}
            recurrent.head_scan(cut(q), cut(k), cut(head_decay), cut(v), o, state, slots, ctx, H, dk, dv, weight=cut(beta), **beside)
        else:
            recurrent.linear_scan(rule, cut(q), cut(k), cut(decay), cut(v), o, state, slots, ctx, H, dk, dv, bonus=bonus if rule == "bonus_read" else None)
        assert int(ctx.error_flag.item()) == 0
        return o, state[:len(which)], n_state[:len(which)], den

    together = run(list(range(A)))
    at = 0
    for a in range(A):
        o, state, n_state, den = run([a])
        assert torch.equal(together[0][at:at + counts[a]], o) and torch.equal(together[1][a], state[0])
        assert torch.equal(together[2][a], n_state[0]) and torch.equal(together[3][at:at + counts[a]], den)
        at += counts[a]


@pytest.mark.gpu
@pytest.mark.parametrize("taps, C", [(2, 12), (3, 260), (4, 1024), (5, 8), (4, 37), (7, 20)])
@pytest.mark.parametrize("partials", [1, 6])
def test_one_token_a_sequence_moves_the_state_on(taps, C, partials):
    """Steps of one token a sequence, and the same tokens in one portion: the same bits and the same state behind them."""
    from microllm_rocm_b200.kernels import recurrent
    A, n = 5, 9
    g = torch.Generator(DEV).manual_seed(C)
    u = torch.randn(partials, A, n, C + 8, generator=g, device=DEV)
    w, bias = torch.randn(C, taps, generator=g, device=DEV), torch.randn(C, generator=g, device=DEV)
    held = torch.randn(A + 1, taps - 1, C, generator=g, device=DEV)
    pos0 = [0, 1, 2, 5, 40]
    one, whole = held.clone(), held.clone()
    ctx, slots = step([n] * A, pos0)
    want = torch.empty(A * n, C, device=DEV)
    recurrent.short_conv(u.reshape(partials, A * n, C + 8), 4, w, whole, slots, ctx, want, silu=True, bias=bias)
    for t in range(n):
        ctx, slots = step([1] * A, [p + t for p in pos0])
        got = torch.empty(A, C, device=DEV)
        recurrent.short_conv(u[:, :, t].contiguous(), 4, w, one, slots, ctx, got, silu=True, bias=bias)
        assert torch.equal(got, want.view(A, n, C)[:, t]) and int(ctx.error_flag.item()) == 0, t
    assert torch.equal(one, whole)


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[2, 0], [0, 2], [3, 0, 0], [0, 1, 2], [1, 0, 1]])
@pytest.mark.parametrize("C", [12, 37])
def test_sequences_without_tokens_beside_others(counts, C):
    """As many tokens as sequences, but not one each: outputs and states of a step that does not name the empty ones, whose states stay."""
    from microllm_rocm_b200.kernels import recurrent
    taps, pos0 = 4, [5, 1, 40][:len(counts)]
    g = torch.Generator(DEV).manual_seed(C)
    u, w = torch.randn(sum(counts), C + 8, generator=g, device=DEV), torch.randn(C, taps, generator=g, device=DEV)
    held = torch.randn(len(counts) + 1, taps - 1, C, generator=g, device=DEV)

    def run(which):
        state, out = held.clone(), torch.empty(sum(counts), C, device=DEV)
        ctx, _ = step([counts[a] for a in which], [pos0[a] for a in which])
        recurrent.short_conv(u, 4, w, state, torch.tensor(which, dtype=torch.int32, device=DEV), ctx, out, silu=True)
        assert int(ctx.error_flag.item()) == 0
        return out, state
    got, want = run(list(range(len(counts)))), run([a for a, n in enumerate(counts) if n])
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("family, dtype", [("matidra", "float32"), ("matidra", "bfloat16"), ("naburax", "float32"), ("lozepel", "bfloat16"), ("fonuvik", "bfloat16")])
def test_branches_side_by_side_have_the_bits_of_one_after_another(family, dtype):
    """A prompt, a step that decodes beside a prompt portion, and decoded tokens."""
    from microllm_rocm_b200.config import find_preset
    from microllm_rocm_b200.engine.loading import make_engine, prepare_kernels, require_gpu, resolve_dtype
    from microllm_rocm_b200.engine.step import StepEntry
    from microllm_rocm_b200.parts import parallel
    from microllm_rocm_b200.parts.base import Runtime
    from microllm_rocm_b200.parts.build import build_model
    arch, cfg = find_preset(family + "-tiny")
    results = []
    for side in (False, True):
        parallel.SIDE_BY_SIDE = side
        try:
            model = build_model(arch.build_spec(cfg), Runtime(require_gpu(), resolve_dtype(dtype)))
            prepare_kernels(model)
            g = torch.Generator(DEV).manual_seed(1)
            made = {}
            for name, spec in model.expected_tensors().items():
                t = torch.randn(tuple(spec.shape), generator=g, device=DEV) * 0.1 + (1.0 if "norm" in name else 0.0)
                made[name] = t if spec.role == "vector" else t.to(resolve_dtype(dtype))
            model.bind(made)
            engine = make_engine(model, 16, 32, 4)
            out = []
            for rid in "ab":
                engine.cache.add(rid)
            out.append(engine.step([StepEntry("a", list(range(5, 50)), [44])]).clone())
            out.append(engine.step([StepEntry("a", [9], [0]), StepEntry("b", list(range(40, 60)), [19])]).clone())
            for t in range(3):
                out.append(engine.step([StepEntry("a", [t], [0]), StepEntry("b", [t + 7], [0])]).clone())
            engine.check_device_errors()
            results.append(torch.cat(out))
        finally:
            parallel.SIDE_BY_SIDE = True
    assert torch.equal(results[0], results[1]) and bool(torch.isfinite(results[0]).all())


@pytest.mark.gpu
def test_library_products_on_the_second_streams_of_two_threads():
    """Long sums into few columns, which the library splits and meets in its workspace: two threads at once get the bits of one after another."""
    import threading

    from microllm_rocm_b200.kernels import gemm_bf16, ops
    g = torch.Generator(DEV).manual_seed(3)
    shapes = [(300, 256, 8192), (300, 384, 6144), (520, 128, 8192)]
    pairs = [[(torch.randn(M, K, generator=g, device=DEV).bfloat16(), torch.randn(N, K, generator=g, device=DEV).bfloat16()) for M, N, K in shapes] for _ in range(2)]
    want = [[gemm_bf16.library_linear(x, w, None, torch.float32, None) for x, w in own] for own in pairs]
    torch.cuda.synchronize()
    got, failures, barrier = [[], []], [], threading.Barrier(2)

    def work(i):
        try:
            kept = {}
            outs = [[torch.empty(x.shape[0], w.shape[0], device=DEV) for x, w in pairs[i]] for _ in range(20)]
            barrier.wait(timeout=60)
            with ops.on_side_stream(lambda size: kept.setdefault(size, torch.empty(size, dtype=torch.uint8, device=DEV))) as side:
                for row in outs:
                    for (x, w), out in zip(pairs[i], row):
                        gemm_bf16.library_linear(x, w, None, torch.float32, out)
            ops.join(side)
            torch.cuda.synchronize()
            got[i] = outs
            assert len(kept) == 1
        except BaseException as e:                        # noqa: BLE001  (reported by the test's thread)
            failures.append(repr(e))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
    for i in range(2):
        for row in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(row, want[i]))


@pytest.mark.gpu
@pytest.mark.parametrize("preset, prompt, requests", [("matidra-tiny", 40, 3), ("lozepel-tiny", 40, 2), ("matidra-3b-layers", 700, 2), ("lozepel-3b-layers", 300, 1)])
def test_branches_side_by_side_in_prompts_of_library_products_and_in_captured_steps(preset, prompt, requests):
    """Logits of a prompt (of hundreds of tokens: products of the library on both streams), then of captured steps, against one branch after the other."""
    from microllm_rocm_b200.config import find_preset
    from microllm_rocm_b200.engine.decode_graph import DecodeGraphPool
    from microllm_rocm_b200.engine.loading import random_engine
    from microllm_rocm_b200.engine.step import StepEntry
    from microllm_rocm_b200.kernels.build import LaunchCounter
    from microllm_rocm_b200.parts import parallel
    from microllm_rocm_b200.sampling import GenerationConfig
    results, products = [], 0
    for side in (False, True):
        parallel.SIDE_BY_SIDE = side
        try:
            engine = random_engine(find_preset(preset)[1], seed=5, dtype="bfloat16", max_tokens=2048, max_requests=requests, draw_on_device=True)
            ids = [f"{i}" for i in range(requests)]
            for rid in ids:
                engine.cache.add(rid)
            before = LaunchCounter.library
            out = [engine.step([StepEntry(rid, [(7 * i + 3 * t) % 250 for t in range(prompt - i)], [prompt - i - 1]) for i, rid in enumerate(ids)]).clone()]
            products = LaunchCounter.library - before
            for rid in ids:
                assert engine.cache.reserve(rid, prompt + 8)
            graph, kept = DecodeGraphPool(engine).get(ids, headroom_tokens=8), {}
            graph.ctx.tensor_sink = lambda name, t: kept.__setitem__(name, t) if name == "logits" else None
            load = lambda: graph.load(ids, [3] * requests, [prompt - i for i in range(requests)], [GenerationConfig(max_new_tokens=8, temperature=0.0)] * requests, [0] * requests)
            load()
            graph.capture()
            load()
            for _ in range(4):
                graph.replay()
                out.append(kept["logits"][:requests].clone())
                out.append(torch.tensor(graph.read_tokens(), device=DEV))
            engine.check_device_errors()
            results.append(out)
        finally:
            parallel.SIDE_BY_SIDE = True
    assert products > 0 or prompt < 300
    for a, b in zip(*results):
        assert torch.equal(a, b) and bool(torch.isfinite(a.float()).all())
