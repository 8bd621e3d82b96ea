"""The Gedalix decoder on the GPU against its plain float64 restatement: each mechanism alone, then whole models cut
in every way (whole prompts, a tail decoded token by token, portions down to two tokens, mixed batches over a pool
so small that pages and slots are used again), in true fp32 and in bf16, and greedy generation through the
scheduler."""
import math

import pytest
import torch

from tests.gedalix_cases import CASES, random_weights, raw_config, write_folder
from tests.helpers import collect, random_tokens, steps_mixed, steps_portions, steps_prefill_then_decode, steps_whole
from tests.plain import gedalix_plain as plain

pytestmark = pytest.mark.gpu

FP32_TOL = 2e-5          # of the largest |logit| (measured worst: 2e-6)
BF16_TOL = 0.03          # of the largest |logit| (measured worst: 0.012)
DEV = "cuda:0"


def tol(dtype):
    return FP32_TOL if dtype == "float32" else BF16_TOL


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    out = {}
    for key in CASES:
        raw = raw_config(key)
        weights = random_weights(raw, seed=len(key) + ord(key[0]))
        out[key] = (write_folder(str(tmp_path_factory.mktemp("gedalix_" + key)), raw, weights), raw, weights)
    return out


def engine_for(folder, dtype, max_tokens=1024, page_size=16, max_requests=4):
    from microllm_rocm_b200.engine.loading import load_engine
    return load_engine(folder, dtype=dtype, page_size=page_size, max_tokens=max_tokens, max_requests=max_requests)


_plain = {}


def plain_logits(key, raw, weights, tokens):
    k = (key, id(weights), tuple(tokens))
    if k not in _plain:
        _plain[k] = plain.forward(raw, weights, list(tokens)).float()
    return _plain[k]


def compare(got, key, raw, weights, requests, dtype):
    worst = 0.0
    for rid, toks in requests.items():
        ref = plain_logits(key, raw, weights, toks)
        rows = torch.stack([got[(rid, p)] for p in range(len(toks))])
        err = (rows - ref).abs().amax(dim=1) / ref.abs().max()
        assert torch.isfinite(rows).all(), f"case {key} request {rid}: logits that are not finite"
        over = err > tol(dtype)
        # bf16 rounds the router's input: where two experts' logits are a rounding error apart the choice may flip, and
        # that position (it alone) lands far off.  Such positions are rare; fp32 allows none.
        allowed = 0 if dtype == "float32" else max(1, len(toks) // 25)
        if int(over.sum()) > allowed:
            pos = int(over.nonzero()[0])
            raise AssertionError(f"case {key} request {rid}: {int(over.sum())} positions over the tolerance {tol(dtype)} ({allowed} allowed), "
                                 f"the first is {pos} of {len(toks)} (error {float(err[pos]):.3e} of the largest |logit|)")
        err = err[~over] if (~over).any() else err
        worst = max(worst, float(err.max()))
    print(f"[gedalix parity] case {key} {dtype}: worst error {worst:.3e} of the largest |logit|")
    return worst


def requests_for(raw, lengths, seed=0):
    return {f"r{i}": random_tokens(n, raw["vocab"], seed + 100 * i + n) for i, n in enumerate(lengths)}


# ------------------------------------------------------------------------------------------- mechanisms alone
@pytest.mark.parametrize("table_dtype", [torch.float32, torch.bfloat16])
def test_scaled_embedding_and_learned_positions(table_dtype):
    from microllm_rocm_b200.kernels import ops
    torch.manual_seed(1)
    table = torch.randn(50, 24, device=DEV).to(table_dtype)
    pos_table = torch.randn(40, 24, device=DEV).to(table_dtype)
    ids = torch.tensor([3, 49, 0, 7, 7], dtype=torch.int32, device=DEV)
    positions = torch.tensor([0, 39, 5, 6, 1], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 24, device=DEV)
    ops.embed_gather_scaled(table, ids, out, 2.5)
    ops.add_table_rows(out, pos_table, positions)
    want = table.float()[ids.long()] * 2.5 + pos_table.float()[positions.long()]
    assert torch.allclose(out, want, atol=1e-6)


def test_scaled_add_norm_and_pass_entry():
    from microllm_rocm_b200.kernels import ops
    torch.manual_seed(2)
    x = torch.randn(7, 40, device=DEV)
    delta = torch.randn(3, 7, 40, device=DEV)                 # three partial sums
    scale, w, v = torch.randn(40, device=DEV), torch.randn(40, device=DEV), torch.randn(40, device=DEV)
    x0 = torch.randn(7, 40, device=DEV)
    want_x = x.double() + scale.double() * delta.double().sum(0)
    want = plain.rms(want_x, 1e-4) * w.double()
    res, out = x.clone(), torch.empty(7, 40, device=DEV)
    ops.add_scaled_rmsnorm(res, delta, scale, w, 1e-4, out)
    assert torch.allclose(res.double(), want_x, atol=1e-5) and torch.allclose(out.double(), want, atol=1e-5)
    res2 = x.clone()
    ops.add_scaled_inplace(res2, delta[0], scale)
    assert torch.allclose(res2, x + scale * delta[0], atol=1e-6)
    a, b = x.clone(), x.clone()
    ops.stream_entry(a, None, v)
    ops.stream_entry(b, x0, v)
    assert torch.allclose(a, x + v, atol=1e-6) and torch.allclose(b, x + x0 + v, atol=1e-6)


@pytest.mark.parametrize("experts, top", [(5, 2), (7, 1), (4, 4), (40, 6)])
def test_router_choice_weights_and_sorted_pairs(experts, top):
    from microllm_rocm_b200.kernels import moe
    torch.manual_seed(experts)
    T, W = 37, 48
    x, wr, b, sg = torch.randn(T, W, device=DEV), torch.randn(experts, W, device=DEV), torch.randn(experts, device=DEV), torch.randn(1, W, device=DEV)
    ids = torch.empty(T, top, dtype=torch.int32, device=DEV)
    weights, gate = torch.empty(T, top, device=DEV), torch.empty(T, device=DEV)
    both = torch.cat([wr, sg, torch.zeros(2, W, device=DEV)])            # router rows, the gate's row, padding
    logits = torch.stack([x[:, :20] @ both[:, :20].T, x[:, 20:] @ both[:, 20:].T])     # two partial sums of a split product
    moe.select(logits, experts, b, top, ids, weights, experts, gate)
    z = x.double() @ wr.double().T + b.double()
    chosen = torch.topk(z, top, dim=-1)
    assert torch.equal(ids.long().cpu(), chosen.indices.cpu())
    assert torch.allclose(weights.double(), torch.softmax(chosen.values, -1), atol=1e-5)
    assert torch.allclose(weights.sum(-1), torch.ones(T, device=DEV), atol=1e-6)
    assert torch.allclose(gate.double(), torch.sigmoid(x.double() @ sg.double().T)[:, 0], atol=1e-5)
    offsets = torch.empty(experts + 1, dtype=torch.int32, device=DEV)
    order = torch.empty(T * top, dtype=torch.int32, device=DEV)
    moe.align(ids, experts, offsets, order)
    offsets, order, flat = offsets.cpu().tolist(), order.cpu().tolist(), ids.cpu().reshape(-1).tolist()
    assert offsets[0] == 0 and offsets[-1] == T * top and sorted(order) == list(range(T * top))
    for e in range(experts):
        assert all(flat[pair] == e for pair in order[offsets[e]:offsets[e + 1]])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows, row_tile", [(5, 16), (100, 64), (100, 16)])
def test_grouped_product_over_sorted_rows_and_per_head(dtype, rows, row_tile):
    from microllm_rocm_b200.kernels import grouped
    torch.manual_seed(rows)
    G, N, K, top = 3, 21, 36, 2
    atol = 1e-4 if dtype == torch.float32 else 0.06
    w = torch.randn(G, N, K, device=DEV).to(dtype)
    # (a) rows sorted by group, read through a list of (token, choice) pairs, written back to the pairs' own rows
    a = torch.randn(rows, K, device=DEV).to(dtype)
    group_of_pair = torch.randint(0, G, (rows * top,))
    order = torch.argsort(group_of_pair, stable=True).to(torch.int32)
    counts = torch.bincount(group_of_pair, minlength=G)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]).to(torch.int32)
    out = torch.zeros(rows * top, N, device=DEV)
    grouped.grouped_linear(a, w, out, rows=rows * top, group_offsets=offsets.to(DEV), a_rows=order.to(DEV), c_rows=order.to(DEV),
                           a_row_div=top, row_tile=row_tile)
    want = torch.stack([a.double()[pair // top] @ w.double()[group_of_pair[pair]].T for pair in range(rows * top)])
    assert torch.allclose(out.double(), want, atol=atol)
    # (b) one product per head over all rows, column blocks of the input and the output, a factor on the result
    a2 = torch.randn(rows, G * K + 5, device=DEV).to(dtype)
    out2 = torch.zeros(rows, G * (N + 2), device=DEV).to(dtype)
    factor = torch.rand(rows, G * (N + 2), device=DEV)
    grouped.grouped_linear(a2, w, out2, rows=rows, a_group_cols=K, c_group_cols=N + 2, factor=factor, row_tile=row_tile)
    for g in range(G):
        want2 = (a2.double()[:, g * K:(g + 1) * K] @ w.double()[g].T) * factor.double()[:, g * (N + 2):g * (N + 2) + N]
        assert torch.allclose(out2.double()[:, g * (N + 2):g * (N + 2) + N], want2, atol=atol)
        assert (out2[:, g * (N + 2) + N:(g + 1) * (N + 2)] == 0).all()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("key", ["a", "b"])
def test_every_run_of_the_layers_against_the_plain_residual_stream(folders, key, dtype):
    """The residual stream after every run (a looped layer counts each time): mixer, feed-forward, scales, pass entries."""
    from microllm_rocm_b200.engine.step import StepEntry
    folder, raw, weights = folders[key]
    tokens = random_tokens(45, raw["vocab"], 5)
    want = []
    plain.forward(raw, weights, tokens, collect=want)
    engine = engine_for(folder, dtype)
    got = {}
    engine.cache.add("x")
    engine.step([StepEntry("x", tokens, [0])], tensor_sink=lambda name, t: got.__setitem__(name, None if t is None else t.detach().clone()))
    engine.check_device_errors()
    runs = [n for n in got if n.endswith(".residual")]
    assert len(runs) == len(want)
    for name, ref in zip(runs, want):
        x = got[name].double()
        delta = got[name.replace(".residual", ".delta")]
        if delta is not None:
            x = x + (delta.double() if delta.dim() == 2 else delta.double().sum(0))
        err = float((x.cpu() - ref).abs().max() / ref.abs().max())
        assert err < (1e-5 if dtype == "float32" else 0.02), f"{name}: {err}"


@pytest.mark.parametrize("rows, row_tile", [(3, 16), (70, 16), (200, 64), (700, 128)])
def test_tensor_core_grouped_product_equals_the_plain_one(rows, row_tile):
    """bf16 operands on mma.sync against float64, sorted rows and per-head column blocks, K with a ragged last tile,
    the gate-times-up epilogue."""
    from microllm_rocm_b200.kernels import grouped
    torch.manual_seed(rows)
    G, N, K, top = 5, 72, 104, 2
    w = (torch.randn(G, N, K, device=DEV) * K ** -0.5).bfloat16()
    a = torch.randn(rows, K, device=DEV).bfloat16()
    assert grouped.mma_supported(a, w)
    group_of_pair = torch.randint(0, G, (rows * top,))
    group_of_pair[group_of_pair == 3] = 4                       # a group without rows
    order = torch.argsort(group_of_pair, stable=True).to(torch.int32).to(DEV)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(group_of_pair, minlength=G).cumsum(0)]).to(torch.int32).to(DEV)
    out = torch.zeros(rows * top, N, device=DEV)
    grouped.grouped_linear(a, w, out, rows=rows * top, group_offsets=offsets, a_rows=order, c_rows=order, a_row_div=top, row_tile=row_tile)
    want = torch.stack([a.double()[pair // top] @ w.double()[group_of_pair[pair]].T for pair in range(rows * top)])
    assert torch.allclose(out.double(), want, atol=2e-3)
    # gate rows over up rows, silu(gate) * up as the epilogue; the output is in sorted order
    w2 = (torch.randn(G, 2 * 40, K, device=DEV) * K ** -0.5).bfloat16()
    act = torch.zeros(rows * top, 40, device=DEV, dtype=torch.bfloat16)
    grouped.grouped_silu_mul(a, w2, act, rows=rows * top, group_offsets=offsets, a_rows=order, a_row_div=top, row_tile=row_tile)
    for place, pair in enumerate(order.cpu().tolist()):
        gu = a.double()[pair // top] @ w2.double()[group_of_pair[pair]].T
        assert torch.allclose(act[place].double(), gu[:40] * torch.sigmoid(gu[:40]) * gu[40:], atol=0.02)
    # per head over all rows, with a factor
    a2 = torch.randn(rows, G * K, device=DEV).bfloat16()
    out2 = torch.zeros(rows, G * N, device=DEV, dtype=torch.bfloat16)
    factor = torch.rand(rows, G * N, device=DEV)
    grouped.grouped_linear(a2, w, out2, rows=rows, a_group_cols=K, c_group_cols=N, factor=factor, row_tile=row_tile)
    want2 = torch.cat([a2.double()[:, g * K:(g + 1) * K] @ w.double()[g].T for g in range(G)], 1) * factor.double()
    assert torch.allclose(out2.double(), want2, atol=0.03)


# ------------------------------------------------------------------------------------------- whole models, every cut
LENGTHS = {"a": [1, 2, 17, 70, 133], "b": [3, 9, 40, 65, 150], "c": [31, 129], "d": [5, 64, 97], "e": [2, 33, 140]}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("key", sorted(CASES))
@pytest.mark.parametrize("cut", ["whole", "tail", "portions"])
def test_one_request_at_a_time(folders, key, dtype, cut):
    folder, raw, weights = folders[key]
    reqs = requests_for(raw, LENGTHS[key])
    steps = {"whole": steps_whole, "tail": steps_prefill_then_decode, "portions": steps_portions}[cut](reqs)
    got = collect(engine_for(folder, dtype), steps)
    compare(got, key, raw, weights, reqs, dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("key", ["a", "b"])
def test_mixed_batches_over_a_tight_pool(folders, key, dtype):
    """Up to four live requests, portions beside single tokens, some left out of a step; the pool holds just the peak,
    so pages go from one request to the next; every position must equal what the request gives alone."""
    folder, raw, weights = folders[key]
    reqs = requests_for(raw, [60, 33, 150, 90, 47, 128, 75, 20, 101, 64], seed=9)
    steps, peak = steps_mixed(reqs, max_live=4, seed=3)
    engine = engine_for(folder, dtype, max_tokens=peak, max_requests=4)
    got = collect(engine, steps)
    compare(got, key, raw, weights, reqs, dtype)
    pool = engine.cache.groups["full"].pool
    assert pool.total_allocations > pool.num_pages, "the pool was never tight enough to use a page again"


@pytest.mark.parametrize("key", ["c", "d"])
def test_tensor_core_attention_and_products_track_the_plain_kernels(folders, key):
    """bf16, the same schedule twice: on the tensor-core kernels (attention with key splits in the decoded tail, grouped
    products) and on the plain ones.  Tiles of 16 (token, head) rows span several tokens here (two and four heads)."""
    from microllm_rocm_b200.kernels import grouped, latent
    folder, raw, weights = folders[key]
    assert latent.mma_supported(raw["layers"][0]["mixer"]["kv_rank"], raw["layers"][0]["mixer"]["rot_dim"])
    reqs = requests_for(raw, [3, 50, 290], seed=2)
    steps, peak = steps_mixed(reqs, max_live=3, seed=5, decode_tail=20)
    fast = collect(engine_for(folder, "bfloat16", max_tokens=peak), steps)
    latent.USE_TENSOR_CORES = grouped.USE_TENSOR_CORES = False
    try:
        slow = collect(engine_for(folder, "bfloat16", max_tokens=peak), steps)
    finally:
        latent.USE_TENSOR_CORES = grouped.USE_TENSOR_CORES = True
    compare(fast, key, raw, weights, reqs, "bfloat16")
    compare(slow, key, raw, weights, reqs, "bfloat16")
    far = [k for k in fast if float((fast[k] - slow[k]).abs().max()) > 0.03 * float(slow[k].abs().max())]
    assert len(far) <= len(fast) // 25, f"{len(far)} of {len(fast)} positions differ between the kernels"


def test_fp32_does_not_depend_on_cuts_batches_or_pages(folders):
    folder, raw, weights = folders["a"]
    reqs = requests_for(raw, [70, 133, 20, 45], seed=4)
    whole = collect(engine_for(folder, "float32"), steps_whole(reqs))
    portions = collect(engine_for(folder, "float32", page_size=8), steps_portions(reqs, sizes=(2, 9, 2, 30, 1, 5)))
    steps, peak = steps_mixed(reqs, max_live=3, seed=1)
    mixed = collect(engine_for(folder, "float32", max_tokens=peak), steps)
    for k in whole:
        assert torch.equal(whole[k], portions[k]) and torch.equal(whole[k], mixed[k]), f"{k} differs between schedules"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_far_keys_page_borders_and_the_sink_decide_the_output(tmp_path_factory, dtype):
    """Peaky attention (queries scaled up): single keys, far back and at page borders, carry a position's output, in a
    prompt of several hundred tokens and in the tokens decoded after it; large sinks take most of the weight elsewhere.
    A key lost at a page's edge, a sink left out or scaled, or a position off by one would show at once."""
    raw = raw_config("c")
    for name, sharp, sink in (("sharp", 5.0, 1.0), ("sinks", 2.0, 4.0)):
        weights = random_weights(raw, seed=11, sharp=sharp, sink=sink)
        folder = write_folder(str(tmp_path_factory.mktemp("gedalix_" + name)), raw, weights)
        reqs = {"long": random_tokens(700, raw["vocab"], 21), "edge": random_tokens(16 * 9 + 1, raw["vocab"], 22)}
        for page_size, steps in ((16, steps_prefill_then_decode(reqs, tail=40)), (32, steps_portions(reqs, sizes=(127, 2, 33, 1, 64, 300)))):
            got = collect(engine_for(folder, dtype, max_tokens=1100, page_size=page_size), steps)
            compare(got, "c-" + name, raw, weights, reqs, dtype)
    # the attention really is peaky: dropping the sinks changes the sharp model's logits by far more than the tolerance
    no_sink = {k: (torch.full_like(v, -30.0) if k.endswith("mix.sink") else v) for k, v in weights.items()}
    a = plain.forward(raw, weights, reqs["edge"][:40])
    b = plain.forward(raw, no_sink, reqs["edge"][:40])
    assert float((a - b).abs().max() / a.abs().max()) > 10 * BF16_TOL


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_mixer_with_a_window_of_keys(dtype):
    """Latent attention takes a window as a parameter (no Gedalix configuration sets one): a model description with
    windows of 40 and 33 keys on its two layers, built from the same parts.  The cache manager gives pages behind a
    window back while the request lives; keys just inside and just outside the window, in prompt portions and in decoded
    tokens, at page borders (pages of 8 and 16), against the plain implementation with the same window."""
    import dataclasses

    from microllm_rocm_b200.config import GedalixConfig, get_architecture
    from microllm_rocm_b200.config.spec import PartSpec
    from microllm_rocm_b200.engine.loading import make_engine, prepare_kernels
    from microllm_rocm_b200.parts.base import Runtime
    from microllm_rocm_b200.parts.build import build_model
    from microllm_rocm_b200.weights.loader import target_dtype
    raw = raw_config("d")
    weights = random_weights(raw, seed=31, sharp=4.0)
    windows = [40, 33]
    spec = get_architecture("Gedalix").build_spec(GedalixConfig.from_dict(raw))
    layers = [dataclasses.replace(layer, mixer=PartSpec(layer.mixer.kind, {**layer.mixer.params, "window": w}))
              for layer, w in zip(spec.layers, windows)]
    spec = dataclasses.replace(spec, layers=layers)
    plain_raw = raw_config("d")
    for layer, w in zip(plain_raw["layers"], windows):
        layer["mixer"]["window"] = w
    reqs = {"w0": random_tokens(150, raw["vocab"], 41), "w1": random_tokens(77, raw["vocab"], 42)}
    rt = Runtime(torch.device(DEV), torch.float32 if dtype == "float32" else torch.bfloat16)
    for page_size, steps in ((8, steps_prefill_then_decode(reqs, tail=60)), (16, steps_portions(reqs, sizes=(39, 2, 41, 1, 33, 7)))):
        model = build_model(spec, rt)
        prepare_kernels(model)
        model.bind({n: weights[n].to(device=DEV, dtype=target_dtype(ws.role, rt)).contiguous() for n, ws in model.expected_tensors().items()})
        engine = make_engine(model, page_size, 64, 4, max_step_tokens=160)
        assert set(engine.cache.groups) == {"window40", "window33"}
        got = collect(engine, steps)
        compare(got, "d-window", plain_raw, weights, reqs, dtype)
        assert engine.cache.pages_released_by_window > 0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_decoding_from_the_first_token(folders, dtype):
    """One token per step from position 0 on, over many pages."""
    folder, raw, weights = folders["d"]
    reqs = {"d": random_tokens(150, raw["vocab"], 8)}
    got = collect(engine_for(folder, dtype, page_size=8), steps_prefill_then_decode(reqs, tail=149))
    compare(got, "d", raw, weights, reqs, dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_greedy_generation_through_the_scheduler(folders, dtype):
    from microllm_rocm_b200.engine.llm import LLM
    from microllm_rocm_b200.sampling import GenerationConfig
    folder, raw, weights = folders["a"]
    prompts = [random_tokens(n, raw["vocab"], 50 + n) for n in (9, 40, 3)]
    llm = LLM(folder, dtype=dtype, page_size=16, max_tokens=512)
    outs = llm.generate(prompts, GenerationConfig(max_new_tokens=12, temperature=0.0))
    for prompt, got in zip(prompts, outs):
        assert len(got) == 12
        seq = list(prompt)
        for i, token in enumerate(got):
            ref = plain.forward(raw, weights, seq)[-1]
            if dtype == "float32":
                assert token == int(ref.argmax()), f"token {i} differs from the plain greedy choice"
            else:       # bf16 may leave the fp32 choice at a near tie: every pick must be a near maximum of the plain logits
                assert float(ref.max() - ref[token]) <= 0.05 * float(ref.abs().max())
            seq.append(token)


@pytest.mark.parametrize("top, width", [(1, 96), (2, 2048), (3, 100), (4, 1028), (6, 2048), (8, 64), (9, 64), (6, 70)])
@pytest.mark.parametrize("partials, gated, scaled", [(0, False, False), (1, True, True), (3, True, False)])
def test_the_experts_results_are_summed_over_tops_and_widths(top, width, partials, gated, scaled):
    """Four columns a thread (up to eight choices, widths that are multiples of four) and column by column (the others)."""
    from microllm_rocm_b200.kernels import moe
    torch.manual_seed(top * width)
    T = 9
    y, w = torch.randn(T * top, width, device=DEV), torch.rand(T, top, device=DEV)
    shared = torch.randn(max(1, partials), T, width, device=DEV)
    gate, scale = torch.rand(T, device=DEV), torch.rand(width, device=DEV)
    out = torch.empty(T, width, device=DEV)
    moe.combine(y, w, out, shared=(shared if partials > 1 else shared[0]) if partials else None, gate=gate if gated else None,
                col_scale=scale if scaled else None)
    want = (y.double().view(T, top, width) * w.double()[:, :, None]).sum(1)
    if partials:
        want = want + shared.double().sum(0) * (gate.double()[:, None] if gated else 1.0)
    if scaled:
        want = want * scale.double()
    # at most top + partials + 2 roundings of terms of a few units
    assert float((out.double() - want).abs().max()) < (top + partials + 2) * 2 ** -24 * 32


# ------------------------------------------------------------------------------------------- two streams in a step
def test_the_shared_expert_beside_the_router_changes_no_bits():
    """Steps of few tokens run the shared expert on the device's second stream: the same logits, step by step and in captured
    decode steps, as with everything on one."""
    import copy

    from microllm_rocm_b200.config.gedalix import PRESETS, GedalixConfig
    from microllm_rocm_b200.engine.decode_graph import DecodeGraphPool
    from microllm_rocm_b200.engine.loading import random_engine
    from microllm_rocm_b200.engine.step import StepEntry
    from microllm_rocm_b200.parts import routed
    from microllm_rocm_b200.sampling import GenerationConfig
    raw = copy.deepcopy(PRESETS["gedalix-small"])
    raw["layers"], raw["max_positions"] = raw["layers"][:3], 256
    config = GedalixConfig.from_dict(raw)
    greedy = GenerationConfig(max_new_tokens=30, temperature=0.0)

    def run(limit):
        kept, routed.SIDE_MAX_TOKENS = routed.SIDE_MAX_TOKENS, limit
        try:
            engine = random_engine(config, seed=3, max_tokens=1024, max_requests=16, draw_on_device=True)
            out = []
            for batch in (1, 8, 13):
                ids = [f"{batch}.{i}" for i in range(batch)]
                for rid in ids:
                    engine.cache.add(rid)
                out.append(engine.step([StepEntry(rid, [7 + i, 11, 13 * i], [2]) for i, rid in enumerate(ids)]).clone())
                out.append(engine.step([StepEntry(rid, [100 + i], [0]) for i, rid in enumerate(ids)]).clone())
                graph = DecodeGraphPool(engine).get(ids, headroom_tokens=30)
                logits = {}
                graph.ctx.tensor_sink = lambda name, t: logits.__setitem__(name, t)
                state = ([5] * batch, [4] * batch, [greedy] * batch, [0] * batch)
                for rid in ids:
                    engine.cache.reserve(rid, 30)
                graph.load(ids, *state)
                graph.capture()
                graph.load(ids, *state)
                for _ in range(20):
                    graph.replay()
                    out.append(logits["logits"][:batch].clone())
                    graph.read_tokens()
                for rid in ids:
                    engine.cache.release(rid)
            engine.check_device_errors()
            return out
        finally:
            routed.SIDE_MAX_TOKENS = kept

    one, two = run(0), run(32)
    assert all(torch.equal(a, b) for a, b in zip(one, two))


# ------------------------------------------------------------------------------- two groups of rows a CTA (latent_mma.cu)
def latent_step(seqs, heads, rank, rot, window, sink, seed=0, page_size=16):
    """A step's queries, cache and context.  seqs: (new tokens, tokens in front) each; the cache's pages are shuffled."""
    from microllm_rocm_b200.parts.base import StepContext
    g = torch.Generator().manual_seed(seed)
    width, T = rank + rot, sum(n for n, _ in seqs)
    q = (torch.randn(T, heads * width, generator=g) * 0.3).bfloat16().to(DEV)
    blocks = [-(-(n + p) // page_size) for n, p in seqs]
    order = torch.randperm(sum(blocks) + 3, generator=g)
    table = torch.full((len(seqs), max(blocks)), -1, dtype=torch.int32)
    at = 0
    for a, b in enumerate(blocks):
        table[a, :b] = order[at:at + b]
        at += b
    pages = torch.randn(sum(blocks) + 3, page_size, width, generator=g).bfloat16().to(DEV)
    starts = [0]
    for n, _ in seqs:
        starts.append(starts[-1] + n)
    on = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    positions = [p + i for n, p in seqs for i in range(n)]

    def context():
        return StepContext(num_tokens=T, num_seqs=len(seqs), token_ids=on(positions), positions=on(positions),
                           token_seq=on([a for a, (n, _) in enumerate(seqs) for _ in range(n)]), seq_starts=on(starts), seq_pos0=on([p for _, p in seqs]),
                           seq_lens=on([n + p for n, p in seqs]), block_tables={}, state_slots=None, logit_rows=None,
                           error_flag=torch.zeros(1, dtype=torch.int32, device=DEV), seq_starts_host=starts, seq_pos0_host=[p for _, p in seqs],
                           max_new_tokens=max(n for n, _ in seqs), max_seq_len=max(n + p for n, p in seqs))
    sinks = torch.randn(heads, generator=g).to(DEV) if sink else None

    def run(groups, pages=pages):
        from microllm_rocm_b200.kernels import latent
        ctx, out = context(), torch.full((T, heads * rank), float("nan"), dtype=torch.bfloat16, device=DEV)
        latent.GROUPS = groups
        try:
            latent.attention(q, pages, out, sinks, ctx, table.to(DEV), heads, rank, rot, width ** -0.5, window)
        finally:
            latent.GROUPS = None
        assert int(ctx.error_flag.item()) == 0
        run.groups = next(iter(ctx.extras.values()))[3]
        assert groups in (None, run.groups)
        return out

    def want():
        """In float64, with the largest value a row of the result may be made of."""
        out, most = torch.empty(T, heads, rank, dtype=torch.float64, device=DEV), torch.empty(T, 1, 1, dtype=torch.float64, device=DEV)
        for a, (n, p) in enumerate(seqs):
            keys = pages.double()[table[a, :blocks[a]].long().to(DEV)].reshape(-1, width)[:n + p]
            query = q.double()[starts[a]:starts[a + 1]].view(n, heads, width)
            scores = torch.einsum("nhw,kw->nhk", query, keys) * width ** -0.5
            i, k = torch.arange(p, p + n, device=DEV)[:, None], torch.arange(n + p, device=DEV)[None]
            seen = (k <= i) & (k > i - (window or 1 << 30))
            scores = scores.masked_fill(~seen[:, None, :], -math.inf)
            if sinks is not None:
                scores = torch.cat([scores, sinks.double()[None, :, None].expand(n, -1, 1)], -1)
            weights = torch.softmax(scores, -1)[..., :n + p]
            out[starts[a]:starts[a + 1]] = weights @ keys[:, :rank]
            most[starts[a]:starts[a + 1]] = keys[:, :rank].abs().max()
        return out.reshape(T, -1), most.reshape(T, 1)
    return run, want, pages, table


# new tokens and tokens in front: 31, 30, 32, 17, 1 and 16 rows in the last pair of groups, a second group without rows, later portions
GROUP_STEPS = {16: [(2, 0), (41, 0), (70, 33), (1, 5)], 5: [(19, 0), (38, 3), (13, 100), (3, 64), (45, 31)], 3: [(11, 7), (53, 0), (75, 40)],
               40: [(4, 0), (9, 60)], 31: [(1, 0), (33, 90)]}


@pytest.mark.parametrize("heads", sorted(GROUP_STEPS))
@pytest.mark.parametrize("window, sink, rank, rot", [(None, False, 256, 32), (None, True, 512, 64), (7, True, 256, 32), (40, False, 512, 64), (33, True, 256, 32)])
def test_two_groups_of_latent_rows_give_the_bits_of_one(heads, window, sink, rank, rot):
    """A row's bits do not follow which rows share its CTA; both against float64."""
    run, want, _, _ = latent_step(GROUP_STEPS[heads], heads, rank, rot, window, sink, seed=heads)
    one, two = run(1), run(2)
    assert torch.equal(one, two)
    ref, most = want()
    # weights are rounded to bf16 (and their sum is of the unrounded ones), the result too: half an ulp each, of the largest value
    # at most; fp32 sums besides
    assert bool(((one.double() - ref).abs() <= 2 ** -7.9 * most).all()), float(((one.double() - ref).abs() / most).max())


@pytest.mark.parametrize("window", [None, 20])
def test_keys_that_only_the_other_group_sees_do_not_reach_a_row(window):
    """Cache rows that are not finite: what a row does not see does not touch it.  16 heads, so that a group is one token's."""
    heads, rank, rot = 16, 256, 32
    seqs = [(64, 0), (37, 50)]
    run, _, pages, table = latent_step(seqs, heads, rank, rot, window, True)
    clean = run(2)
    for a, position in ((0, 1), (0, 32), (0, 63), (1, 51), (1, 86), (1, 31)):
        spoiled = pages.clone()
        spoiled[int(table[a, position // 16]), position % 16] = float("nan")
        one, two = run(1, spoiled), run(2, spoiled)
        assert torch.equal(one.view(torch.int16), two.view(torch.int16)), (a, position)
        start, (n, p) = (0, 64)[a], seqs[a]
        for i in range(n):
            sees = p + i >= position and (window is None or p + i - window < position)
            assert bool(torch.isnan(two[start + i].float()).any()) == sees, (a, position, i)
            if not sees:
                assert torch.equal(two[start + i], clean[start + i])


@pytest.mark.parametrize("seqs, groups", [([(760, 0), (33, 7)], 2), ([(300, 400), (330, 300)], 2), ([(300, 0), (200, 0)], 1)])
def test_a_step_of_many_latent_rows_holds_two_groups_a_cta(seqs, groups):
    """A long prompt, later portions behind many keys, and a step too small for it (148 SMs)."""
    run, _, _, _ = latent_step(seqs, 16, 256, 32, None, True)
    by_itself = run(None)
    assert run.groups == groups or torch.cuda.get_device_properties(0).multi_processor_count != 148
    assert torch.equal(by_itself, run(2)) and torch.equal(run(1), run(2))



# ---------------------------------------------------------------------- rows in registers, and partial results asked for together
@pytest.mark.parametrize("width", [1, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 3000])
@pytest.mark.parametrize("partials, scaled, out_dtype", [(1, True, torch.float32), (2, False, torch.bfloat16), (3, True, torch.bfloat16),
                                                         (4, True, torch.float32), (5, False, torch.float32), (8, True, torch.float32)])
def test_scaled_add_norm_over_widths_and_partial_results(width, partials, scaled, out_dtype):
    """Four columns a thread, eight, and any number; whole and partial rounds of three further partial results."""
    from microllm_rocm_b200.kernels import ops
    torch.manual_seed(width * 10 + partials)
    rows, eps = 5, 1e-5
    x, delta = torch.randn(rows, width, device=DEV), torch.randn(partials, rows, width, device=DEV)
    scale = torch.randn(width, device=DEV) if scaled else None
    weight = torch.randn(width, device=DEV)
    d = delta[0].clone()                                  # the order of additions: one partial result after the other
    for k in range(1, partials):
        d += delta[k]
    want_x = x.double() + d.double() * (scale.double() if scaled else 1.0)
    res, out = x.clone(), torch.empty(rows, width, dtype=out_dtype, device=DEV)
    ops.add_scaled_rmsnorm(res, delta if partials > 1 else delta[0], scale, weight, eps, out)
    # fp32 sums in that order are exact here; then one fused multiply-add: half an ulp of the result
    assert bool(((res.double() - want_x).abs() <= 2 ** -24 * want_x.abs() * 1.0001 + 1e-38).all())
    want = plain.rms(res.double(), eps) * weight.double()
    # the sum of squares (a few dozen additions a thread and across threads), root, quotient and two products: well within 16 ulps
    rel = 2 ** -8 if out_dtype == torch.bfloat16 else 16 * 2 ** -24
    assert bool(((out.double() - want).abs() <= rel * want.abs() + 1e-30).all()), float(((out.double() - want).abs() / want.abs()).max())


@pytest.mark.parametrize("experts", [1, 31, 32, 127, 128, 129, 200, 256])
@pytest.mark.parametrize("partials, gated", [(1, True), (1, False), (4, True), (5, True), (6, False)])
def test_router_choice_over_numbers_of_experts_and_partial_results(experts, partials, gated):
    """The gate's column travels with the logits, four columns a lane and four partial results at a time: on both sides of a lane's
    and of a round's end."""
    from microllm_rocm_b200.kernels import moe
    torch.manual_seed(experts + partials)
    T, top = 7, min(6, experts)
    gate_col = experts + 2 if gated else -1               # (with padding in front of it)
    logits = torch.randn(partials, T, experts + 5, device=DEV)
    bias = torch.randn(experts, device=DEV)
    ids, weights = torch.empty(T, top, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    gate = torch.full((T,), -9.0, device=DEV) if gated else None
    moe.select(logits if partials > 1 else logits[0], experts, bias, top, ids, weights, gate_col, gate)
    z = logits[0].clone()
    for k in range(1, partials):                          # the order of additions
        z += logits[k]
    chosen = torch.topk(z[:, :experts] + bias, top, dim=-1)
    assert torch.equal(ids.long(), chosen.indices)
    # softmax of numbers of a few units: exponential, sum of six and a quotient
    assert torch.allclose(weights.double(), torch.softmax(chosen.values.double(), -1), rtol=2e-6, atol=0)
    if gated:
        assert torch.allclose(gate.double(), torch.sigmoid(z[:, gate_col].double()), rtol=1e-6, atol=0)


def test_the_second_stream_is_used_up_to_its_limit_and_not_beyond(monkeypatch):
    """What test_the_shared_expert_beside_the_router_changes_no_bits compares are two ways and not one twice."""
    import copy
    import contextlib

    from microllm_rocm_b200.config.gedalix import PRESETS, GedalixConfig
    from microllm_rocm_b200.engine.loading import random_engine
    from microllm_rocm_b200.engine.step import StepEntry
    from microllm_rocm_b200.kernels import ops
    from microllm_rocm_b200.parts import routed
    raw = copy.deepcopy(PRESETS["gedalix-small"])
    raw["layers"], raw["max_positions"] = raw["layers"][:3], 256
    engine = random_engine(GedalixConfig.from_dict(raw), seed=3, max_tokens=1024, max_requests=64, draw_on_device=True)
    engine.model.replay_layers = False                    # (a recorded layer is issued again without this function)
    entered, real = [], ops.on_side_stream

    @contextlib.contextmanager
    def counted():
        entered.append(ops._stream())
        with real() as side:
            yield side
    monkeypatch.setattr(ops, "on_side_stream", counted)
    routed_layers = sum(isinstance(b.feed_forward, routed.RoutedExperts) for b in engine.model.blocks)
    assert routed_layers > 0
    for tokens, limit, uses in ((1, 32, True), (8, 32, True), (32, 32, True), (33, 32, False), (8, 0, False), (8, 8, True), (9, 8, False)):
        monkeypatch.setattr(routed, "SIDE_MAX_TOKENS", limit)
        entered.clear()
        ids = [f"{tokens}.{limit}.{i}" for i in range(tokens)]
        for rid in ids:
            engine.cache.add(rid)
        engine.step([StepEntry(rid, [5 + i], [0]) for i, rid in enumerate(ids)])
        for rid in ids:
            engine.cache.release(rid)
        assert bool(entered) == uses and (not uses or len(entered) >= routed_layers), (tokens, limit, entered)
    engine.check_device_errors()


def test_every_host_thread_has_a_second_stream_of_its_own():
    """Two threads fork, launch and join side by side, each on its own stream and events."""
    import threading

    from microllm_rocm_b200.kernels import ops
    n, failures, handles = 1 << 20, [], {}
    barrier = threading.Barrier(2)

    def work(name):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                x, one = torch.zeros(n, device=DEV), torch.ones(n, device=DEV)
                handles[name] = ops.side_stream()
                barrier.wait(timeout=30)
                for i in range(50):
                    with ops.on_side_stream() as side:
                        assert side == handles[name] and ops._stream() == side
                        ops.add_inplace(x, one)
                    ops.join(side)
                    ops.add_inplace(x, one)               # behind the join: on the thread's own stream
                stream.synchronize()
                assert bool((x == 100).all())
        except BaseException as e:                        # noqa: BLE001  (reported by the test's thread)
            failures.append((name, repr(e)))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
    assert len(set(handles.values())) == 2 and ops.side_stream() not in handles.values()
