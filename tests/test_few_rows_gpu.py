"""Kernels whose tiles or pieces follow the sizes: fp32 products of more rows than the streaming kernel's, the split of latent attention's projection, the
stores of the grouped product."""
import pytest
import torch

DEV = "cuda"


@pytest.mark.gpu
@pytest.mark.parametrize("M", [33, 40, 41, 48, 49, 57, 64, 65, 81, 97, 113, 129, 333])
@pytest.mark.parametrize("N, K", [(64, 512), (131, 1000), (200, 77)])
def test_fp32_rows_have_the_bits_of_a_row_alone(M, N, K):
    """Every size of row tile (40, 48, 56 and 64 rows), last tiles and last columns that are not full, rows that travel in fours."""
    from microllm_rocm_b200.kernels import ops
    g = torch.Generator(DEV).manual_seed(M)
    x, w, bias = (torch.randn(*s, generator=g, device=DEV) for s in ((M, K), (N, K), (N,)))
    out = torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_f32(x, w, out, bias=bias)
    for m in (0, 31, 32, M // 2, M - 2, M - 1):
        row = torch.empty(1, N, device=DEV)
        ops.gemm_f32(x[m:m + 1].contiguous(), w, row, bias=bias)
        assert torch.equal(out[m:m + 1], row), m
    assert bool(torch.isfinite(out).all())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, dim, rot, rot_dims, interleaved, partials", [(3, 128, 64, 64, False, 1), (16, 128, 64, 32, False, 5), (5, 32, 16, 8, True, 3), (2, 64, 64, 64, True, 1)])
def test_the_split_of_a_projection_four_columns_at_a_time(dtype, heads, dim, rot, rot_dims, interleaved, partials):
    """Rows that start on 16 bytes go four columns a thread, the same rows one column further on do not: the same bits."""
    from microllm_rocm_b200.kernels import latent
    rank, T, page = 64, 9, 4
    width = heads * (dim + rot) + rank + rot + heads * 32
    g = torch.Generator(DEV).manual_seed(dim + rot_dims)
    proj = torch.randn(partials, T, width, generator=g, device=DEV)
    norm, freq = torch.rand(rank, generator=g, device=DEV), torch.rand(rot_dims // 2, generator=g, device=DEV)
    on = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    positions, seq, table = on([0, 1, 2, 900, 901, 902, 5, 6, 7]), on([0] * 3 + [1] * 3 + [2] * 3), torch.full((3, 226), -1, dtype=torch.int32, device=DEV)
    table[0, 0], table[1, 225], table[2, 1] = 3, 1, 0
    results = []
    for shift in (0, 1):
        src = torch.zeros(partials, T, width + 4, device=DEV)
        src[..., shift:shift + width] = proj
        q_plain, q_full = torch.zeros(T, heads * dim, dtype=dtype, device=DEV), torch.zeros(T, heads * (rank + rot), dtype=dtype, device=DEV)
        gate, pages = torch.zeros(T, heads * 32, device=DEV), torch.zeros(4, page, rank + rot, dtype=dtype, device=DEV)
        flag = torch.zeros(1, dtype=torch.int32, device=DEV)
        latent.prepare(src, q_col=shift, kv_col=shift + heads * (dim + rot), gate_col=shift + heads * (dim + rot) + rank + rot, norm_weight=norm, eps=1e-5,
                       positions=positions, token_seq=seq, block_table=table, inv_freq=freq, rot_dims=rot_dims, q_plain=q_plain, q_full=q_full, pages=pages,
                       gate_out=gate, heads=heads, dim=dim, rot_dim=rot, rank=rank, error_flag=flag, interleaved=interleaved, magnitude=1.25)
        results.append((q_plain, q_full, gate, pages))
        assert int(flag.item()) == 0
    for a, b in zip(*results):
        assert torch.equal(a, b) and bool((a != 0).any())


@pytest.mark.gpu
@pytest.mark.parametrize("row_tile", [16, 64, 128])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N, K, factor, listed", [(512, 128, False, False), (128, 512, True, False), (72, 64, True, False), (96, 40, False, True)])
def test_outputs_stored_together_have_the_bits_of_each_alone(row_tile, out_dtype, N, K, factor, listed):
    """Rows that start on 16 bytes take several columns to a store, rows of an odd pitch one: whole tiles and parts, rows that nobody wants."""
    from microllm_rocm_b200.kernels import grouped
    G, rows = 3, 131
    g = torch.Generator(DEV).manual_seed(N)
    w = (torch.randn(G, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    on = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kw, width = (dict(a_group_cols=K, c_group_cols=N), G * N) if not listed else \
        (dict(group_offsets=on([0, 70, 70, rows]), a_rows=on([(7 * i) % rows for i in range(rows)]), c_rows=on([-1 if i % 5 == 0 else i for i in range(rows)])), N)
    a = torch.randn(rows, K if listed else G * K, generator=g, device=DEV).bfloat16()
    by = torch.rand(rows, width + 1, generator=g, device=DEV)
    results = []
    for extra in (0, 1):
        out = torch.full((rows, width + extra), 7.0, dtype=out_dtype, device=DEV)
        grouped.USE_PAIRS = False
        try:
            grouped.grouped_linear(a, w, out, rows=rows, factor=by[:, :width + extra].contiguous() if factor else None, row_tile=row_tile, **kw)
        finally:
            grouped.USE_PAIRS = None
        results.append(out[:, :width])
    assert torch.equal(*results) and int((results[0] == 7.0).sum()) == (len(range(0, rows, 5)) * N if listed else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("w_constant", [False, True])
def test_products_of_weights_that_the_kernel_in_front_writes(w_constant):
    """Without the caller's word nothing is read before that kernel has ended; with it the weights are as they were all along."""
    from microllm_rocm_b200.kernels import grouped, ops
    G, N, K, rows = 16, 512, 512, 8
    g = torch.Generator(DEV).manual_seed(1)
    a = torch.randn(rows, G * K, generator=g, device=DEV).bfloat16()
    source = torch.randn(8, G, N, K, generator=g, device=DEV)
    for i in range(8):
        w, out, want = torch.zeros(G, N, K, dtype=torch.bfloat16, device=DEV), torch.empty(rows, G * N, device=DEV), torch.empty(rows, G * N, device=DEV)
        ops.cast_f32_bf16(source[i], w)
        if w_constant:
            torch.cuda.synchronize()
        grouped.grouped_linear(a, w, out, rows=rows, a_group_cols=K, c_group_cols=N, row_tile=16, w_constant=w_constant)
        torch.cuda.synchronize()
        grouped.grouped_linear(a, w, want, rows=rows, a_group_cols=K, c_group_cols=N, row_tile=16)
        assert torch.equal(out, want) and bool((want != 0).any())
