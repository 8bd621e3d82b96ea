"""Kernels whose tiles or pieces follow the sizes: fp32 products of more rows than the streaming kernel's, the split of latent attention's projection."""
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
