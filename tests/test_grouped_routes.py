"""What the grouped products hand to their launchers, on the CPU: the launchers are stand-ins that note their arguments, so a call
that would write or read out of range on a device shows as an argument."""
import pytest
import torch

from microllm_rocm_b200.kernels import grouped, ops
from microllm_rocm_b200.kernels.build import KernelError


@pytest.fixture
def calls(monkeypatch):
    """[(launcher, {argument name: value})] of the calls made."""
    import re

    from microllm_rocm_b200.kernels import build
    made = []

    class Library:
        def __init__(self, source):
            text = open(f"{build.CSRC}/{source}").read()
            self.names = {fn: [p.strip().split()[-1].lstrip("*") for p in params.split(",")]
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
    monkeypatch.setattr(grouped, "sm_count", lambda device: 148)
    return made


ROUTES = {"pair": (True, True), "mma": (False, True), "plain": (False, False)}       # USE_PAIRS, USE_TENSOR_CORES


def use(monkeypatch, route):
    pairs, tensor_cores = ROUTES[route]
    monkeypatch.setattr(grouped, "USE_PAIRS", pairs)
    monkeypatch.setattr(grouped, "USE_TENSOR_CORES", tensor_cores)


def operands(rows=24, G=3, N=32, K=64):
    a, w = torch.zeros(rows, K, dtype=torch.bfloat16), torch.zeros(G, N, K, dtype=torch.bfloat16)
    return a, w, torch.tensor([0, 8, 8, rows], dtype=torch.int32), torch.zeros(1, dtype=torch.int32)


@pytest.mark.parametrize("route", sorted(ROUTES))
@pytest.mark.parametrize("dtype", [torch.float16, torch.int32, torch.float64])
def test_outputs_of_other_types_are_refused_on_every_route(calls, monkeypatch, route, dtype):
    use(monkeypatch, route)
    a, w, offsets, flag = operands()
    with pytest.raises(KernelError, match="dtype"):
        grouped.grouped_linear(a, w, torch.zeros(24, 32, dtype=dtype), rows=24, group_offsets=offsets, error_flag=flag)
    with pytest.raises(KernelError, match="dtype"):
        grouped.grouped_silu_mul(a, w, torch.zeros(24, 16, dtype=dtype), rows=24, group_offsets=offsets, error_flag=flag)
    assert not [fn for fn, _ in calls if fn in ("mlb_grouped_pair", "mlb_grouped_mma", "mlb_gather_rows")]


@pytest.mark.parametrize("rows, held", [(64, 24), (24, 24), (20, 24), (0, 24)])
def test_the_pair_kernel_reads_no_row_behind_the_matrix(calls, monkeypatch, rows, held):
    """`rows` may be more than the list holds, and than `a` has: the kernel's copies take whole boxes of rows up to the number it is
    given, so that number stays within the matrix they come from."""
    use(monkeypatch, "pair")
    a, w, offsets, flag = operands(held)
    order = torch.zeros(rows, dtype=torch.int32)
    grouped.grouped_linear(a, w, torch.zeros(rows, 32), rows=rows, group_offsets=offsets, error_flag=flag)
    grouped.grouped_silu_mul(a, w, torch.zeros(rows, 16), rows=rows, group_offsets=offsets, error_flag=flag)
    grouped.grouped_silu_mul(a, w, torch.zeros(rows, 16), rows=rows, group_offsets=offsets, a_rows=order, error_flag=flag)
    given = [args["M"] for fn, args in calls if fn == "mlb_grouped_pair"]
    assert given == ([min(rows, held), min(rows, held), rows] if rows else [])          # with a list the rows are gathered first, all of them


def test_the_pair_route_refuses_what_the_others_refuse(calls, monkeypatch):
    use(monkeypatch, "pair")
    a, w, offsets, flag = operands()
    for bad in ({"row_tile": 32}, {"a_row_div": 0}, {"a_row_div": -2}, {"rows": -1}):
        out = {"rows": 24, "group_offsets": offsets, "error_flag": flag, **bad}
        with pytest.raises(KernelError):
            grouped.grouped_linear(a, w, torch.zeros(24, 32), **out)
        with pytest.raises(KernelError):
            grouped.grouped_silu_mul(a, w, torch.zeros(24, 16), **out)
    assert not calls


def test_the_pair_launcher_refuses_unknown_activations():
    """The library itself, which answers before it touches a device."""
    L = ops.lib(grouped.PAIR_SOURCE)
    matrix = torch.zeros(64, 64, dtype=torch.bfloat16)
    list_of = torch.zeros(2, dtype=torch.int32)
    at = matrix.data_ptr()

    def status(act, dual, row_scale):
        return L.mlb_grouped_pair(at, 64, at, at, 64, list_of.data_ptr(), None, row_scale, None, 1, dual, act, 16 if dual else 0, 0, 16, 64, 1,
                                  64, 64, 148, None, 0)
    assert status(0, 1, None) == 0 and status(0, 0, None) == 0 and status(0x3f400000, 1, at) == 0       # (no rows: nothing to do)
    for refused in ((1, 1, None), (-1, 1, None), (0, 0, at)):
        assert status(*refused) != 0
