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
