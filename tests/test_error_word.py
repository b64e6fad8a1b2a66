"""A kernel that gave up a wait leaves a code in the error word and incomplete sums: whoever hands out a step's logits looks there
first. No GPU: the step's model writes the code itself."""
import types

import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api
from dryft_challenge_htn_2026_b200.engine.generate import DecodeLoop
from dryft_challenge_htn_2026_b200.engine.runner import Runner


@pytest.fixture
def word(monkeypatch):
    word = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(api, "_tc_err", word)
    return word


class Step:
    """A runner whose model leaves ``code`` in the error word."""

    def __init__(self, word, is_decode):
        self.code, self.device = 0, torch.device("cpu")
        self.cache = types.SimpleNamespace(commit=lambda slot, n: None)
        self.is_decode = is_decode
        self.model = types.SimpleNamespace(forward=lambda ctx, cache, tap=None: word.fill_(self.code).float())

    def context(self, entries):
        return types.SimpleNamespace(is_decode=self.is_decode)

    step = Runner.step


@pytest.mark.parametrize("is_decode", [False, True])
@pytest.mark.parametrize("code,kernel", [(1, "gemm_tc"), (13, "gemm_f32_tc")])
def test_a_step_that_gave_up_a_wait_raises(word, is_decode, code, kernel):
    run = Step(word, is_decode)
    run.step([(0, [5], [0])])
    run.code = code
    with pytest.raises(api.KernelError, match=f"^{kernel}.*bounded wait.*{code}"):
        run.step([(0, [5], [0])])
    run.code = 0
    run.step([(0, [5], [0])])                # the word was cleared


def test_a_forced_token_that_gave_up_a_wait_raises(word):
    state = types.SimpleNamespace(filled=[(0, 1)], lengths=[3], width=4, graph=None, logits=torch.zeros(1, 8), code=12,
                                  set_tokens=lambda tokens: None, run=lambda: word.fill_(state.code))
    model = types.SimpleNamespace(generation=0, prepare=lambda n: 0)
    cache = types.SimpleNamespace(reserve=lambda slot, n: None, pages_held=lambda slot: 1, length=[3], commit=lambda slot, n: None)
    loop = DecodeLoop(types.SimpleNamespace(model=model, cache=cache), use_graph=False)
    loop.state = state
    with pytest.raises(api.KernelError, match="gemm_f32_tc"):
        loop.forced_step([(0, [7], [0])])
