"""Dependent launches change no bit: whole models of every design through prompts, portions and single tokens, launched plainly and
replayed, with every kernel behind the full end of the one before, with dependent launches in the steps (as users run), and with
all of them dependent. The kernels of these small models take a few microseconds each, so one that read before its wait what the
one before it writes would meet it unfinished."""
import importlib

import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api
from dryft_challenge_htn_2026_b200.engine import DecodeLoop, Runner, load_model
from helpers import make_folder, random_tokens

pytestmark = pytest.mark.gpu
DESIGNS = {"qwen3": "BDE", "nilivik": "PR", "pibulix": "AC", "venidra": "AC", "nevotar": "AC", "fukatar": "AC", "mozutar": "AC"}


def rows(runner, loop, vocab):
    """Logits of every kind of step, in one tensor."""
    out = []
    seqs = [random_tokens(vocab, n, 7 + n) for n in (1, 70, 23, 190)]
    slots = [runner.begin() for _ in seqs]
    for graph in (False, True, True):                                        # plain, captured's first plain run, captured
        again = [runner.begin() for _ in seqs]
        out.append(runner.step([(s, t, [0, len(t) - 1]) for s, t in zip(again, seqs)], graph=graph).clone())
        for s in again:
            runner.end(s)
    out.append(runner.step([(s, t, [len(t) - 1]) for s, t in zip(slots, seqs)]).clone())
    out.append(runner.step([(s, random_tokens(vocab, 5, s), [4]) for s in slots]).clone())
    for k in range(6):                                                       # single tokens: step function
        out.append(runner.step([(s, [(11 * k + s) % vocab], [0]) for s in slots]).clone())
    for k in range(6):                                                       # and decode state, plain or replayed
        out.append(loop.forced_step([(s, [(13 * k + s) % vocab], [0]) for s in slots]).clone())
    for s in slots:
        runner.end(s)
    return torch.cat(out)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("design,name", [(d, n) for d, names in DESIGNS.items() for n in names])
def test_a_models_bits_do_not_hang_on_how_its_kernels_are_launched(tmp_path, design, name, dtype):
    folder = make_folder(tmp_path, name) if design == "qwen3" else importlib.import_module(f"test_{design}_gpu").make_model(tmp_path, name)[0]
    model = load_model(folder, dtype)
    want = None
    for on in (False, None, True):
        api.set_pdl(on)
        for use_graph in (False, True):
            runner = Runner(model, 64 * 40, 10)
            got = rows(runner, DecodeLoop(runner, use_graph), model.spec.vocab_size)
            if want is None:
                want = got
            assert torch.equal(got, want), (on, use_graph)
