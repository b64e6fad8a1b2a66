"""Single tokens of the recurrences with a state: padding rows, and tokens of one state directly behind one another."""
import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api

pytestmark = pytest.mark.gpu
DEV = "cuda"
H = 2


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV) * 0.1


def i32(*v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def steps(op, dtype, D, n, seed):
    """One single-token step of ``op`` for n rows: (run(out, state, positions, slots), its decays and inputs made from ``seed``)."""
    q, k, v = (rnd(n, H * D, seed=seed + i).to(dtype) for i in range(3))
    if op == "linear":
        decay = 0.5 + 0.1 * torch.arange(H, device=DEV, dtype=torch.float32)
        return lambda out, state, pos, slot: api.linear_attention(q, k, v, out, state, None, pos, slot, decay, n, H, D, D)
    z, bias = rnd(n, H * D, seed=seed + 3), rnd(H * D, seed=seed + 4)
    return lambda out, state, pos, slot: api.gated_linear_attention(q, k, v, out, state, None, pos, slot, z.clone(), bias, 4.0, 1.0, n,
                                                                    H, D, D)


OPS = [("linear", torch.float32, 24), ("linear", torch.bfloat16, 64), ("gated", torch.float32, 24), ("gated", torch.bfloat16, 128)]


@pytest.mark.parametrize("op,dtype,D", OPS)
def test_padding_rows_behind_the_end_of_the_slots(op, dtype, D):
    """A padded decode step has a position for every row and slots for its sequences only: what lies behind them is not used."""
    n, real = 5, 2
    run = steps(op, dtype, D, n, 20)
    start, out = rnd(3, H, D, D, seed=30), torch.full((n, H * D), 7.0, device=DEV)
    state, pos = start.clone(), i32(3, 9, -1, -1, -1)
    run(out, state, pos, i32(2, 0))
    whole, other = torch.full((n, H * D), 7.0, device=DEV), start.clone()
    run(whole, other, pos, i32(2, 0, 1, 1, 1))
    assert torch.equal(out, whole) and torch.equal(state, other)
    assert not bool(out[real:].any()) and torch.equal(state[1], start[1]) and not torch.equal(state[0], start[0])


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("op,dtype,D", OPS)
def test_tokens_of_one_state_directly_behind_one_another(op, dtype, D, captured):
    """Dependent launches, in a step and for every call, against launches behind the full end of the one before: each token works from
    the state that the one before it left."""
    n, tokens = 40, 12
    runs = [steps(op, dtype, D, n, 40 + 10 * t) for t in range(tokens)]
    start, slot = rnd(n, H, D, D, seed=31), torch.randperm(n, generator=torch.Generator().manual_seed(32)).int().to(DEV)
    pos = torch.arange(n, dtype=torch.int32, device=DEV) - 1                     # the first row is padding
    state, outs = start.clone(), [torch.zeros(n, H * D, device=DEV) for _ in runs]

    def chain():
        for run, out in zip(runs, outs):
            run(out, state, pos, slot)

    def result(go):
        state.copy_(start)
        torch.cuda.synchronize()
        go()
        return torch.cat([state.flatten()] + [o.flatten() for o in outs])

    def replayed(body):
        body()                                                                    # sizes everything
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            body()
        return graph.replay

    def step():
        with api.dependent_launches():
            chain()

    try:
        api.set_pdl(False)
        want = result(chain)
        assert not torch.equal(want[:start.numel()].view_as(start), start)
        api.set_pdl(True)
        every = replayed(chain) if captured else chain
        for _ in range(3):
            assert torch.equal(result(every), want)
        api.set_pdl(None)
        in_step = replayed(step) if captured else step
        for _ in range(3):
            assert torch.equal(result(in_step), want)
    finally:
        api.set_pdl(None)
