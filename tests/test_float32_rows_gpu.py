"""In float32 a row's bits depend on the row and the weights alone: not on how many rows are beside it, nor on whether the product in
front of a norm left parts at that row count."""
import pytest
import torch

import dryft_challenge_htn_2026_b200 as dk
from dryft_challenge_htn_2026_b200.csrc import api
from dryft_challenge_htn_2026_b200.engine import Runner
from dryft_challenge_htn_2026_b200.parts.linear import linear
from helpers import random_tokens

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


@pytest.mark.parametrize("N,K", [(2560, 4096), (5120, 5120), (1000, 1088)])
def test_product_and_norm_at_any_number_of_rows(N, K):
    most = 3000 if N == 1000 else 544
    x, w, h = rnd(most, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5), rnd(most, N, seed=3)
    norm = 1 + 0.1 * rnd(N, seed=4)
    split, got = set(), {}
    for M in (1, 64, 65, 130, 256, most):
        y = linear(x[:M].contiguous(), w, allow_partial=True)
        split.add(isinstance(y, api.Partial))
        stream, a = h[:M].clone(), torch.empty(M, N, device=DEV)
        api.add_rmsnorm(stream, y, norm, 1e-6, a)
        rows = torch.tensor([0, M - 1], dtype=torch.int32, device=DEV)
        at = torch.empty(2, N, device=DEV)
        api.add_rmsnorm(h[:M].clone(), y, norm, 1e-6, at, rows)
        assert torch.equal(at, a[rows.long()])
        for r in (0, 63, 64):
            if r < M:
                for bits, new in zip(got.setdefault(r, (stream[r], a[r])), (stream[r], a[r])):
                    assert torch.equal(bits, new), (M, r)
    assert split == {True, False}                # both kinds of plans were among these row counts


def test_rows_off_16_byte_boundaries_and_widths_of_no_multiple_of_four():
    for H, shift in ((256, 1), (258, 0), (8196, 0)):
        buf = rnd(80 * H + 1, seed=5)
        h = buf[shift:shift + 80 * H].view(80, H).clone() if shift == 0 else buf[shift:].view(80, H)
        norm, a = 1 + 0.1 * rnd(H, seed=6), torch.empty(80, H, device=DEV)
        ref = h.double() * torch.rsqrt((h.double() ** 2).mean(-1, keepdim=True) + 1e-6) * norm.double()
        api.add_rmsnorm(h, None, norm, 1e-6, a)
        assert float((a.double() - ref).abs().max()) <= 4e-6 * float(ref.abs().max())     # H * 2^-25 of a mean of squares, halved by the root


def test_a_whole_model_gives_a_sequence_the_same_bits_however_it_comes(tmp_path):
    """Prompts alone and in batches of 20 to over 500 rows, portions, and single tokens beside others: widths whose products leave
    parts at some of these row counts."""
    cfg = dk.Qwen3Config.from_dict(dict(
        architectures=["Qwen3ForCausalLM"], vocab_size=300, hidden_size=1024, intermediate_size=1088, num_hidden_layers=2,
        num_attention_heads=16, num_key_value_heads=4, head_dim=64, rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False,
        max_position_embeddings=1024))
    folder = str(tmp_path / "wide")
    dk.write_random_model(cfg, folder, seed=0, dtype=torch.float32, matrix_std=0.03)
    runner = Runner(dk.load_model(folder, torch.float32), 64 * 40, 8)
    seq, others = random_tokens(300, 40, 1), [random_tokens(300, n, 2 + n) for n in (3, 50, 400, 90)]

    def run(beside, cut):
        slots = [runner.begin() for _ in range(1 + len(beside))]
        out = runner.step([(slots[0], seq[:cut], list(range(cut)))] + [(s, o[:-24], []) for s, o in zip(slots[1:], beside)]).clone()
        rows = [out]
        for k in range(cut, 40, 3 if cut % 2 else 1):
            new = seq[k:k + (3 if cut % 2 else 1)]
            at = k - cut
            rows.append(runner.step([(slots[0], new, list(range(len(new))))] +
                                    [(s, o[len(o) - 24 + at:len(o) - 24 + at + len(new)], []) for s, o in zip(slots[1:], beside)]).clone())
        for s in slots:
            runner.end(s)
        return torch.cat(rows)

    want = run([], 40)
    for beside, cut in ((others[1:2], 40), (others[1:], 40), (others[1:], 20), ([], 28), (others[1:3], 31)):
        assert torch.equal(run(beside, cut), want), (len(beside), cut)
