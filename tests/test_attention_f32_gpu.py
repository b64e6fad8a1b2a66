"""Float32 attention of prompts and of single tokens over the paged cache against float64: ragged portions, pages that end inside a
tile, windows, groups that do not divide a tile, and bits that do not depend on which of the two kernels a token goes through."""
import numpy as np
import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api
from dryft_challenge_htn_2026_b200.parts.attention import QueryTiles
from test_kernels_gpu import paged_setup, rnd

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ref64(q, s, nh, nkv, hd, window):
    out = torch.empty(q.shape[0], nh, hd, dtype=torch.float64, device=DEV)
    qd = q.double().view(-1, nh, hd)
    for t in range(q.shape[0]):
        i, p = int(s["row_seq"][t]), int(s["row_pos"][t])
        lo = max(0, p - window + 1) if window else 0
        K, V = (s[x][i][lo:p + 1].double().repeat_interleave(nh // nkv, 1) for x in ("dense_k", "dense_v"))
        w = torch.softmax(torch.einsum("phd,hd->hp", K, qd[t]) * hd ** -0.5, -1)
        out[t] = torch.einsum("hp,phd->hd", w, V)
    return out.view(q.shape[0], nh * hd)


@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 2, 128, 0), (4, 4, 64, 0), (6, 2, 128, 90), (16, 1, 64, 7), (10, 2, 64, 64)])
def test_attention_f32(nh, nkv, hd, window):
    before, new = [0, 100, 0, 63, 130, 640], [70, 150, 1, 2, 65, 17]
    s = paged_setup(before, new, nkv, hd, torch.float32, seed=5)
    s["k_store"].masked_fill_(s["k_store"] == 0, float("nan"))      # what no token wrote must not reach any result
    s["v_store"].masked_fill_(s["v_store"] == 0, float("nan"))
    q = rnd(s["n_tok"], nh * hd, seed=6)
    plan = QueryTiles(api.F32_TILE_ROWS // (nh // nkv)).build(new, before, False)
    out = torch.full_like(q, float("nan"))
    api.attention_prompt_f32(q, out, s["k_store"], s["v_store"], torch.tensor(plan, device=DEV), s["cu_q"], s["pos0"], s["table"], nh,
                             nkv, hd, window, hd ** -0.5)
    ref = ref64(q, s, nh, nkv, hd, window)
    # scores of unit normal heads: below 8 with hd / 4 roundings of 2^-24 of their terms each, as an error of the weights; the
    # values' sum adds 64 + pages more: 2e-5 of the largest value (4.5) bounds both
    assert float((out.double() - ref).abs().max()) <= 2e-5 * 4.5
    # the same tokens one by one, the sequences in another order and a padding row among them
    rows = torch.tensor([0, 69, 70, 219, 220, 221, 222, 230, 287, s["n_tok"] - 1], device=DEV)
    pos, seq = s["row_pos"][rows].clone(), s["row_seq"][rows].long()
    pos[4] = -1
    one = torch.full((len(rows), nh * hd), float("nan"), device=DEV)
    api.attention_decode_f32(q[rows].contiguous(), one, s["k_store"], s["v_store"], pos, s["table"][seq].contiguous(), nh, nkv, hd,
                             window, hd ** -0.5)
    assert float(one[4].abs().max()) == 0.0
    keep = np.array([i for i in range(len(rows)) if i != 4])
    assert torch.equal(one[keep], out[rows][keep])


@pytest.mark.parametrize("hd", [64, 128])
def test_pages_of_keys_with_infinitely_low_scores(hd):
    """Keys whose score is -inf weigh nothing, also where a page holds (or shows a query) no others: before, between and after
    pages with finite ones, as a page's first visible key, and NaN and +inf still come through."""
    n = 200
    s = paged_setup([0], [n], 1, hd, torch.float32, seed=11)
    q = rnd(n, 2 * hd, seed=12).abs() + 0.1             # positive: a key of -inf scores -inf
    low = [slice(0, 64), slice(100, 128), slice(128, 192)]
    page = s["table"][0].long()
    for part in low:
        for j in range(part.start, part.stop):
            s["k_store"][page[j // 64], 0, j % 64] = float("-inf")
            s["dense_k"][0][j, 0] = float("-inf")
    plan = QueryTiles(api.F32_TILE_ROWS // 2).build([n], [0], False)

    def both():
        out, one = torch.empty_like(q), torch.empty_like(q)
        api.attention_prompt_f32(q, out, s["k_store"], s["v_store"], torch.tensor(plan, device=DEV), s["cu_q"], s["pos0"], s["table"],
                                 2, 1, hd, 0, hd ** -0.5)
        api.attention_decode_f32(q, one, s["k_store"], s["v_store"], s["row_pos"], s["table"].expand(n, -1).contiguous(), 2, 1, hd, 0,
                                 hd ** -0.5)
        return out, one

    out, one = both()
    ref = ref64(q, s, 2, 1, hd, 0)
    assert bool(out[:64].isnan().all()) and bool(ref[:64].isnan().all())           # none but -inf in sight: 0 / 0
    assert float((out[64:].double() - ref[64:]).abs().max()) <= 2e-5 * 4.5         # the bound of the test above
    assert torch.equal(one[64:], out[64:]) and bool(one[:64].isnan().all())
    for value in (float("nan"), float("inf")):
        s["k_store"][page[2], 0, 5] = value                                       # position 133, in a page of -inf
        out, one = both()
        assert bool(out[133:].isnan().all()) and bool(one[133:].isnan().all()) and not bool(out[64:133].isnan().any())


@pytest.mark.parametrize("share", [1, 2, 4])
def test_sequences_in_several_launches(monkeypatch, share):
    """The bits of one launch, whatever the share of sequences a launch takes."""
    nh, nkv, hd, before = 4, 2, 64, [0, 100, 63, 640, 64, 5, 200]
    s = paged_setup(before, [1] * 7, nkv, hd, torch.float32, seed=13)
    q, out = rnd(7, nh * hd, seed=14), []
    for limit in (api.F32_DECODE_BYTES, share * 4 * nh * s["table"].shape[1] * (hd + 2)):
        monkeypatch.setattr(api, "F32_DECODE_BYTES", limit)
        out.append(torch.empty_like(q))
        api.attention_decode_f32(q, out[-1], s["k_store"], s["v_store"], s["row_pos"], s["table"], nh, nkv, hd, 0, hd ** -0.5)
    assert torch.equal(out[0], out[1])


def test_refusals():
    s = paged_setup([0], [3], 1, 32, torch.float32, seed=7)
    q = rnd(3, 64, seed=8)
    with pytest.raises(api.KernelError):
        api.attention_decode_f32(q, torch.empty_like(q), s["k_store"], s["v_store"], s["row_pos"], s["table"], 2, 1, 32, 0, 0.1)


@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 2, 128, 0), (4, 4, 64, 0), (6, 2, 128, 90), (16, 1, 64, 7), (10, 2, 64, 64), (3, 1, 128, 0)])
def test_short_tiles_give_the_bits_of_long_ones(nh, nkv, hd, window):
    """Tiles of 32 rows against tiles of 64 (5 and 3 heads a kv head leave rows of both unused): the same order of arithmetic a row;
    portions that start and end anywhere in a page, and what no token wrote is NaN."""
    before, new = [0, 100, 0, 63, 130, 640, 3], [70, 150, 1, 2, 65, 17, 62]
    s = paged_setup(before, new, nkv, hd, torch.float32, seed=15)
    s["k_store"].masked_fill_(s["k_store"] == 0, float("nan"))
    s["v_store"].masked_fill_(s["v_store"] == 0, float("nan"))
    q, out = rnd(s["n_tok"], nh * hd, seed=16), []
    for rows in (api.F32_TILE_ROWS, api.F32_SHORT_TILE_ROWS):
        plan = torch.tensor(QueryTiles(rows // (nh // nkv)).build(new, before, False), device=DEV)
        out.append(torch.full_like(q, float("nan")))
        api.attention_prompt_f32(q, out[-1], s["k_store"], s["v_store"], plan, s["cu_q"], s["pos0"], s["table"], nh, nkv, hd, window,
                                 hd ** -0.5, rows)
    assert torch.equal(out[0], out[1]) and bool(out[0].isfinite().all())
    with pytest.raises(api.KernelError):
        api.attention_prompt_f32(q, out[0], s["k_store"], s["v_store"], plan, s["cu_q"], s["pos0"], s["table"], nh, nkv, hd, window, 0.1, 48)
