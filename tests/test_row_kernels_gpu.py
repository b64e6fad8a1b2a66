"""Row kernels at the edges of the forms they come in, against float64."""
import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def near(got, want, dtype, terms=1):
    """bfloat16: half a unit in the last place of 8 bits; both: a few float32 roundings a term of the sums behind a value."""
    slack = (terms + 8) * 2.0 ** -23
    bound = (slack + (2.0 ** -8 if dtype == torch.bfloat16 else 0)) * want.abs() + slack * float(want.abs().max())
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hd,nh,nkv", [(64, 3, 1), (128, 4, 2)])
@pytest.mark.parametrize("rows,parts", [(1, 1), (5, 3), (70, 8), (9, 9), (3, 17)])
def test_norm_rotation_and_cache_write_of_float32_rows(dtype, hd, nh, nkv, rows, parts):
    """Heads of 64 and 128 as parts (one, a batch of eight, more) and as a float32 projection: q, the cache, what must stay untouched,
    padding rows; without norm, without rotation, into a dense result, and for a layer that only reads the cache."""
    heads = nh + 2 * nkv
    ws = rnd(parts, rows, heads * hd, seed=1)
    x = ws.double().sum(0).view(rows, heads, hd)
    qn, kn = 1 + 0.1 * rnd(hd, seed=2), 1 + 0.1 * rnd(hd, seed=3)
    ang = rnd(200, hd // 2, seed=4)
    cos, sin = ang.cos(), ang.sin()
    pos = (torch.arange(rows, dtype=torch.int32, device=DEV) * 37) % 190
    if rows > 2:
        pos[1] = -1
    seq = torch.arange(rows, dtype=torch.int32, device=DEV)
    table = torch.arange(rows * 3, dtype=torch.int32, device=DEV).view(rows, 3).flip(1).contiguous()
    live = (pos >= 0).nonzero().flatten()

    def want(norm, turn):
        y = x[live].clone()
        for lo, hi, w in ((0, nh, qn), (nh, nh + nkv, kn)):
            if norm:
                y[:, lo:hi] = y[:, lo:hi] * torch.rsqrt(y[:, lo:hi].pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
        if turn:
            c, s = cos[pos[live].long()].double()[:, None], sin[pos[live].long()].double()[:, None]
            a, b = y[:, :nh + nkv, :hd // 2].clone(), y[:, :nh + nkv, hd // 2:].clone()
            y[:, :nh + nkv] = torch.cat([a * c - b * s, b * c + a * s], -1)
        return y

    pages, slots = table[live, (pos[live] // 64).long()].long(), (pos[live] % 64).long()
    for norm, turn, writes in ((True, True, True), (False, True, True), (True, False, False)):
        rows_in = [api.Partial(ws)] + ([ws[0]] if dtype == torch.float32 and parts == 1 else [])
        for src in rows_in:
            q = torch.full((rows, nh * hd), 7.0, dtype=dtype, device=DEV)
            k = torch.full((rows * 3, nkv, 64, hd), 7.0, dtype=dtype, device=DEV)
            v = k.clone()
            api.qk_norm_rope_write(src, q, qn if norm else None, kn if norm else None, cos if turn else None, sin if turn else None,
                                   pos, seq, table, k, v, nh, nkv, hd, 1e-6, write_kv=writes)
            y = want(norm, turn)
            near(q[live].view(-1, nh, hd), y[:, :nh], dtype, parts + hd)
            assert bool((q[pos < 0] == 7.0).all())
            touched = torch.zeros(k.shape[0], 64, dtype=torch.bool, device=DEV)
            if writes:
                near(k[pages, :, slots], y[:, nh:nh + nkv], dtype, parts + hd)
                near(v[pages, :, slots], y[:, nh + nkv:], dtype, parts)
                touched[pages, slots] = True
            for store in (k, v):
                assert bool((store.transpose(1, 2)[~touched] == 7.0).all())
            dense = torch.full((rows, heads * hd), 7.0, dtype=dtype, device=DEV)
            api.qk_norm_rope_write(src, None, qn if norm else None, kn if norm else None, None, None, pos, seq, table, k, v, nh, nkv, hd,
                                   1e-6, dense_out=dense)
            near(dense[live].view(-1, heads, hd), want(norm, False), dtype, parts + hd)
            assert bool((dense[pos < 0] == 7.0).all())
