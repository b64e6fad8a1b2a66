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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hd,nh,nkv", [(64, 3, 1), (128, 4, 2)])
@pytest.mark.parametrize("rows,parts", [(1, 1), (33, 4), (70, 9)])
def test_norm_and_rotation_give_the_same_bits_wherever_the_rows_lie(dtype, hd, nh, nkv, rows, parts):
    """Rows on 16-byte boundaries (four columns a lane) and 4 bytes off them (a number at a time): one order of every sum. In float32
    numbers of any exponent and zeros of both signs beside them, whose last bit shows a different order."""
    heads = nh + 2 * nkv
    ws = rnd(parts * rows * heads * hd, seed=12) * torch.exp2(torch.randint(-9, 9, (parts * rows * heads * hd,), device=DEV))
    ws[::17] = -0.0
    qn, kn, ang = 1 + 0.1 * rnd(hd, seed=13), 1 + 0.1 * rnd(hd, seed=14), rnd(200, hd // 2, seed=15)
    pos = (torch.arange(rows, dtype=torch.int32, device=DEV) * 37) % 190
    seq = torch.arange(rows, dtype=torch.int32, device=DEV)
    table = torch.arange(rows * 3, dtype=torch.int32, device=DEV).view(rows, 3)
    for direct in (False, True) if dtype == torch.float32 and parts == 1 else (False,):
        got = []
        for off in (0, 1):
            flat = torch.empty(ws.numel() + 4, device=DEV)[off:off + ws.numel()]
            src = flat.copy_(ws).view(parts, rows, heads * hd)
            q = torch.zeros(rows, nh * hd, dtype=dtype, device=DEV)
            k = torch.zeros(rows * 3, nkv, 64, hd, dtype=dtype, device=DEV)
            v = k.clone()
            api.qk_norm_rope_write(src[0] if direct else api.Partial(src), q, qn, kn, ang.cos(), ang.sin(), pos, seq, table, k, v, nh, nkv,
                                   hd, 1e-6)
            bits = torch.int16 if dtype == torch.bfloat16 else torch.int32
            got.append([t.view(bits) for t in (q, k, v)])
        for a, b in zip(*got):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,shift", [(4, 0), (516, 0), (2560, 0), (8192, 0), (2560, 1), (8196, 0), (258, 0)])
def test_embedding_with_a_position_vector(dtype, H, shift):
    """Rows of whole fours up to 8,192 on 16-byte boundaries, and rows that are not; a padding row, token ids out of range, far positions."""
    V, rows = 40, 5
    embed = rnd(V * H + shift, seed=5).to(dtype)[shift:].view(V, H)
    tok = torch.tensor([3, 39, 0, 99, -2], dtype=torch.int32, device=DEV)
    pos = torch.tensor([0, 1, -1, 100000, 777], dtype=torch.int32, device=DEV)
    inv = 10000.0 ** (-torch.arange(0, H, 2, device=DEV, dtype=torch.float64) / H)
    w = 1 + 0.1 * rnd(H, seed=6)
    for table, weight in ((inv, w), (None, w), (inv, None)):
        h, a = torch.full((rows, H), 7.0, device=DEV), torch.full((rows, H), 7.0, dtype=dtype, device=DEV)
        api.embed_position_rmsnorm(tok, embed, 1.5, pos, table, weight, 1e-6, h, a)
        want = embed[tok.long().clamp(0, V - 1)].double() * 1.5
        if table is not None:
            ang = pos.clamp(min=0).double()[:, None] * inv
            want = want + torch.stack([ang.sin(), ang.cos()], -1).view(rows, -1)
        near(h, want, torch.float32)
        if weight is not None:
            near(a, want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double(), dtype, H)
        else:
            assert bool((a == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H", [4, 132, 516, 1024, 2560, 8192])
def test_an_embedding_gives_the_same_bits_wherever_its_rows_lie(dtype, H):
    """Table and weights on 16-byte boundaries (four columns a thread) and one number off them (a number at a time), with and without
    positions: products, sines and the sum of squares are rounded alike."""
    V, rows = 40, 129
    table, weight = rnd(V * H, seed=16).to(dtype), 1 + 0.1 * rnd(H, seed=17)
    tok = torch.randint(0, V, (rows,), generator=torch.Generator().manual_seed(18), dtype=torch.int32).to(DEV)
    pos = torch.arange(rows, dtype=torch.int32, device=DEV) * 397 - 1
    for inv in (10000.0 ** (-torch.arange(0, H, 2, device=DEV, dtype=torch.float64) / H), None):
        got = []
        for off in (0, 1):
            embed = torch.empty(V * H + 8, dtype=dtype, device=DEV)[off:off + V * H].copy_(table).view(V, H)
            w = torch.empty(H + 8, device=DEV)[off:off + H].copy_(weight)
            h, a = torch.empty(rows, H, device=DEV), torch.empty(rows, H, dtype=dtype, device=DEV)
            api.embed_position_rmsnorm(tok, embed, 1.3, pos, inv, w, 1e-6, h, a)
            got.append((h.view(torch.int32), a.view(torch.int16 if dtype == torch.bfloat16 else torch.int32)))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nkv,hd,hdv,extra,shift", [(8, 128, 128, 0, 0), (2, 64, 32, 8, 0), (3, 20, 12, 0, 0), (1, 128, 128, 3, 0),
                                                   (2, 64, 64, 0, 1), (1, 576, 0, 0, 0)])
def test_keys_and_values_into_the_cache(dtype, nkv, hd, hdv, extra, shift):
    """Rows of wider matrices, heads and rows of whole 16-byte pieces and not, addresses off them, padding rows, and no values of their own to store."""
    rows, ld = 7, nkv * (hd + hdv) + extra
    proj = rnd(rows * ld + shift, seed=7).to(dtype)[shift:].view(rows, ld)
    k, v = proj[:, :nkv * hd], proj[:, nkv * hd:nkv * (hd + hdv)] if hdv else proj[:, :nkv * hd]
    ks = torch.full((4, nkv, 64, hd), 7.0, dtype=dtype, device=DEV)
    vs = torch.full((4, nkv, 64, hdv), 7.0, dtype=dtype, device=DEV) if hdv else None
    pos = torch.tensor([0, 63, 64, 100, -1, 5, 127], dtype=torch.int32, device=DEV)
    seq = torch.tensor([0, 0, 0, 0, 1, 1, 1], dtype=torch.int32, device=DEV)
    table = torch.tensor([[2, 0], [3, 1]], dtype=torch.int32, device=DEV)
    api.kv_write(k, v, ks, vs, pos, seq, table, nkv, hd, hdv if hdv else hd)
    live = (pos >= 0).nonzero().flatten()
    pages, slots = table[seq[live].long(), (pos[live] // 64).long()].long(), (pos[live] % 64).long()
    for store, x, d in ((ks, k, hd), (vs, v, hdv)):
        if store is None:
            continue
        want = torch.full_like(store, 7.0)
        want[pages, :, slots] = x[live].reshape(len(live), nkv, d)
        assert torch.equal(store, want)


@pytest.mark.parametrize("M,N", [(9, 40000), (128, 31000), (33, 2564)])
def test_heads_of_every_tile_height(M, N):
    """The decode form of the tensor-core product with a float32 result, several tiles a block, a last one that is not full."""
    K = 136
    x, w = rnd(M, K, seed=8).to(torch.bfloat16), rnd(N, K, seed=9, scale=K ** -0.5).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    for bn in api.TC_TILE_HEIGHTS:
        out = torch.full((M, N), float("nan"), device=DEV)
        api.gemm_tc(x, w, api.MODE_STORE_F32, out, (bn, 1))
        assert bool(((out.double() - want).abs() <= K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())).all()), bn
    api.gemm_tc_check()


@pytest.mark.parametrize("lens", [[130] * 8, [64, 1, 200, 63, 65, 300, 2, 128], [70] * 4])
def test_recurrence_in_chunks_of_64_value_columns(lens):
    """Heads enough for blocks of 64 value columns (and, in four sequences of 16 heads, for blocks of 32) against the plain recurrence
    in float64: outputs and states; silu of q, k and v is rounded to bfloat16 as the kernel rounds it."""
    nh, hd, T, n = 16, 128, sum(lens), len(lens)
    proj = rnd(T, 3 * nh * hd, seed=10).to(torch.bfloat16)
    decay = 1.0 - 2.0 ** -(2 + 4 * torch.arange(nh, device=DEV, dtype=torch.float32) / nh)
    state = rnd(n, nh, hd, hd, seed=11)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    act = torch.nn.functional.silu(proj.float()).to(torch.bfloat16).double().view(T, 3, nh, hd)
    want, last = torch.empty(T, nh, hd, dtype=torch.float64, device=DEV), state.double()
    for s in range(n):
        S = last[s]
        for t in range(int(cu[s]), int(cu[s + 1])):
            S = decay.double()[:, None, None] * S + act[t, 1][:, :, None] * act[t, 2][:, None, :]
            want[t] = (act[t, 0][:, :, None] * S).sum(1)
        last[s] = S
    out = torch.full((T, nh * hd), float("nan"), device=DEV)
    slot = torch.arange(n, dtype=torch.int32, device=DEV)
    q, k, v = proj.split(nh * hd, 1)
    api.linear_attention_chunk_bf16(q, k, v, out, state, cu, slot, decay, n, nh, hd, hd)
    # scores and weights are bfloat16 operands of the products: 2^-8 of the terms' norm, states 2^-16
    assert float((out.double().view_as(want) - want).norm() / want.norm()) <= 2.0 ** -7
    assert float((state.double() - last).norm() / last.norm()) <= 2.0 ** -13


@pytest.mark.parametrize("hdv", [64, 128])
def test_value_columns_a_block_change_no_bit_of_the_recurrence(hdv):
    """The same sequences together (blocks of 64 value columns), by halves (32) and one by one (16): outputs and states."""
    nh, hd, lens = 16, 128, [64, 130, 1, 200, 63, 65, 300, 128] * (128 // hdv)
    n, T = len(lens), sum(lens)
    proj = rnd(T, 2 * nh * hd + nh * hdv, seed=19).to(torch.bfloat16)
    decay = 1.0 - 2.0 ** -(2 + 4 * torch.arange(nh, device=DEV, dtype=torch.float32) / nh)
    start, first = rnd(n, nh, hd, hdv, seed=20), [sum(lens[:i]) for i in range(n + 1)]

    def run(at_once):
        state, out = start.clone(), torch.full((T, nh * hdv), float("nan"), device=DEV)
        for s in range(0, n, at_once):
            e = min(n, s + at_once)
            rows = proj[first[s]:first[e]].clone()            # q, k and v are overwritten by their activation
            cu = torch.tensor([f - first[s] for f in first[s:e + 1]], dtype=torch.int32, device=DEV)
            slot = torch.arange(s, e, dtype=torch.int32, device=DEV)
            q, k, v = rows.split([nh * hd, nh * hd, nh * hdv], 1)
            api.linear_attention_chunk_bf16(q, k, v, out[first[s]:first[e]], state, cu, slot, decay, e - s, nh, hd, hdv)
        return out, state

    want = run(n)
    assert bool(want[0].isfinite().all())
    for at_once in (n // 2, 1):
        for a, b in zip(run(at_once), want):
            assert torch.equal(a, b)
