"""The float32 tensor-core product (gemm_f32_tc) against float64, at the edges of its tiles, chunks and groups."""
import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(DEV)


def bound(x, w):
    """|error| of a sum of K terms: the pieces leave out 2^-24 of |x||w|; a chunk adds at most 8 times to a 24-bit sum that may be cut
    off (2^-23), the chunks and groups at most K / 64 + 2 times in float32 (2^-24). Each relative to sum |x w|."""
    K = x.shape[1]
    return (2.0 ** -24 + 8 * 2.0 ** -23 + (K // 64 + 3) * 2.0 ** -24) * (x.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("N,K", [(1, 4), (64, 64), (129, 68), (257, 1028), (130, 4096), (20000, 260)])
@pytest.mark.parametrize("M", [1, 16, 17, 129])
def test_plain_product(M, N, K):
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2)
    ref = x.double() @ w.double().T
    out = api.gemm_f32_tc(x, w)
    assert bool(((out.double() - ref).abs() <= bound(x, w)).all())
    # the same sums in the same order, whatever the tiles, the split and the rows beside
    for plan in [(32, 16, False), (128, 128, False)] + ([(128, 48, True)] if api.f32_groups(N, K)[0] > 1 else []):
        again = api.gemm_f32_tc(x, w, plan=plan)
        again = again.sum(torch.float32) if isinstance(again, api.Partial) else again
        assert torch.equal(again, out), plan
    assert torch.equal(api.gemm_f32_tc(x[M // 2:M // 2 + 1].clone(), w)[0], out[M // 2])
    api.gemm_tc_check()


@pytest.mark.parametrize("M,N,K", [(1, 65, 72), (40, 200, 260), (130, 64, 128)])
def test_activations(M, N, K):
    x, w = rnd(M, K, seed=3), rnd(2 * N, K, seed=4, scale=0.3)
    y, slack = x.double() @ w.double().T, bound(x, w)
    g, u = y[:, :N], y[:, N:]
    out = torch.empty(M, N, device=DEV)
    for act in ((0.0, 0.0), api.GATE_GELU, api.gate_clamped(1.5)):
        got = api.gemm_f32_tc(x, w, api.MODE_SILU, act=act)
        api.sgemm(x, w, out, api.MODE_SILU, act)
        # slopes of the gates are at most 1.2 in g; sgemm's own sums are off by K roundings
        far = (1 + K / 16) * 1.2 * (slack[:, :N] * (u.abs() + 1) + slack[:, N:] * (g.abs() + 1)) + 1e-6
        assert bool(((got - out).abs() <= far).all()), act
    z = y[:, :N]
    got = api.gemm_f32_tc(x, w[:N].contiguous(), api.MODE_XIELU, act=(0.7, 0.3))
    ref = torch.where(z > 0, 0.7 * z * z, 0.3 * (torch.expm1(z) - z)) + 0.5 * z
    assert bool(((got.double() - ref).abs() <= slack[:, :N] * (1.4 * z.abs() + 1) + 1e-6).all())


def test_values_that_are_not_finite():
    """An infinity, a NaN and a number that rounds to infinity in bfloat16 give what the FMA product gives, and only there."""
    x, w = rnd(5, 300, seed=5), rnd(200, 300, seed=6)
    clean = api.gemm_f32_tc(x, w)
    x[1, 3], x[2, 7], w[9, 4], x[3, 9] = float("inf"), float("nan"), float("-inf"), 3.4e38
    got, ref = api.gemm_f32_tc(x, w), torch.empty(5, 200, device=DEV)
    api.sgemm(x, w, ref)
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf())
    assert torch.equal(got[got.isinf()], ref[ref.isinf()])
    assert torch.allclose(got[3][ref[3].isfinite()], ref[3][ref[3].isfinite()], rtol=1e-5)
    keep = torch.ones(200, dtype=torch.bool, device=DEV)
    keep[9] = False
    assert torch.equal(got[[0, 4]][:, keep], clean[[0, 4]][:, keep])


def test_refusals():
    x, w = rnd(2, 64, seed=7), rnd(8, 64, seed=8)
    with pytest.raises(api.KernelError):
        api.gemm_f32_tc(x[:, :62].contiguous(), w[:, :62].contiguous())
    with pytest.raises(api.KernelError):
        api.gemm_f32_tc(x, rnd(8 * 64 + 1, seed=9)[1:].view(8, 64))
    with pytest.raises(api.KernelError):
        api.gemm_f32_tc(x, w, plan=(32, 16, True))


@pytest.mark.parametrize("ex,ew", [(-115, 0), (-120, 0), (-126, 0), (-130, 5), (-140, 20), (0, -125), (100, -120), (115, 2), (-60, -60)])
def test_small_and_large_numbers_keep_their_bits(ex, ew):
    """Numbers near and under 2^-126, whose second and third piece bfloat16 has no room for as they stand, and large ones: the error
    (2-norm, relative) that K = 1,024 has at any size, below sgemm's. Numbers under 2^-133 have no first piece: their largest is the
    second or the third, and of the products the one with the other operand's third, or second and third, is not taken: 2^-9 of
    such a term at most (the other operand rounded to its first 8 bits)."""
    x, w = rnd(8, 1024, seed=10, scale=2.0 ** ex), rnd(256, 1024, seed=11, scale=2.0 ** ew)
    ref = x.double() @ w.double().T
    out = torch.empty(8, 256, device=DEV)
    api.sgemm(x, w, out)
    err = [float((o.double() - ref).norm() / ref.norm()) for o in (api.gemm_f32_tc(x, w), out)]
    assert err[0] <= (2.0 ** -9 if ex < -133 else min(err[1], 3e-7)), err


@pytest.mark.parametrize("mode", [api.MODE_STORE, api.MODE_SILU, api.MODE_XIELU])
@pytest.mark.parametrize("M", [256, 257, 700])
def test_rows_in_several_launches(monkeypatch, mode, M):
    """The bits of one launch, whatever the share of rows a launch takes (here one tile of 128)."""
    x, w = rnd(M, 1028, seed=12), rnd(2 * 72, 1028, seed=13, scale=0.1)
    whole = api.gemm_f32_tc(x, w, mode, act=(0.7, 0.3) if mode == api.MODE_XIELU else (0.0, 0.0))
    monkeypatch.setattr(api, "F32_PIECES_BYTES", 6 * 1032 * 128)
    assert api.f32_rows_a_launch(M, 1028) == 128 and api.f32_rows_a_launch(128, 1028) == 128
    cut = api.gemm_f32_tc(x, w, mode, (64, 64, False), act=(0.7, 0.3) if mode == api.MODE_XIELU else (0.0, 0.0))
    assert torch.equal(cut, whole)
    api.gemm_tc_check()


@pytest.mark.parametrize("M,N,K", [(1, 512, 2560), (3, 512, 4096), (130, 512, 9728)])
def test_all_24_bits_count(M, N, K):
    """The 2-norm of the error, relative: 1.1e-7 to 1.3e-7 was measured. Operands of 16 bits (without the third pieces) leave out 2^-17 a
    term, 3.5e-6 in all, whatever the inner size; the bound lies between, and below what one float32 FMA chain over K gives."""
    x, w = rnd(M, K, seed=14), rnd(N, K, seed=15)
    ref = x.double() @ w.double().T
    out = torch.empty(M, N, device=DEV)
    api.sgemm(x, w, out)
    err = [float((o.double() - ref).norm() / ref.norm()) for o in (api.gemm_f32_tc(x, w), out)]
    assert err[0] <= 3e-7 < err[1], err


@pytest.mark.parametrize("M", [1, 3, 4, 5, 32])
@pytest.mark.parametrize("N,K", [(300, 68), (40000, 260), (700, 2564)])
def test_few_rows_give_the_bits_of_many(M, N, K):
    """Tiles of at most 32 rows (two groups of converting warps; up to 4 rows taken apart by the product itself, from any address
    that a float has) against tiles of 64: the same arithmetic, so the same bits. Tile heights that leave converting warps with
    some rows, none or all; more units than blocks; a last chunk that is not whole; a gated product."""
    x, w = rnd(M * K + 1, seed=11)[1:].view(M, K), rnd(N, K, seed=12)
    nt = (M + 15) // 16 * 16
    want = api.gemm_f32_tc(x, w, plan=(128, 64, False))
    assert bool(((want.double() - x.double() @ w.double().T).abs() <= bound(x, w)).all())
    for height in (128, 120, 65, 33, 32, 17):
        assert torch.equal(api.gemm_f32_tc(x, w, plan=(height, nt, False)), want), height
        assert torch.equal(api.gemm_f32_tc(x.clone(), w, plan=(height, nt, False)), want), height
    gated = api.gemm_f32_tc(x, w, api.MODE_SILU, plan=(64, 64, False))
    for height in (64, 60, 33, 24, 16):
        assert torch.equal(api.gemm_f32_tc(x, w, api.MODE_SILU, plan=(height, nt, False)), gated), height
    api.gemm_tc_check()


@pytest.mark.parametrize("nt", [16, 32, 48, 64, 96, 112])
def test_groups_summed_in_tensor_memory_or_in_the_output(nt):
    """A unit of several groups of K (the last one shorter): row tiles whose buffers leave tensor memory room for their sum (of these 16,
    48 and 96 rows) and ones that do not (32, 64, 112), full and ragged, against the groups left in parts and added in order. (Products
    with an activation have one group.)"""
    M, N, K = 150, 200, 2884
    groups, length = api.f32_groups(N, K)
    assert groups > 2 and groups * length > (K + 63) // 64
    x, w = rnd(M, K, seed=13), rnd(N, K, seed=14)
    parts = api.gemm_f32_tc(x, w, plan=(128, 64, True)).ws
    want = parts[0]
    for p in parts[1:]:
        want = want + p
    assert bool(((want.double() - x.double() @ w.double().T).abs() <= bound(x, w)).all())
    assert torch.equal(api.gemm_f32_tc(x, w, plan=(120, nt, False)), want)
    x[3, 5] = float("inf")
    out = api.gemm_f32_tc(x, w, plan=(128, nt, False))
    keep = torch.arange(M, device=DEV) != 3
    assert torch.equal(out[keep], want[keep]) and not bool(out[3].isfinite().any())
    api.gemm_tc_check()
