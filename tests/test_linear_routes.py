"""What the linear part makes of calls at the edge of a route (no GPU: none of these comes to a launch)."""
import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api
from dryft_challenge_htn_2026_b200.parts.linear import SILU, STORE, STORE_F32, XIELU, linear


@pytest.mark.parametrize("K", [256, 300, 4096])
@pytest.mark.parametrize("mode", [STORE, STORE_F32, SILU, XIELU])
@pytest.mark.parametrize("allow_partial", [False, True])
def test_no_rows_in_float32_give_no_rows(monkeypatch, K, mode, allow_partial):
    """From an inner size of 256 on, the tensor-core product: an empty result, as sgemm gives below."""
    monkeypatch.setattr(api, "_need", lambda *a: None)
    out = linear(torch.empty(0, K), torch.empty(40, K), mode, allow_partial=allow_partial and mode in (STORE, STORE_F32))
    assert isinstance(out, torch.Tensor) and out.dtype == torch.float32 and tuple(out.shape) == (0, 20 if mode == SILU else 40)


class _Launches:
    """A library that notes the arguments of its launches."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, [a.value if hasattr(a, "value") else a for a in args]))
            return 0
        return call


@pytest.fixture
def launches(monkeypatch):
    lib, sizes, empty = _Launches(), [], torch.empty

    def noted(*shape, **kw):
        out = empty(*shape, **kw)
        sizes.append(out.numel() * out.element_size())
        return out

    monkeypatch.setattr(api, "_need", lambda *a: None)
    monkeypatch.setattr(api, "_lib", lambda source, defines=None: lib)
    monkeypatch.setattr(api, "_stream", lambda: None)
    monkeypatch.setattr(api, "_tc_err", torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(torch, "empty", noted)
    lib.sizes = sizes
    return lib


@pytest.mark.parametrize("M,N,K", [(1, 64, 256), (544, 96, 9728), (9000, 32, 9728), (30000, 8, 4100), (4609, 24, 9732)])
@pytest.mark.parametrize("partial", [False, True])
def test_scratch_of_the_float32_product_is_bounded(launches, M, N, K, partial):
    """However many rows: at most 256 MB of pieces, every row in one launch, in order, the pieces' buffer the same for all."""
    x = torch.zeros(1).expand(M, K)          # no memory of its own: nothing is read here
    out = linear(x, torch.zeros(1).expand(N, K), STORE, allow_partial=partial)
    assert max(launches.sizes) <= max(256 << 20, 4 * M * N * (api.f32_groups(N, K)[0] if isinstance(out, api.Partial) else 1))
    at = 0
    for name, a in launches.calls:
        rows = a[4]
        assert name == "dk_gemm_f32_tc" and a[0] == x.data_ptr() + 4 * at * K and a[3] == launches.calls[0][1][3]
        assert 6 * rows * ((K + 7) // 8 * 8) <= 256 << 20 and 3 * rows <= 1 << 30
        if not isinstance(out, api.Partial):
            assert a[2] == out.data_ptr() + 4 * at * N and tuple(out.shape) == (M, N)
        else:
            assert len(launches.calls) == 1 and rows == M
        at += rows
    assert at == M


@pytest.mark.parametrize("n,nh,nkv,hd,pages", [(1, 32, 8, 128, 4), (0, 32, 8, 128, 4), (64, 32, 8, 128, 1024), (16, 128, 8, 64, 16384),
                                               (70000, 2, 2, 64, 1)])
def test_scratch_of_the_float32_decode_attention_is_bounded(launches, n, nh, nkv, hd, pages):
    """However many sequences and pages: 256 MB of pages' results, or one sequence's; every sequence in one launch, in order."""
    q, store, pos = torch.zeros(1).expand(n, nh * hd), torch.zeros(1), torch.zeros(1, dtype=torch.int32)
    table = pos.expand(n, pages)
    api.attention_decode_f32(q, q, store, store, pos, table, nh, nkv, hd, 0, 0.1)
    one = 4 * nh * pages * (hd + 2)
    assert max(launches.sizes) <= max(256 << 20, one)
    at = 0
    for name, a in launches.calls:
        assert name == "dk_attn_f32_decode" and a[0] == a[1] == q.data_ptr() + 4 * at * nh * hd
        assert a[4] == pos.data_ptr() + 4 * at and a[5] == table.data_ptr() + 4 * at * pages
        assert a[7] <= 65535 and one * a[7] <= max(256 << 20, one)
        assert a[13] - a[12] == 4 * min(n, launches.sizes[0] // one) * nh * pages * hd
        at += a[7]
    assert at == n


LAYER = [(6144, 2560, STORE, True), (2560, 4096, STORE, True), (9728, 2560, SILU, False), (2560, 9728, STORE, True),
         (151936, 2560, STORE_F32, False)]


@pytest.mark.parametrize("M", [1, 8, 16])
def test_a_product_of_a_shape_seen_before_is_not_planned_again(launches, monkeypatch, M):
    """Every plainly launched step of few rows pays for its plans on the host, layer by layer."""
    made = [0]
    real = {name: getattr(api, name) for name in ("_stream_smem", "_few_units_plan")}

    def counted(name):
        def fn(*a):
            made[0] += 1
            return real[name](*a)
        return fn

    for name in real:
        monkeypatch.setattr(api, name, counted(name))
    w = torch.zeros(1, dtype=torch.bfloat16)
    products = [(torch.zeros(M, K, dtype=torch.bfloat16), w.expand(2 * N if mode == SILU else N, K), mode, partial)
                for N, K, mode, partial in LAYER]
    for x, weights, mode, partial in products:
        linear(x, weights, mode, partial)
    made[0] = 0
    for x, weights, mode, partial in products:
        linear(x, weights, mode, partial)
    streamed = sum(name == "dk_gemv_stream" for name, _ in launches.calls) // 2
    assert made[0] == streamed                          # gemv_stream's look at the plan it is given, and nothing else


def test_one_slice_goes_on_in_float32_exactly_where_it_takes_the_place_of_several():
    for M in (1, 8):
        for N in (72, 2560, 4096, 5120):
            for K in (304, 2560, 2896, 4096, 5120, 5568, 9728):
                for mode in (STORE, STORE_F32):
                    for partial in (False, True):
                        plan, one = api.few_rows_plan(M, N, K, mode, partial)
                        several = plan is not None and plan[0] == 1 and (api.stream_plan(M, N, K, mode, partial) or (1,))[0] > 1
                        assert one == several, (M, N, K, mode, partial)
