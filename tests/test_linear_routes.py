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
