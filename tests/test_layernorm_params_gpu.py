"""Layer normalisation takes its parameters in whole vectors where their address allows: the same bits as
from an address that does not, in every width a warp's row can have."""
import pytest
import torch

from tests.parity import randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("features", [8, 248, 384, 768, 776, 2048])
def test_layernorm_parameters_at_any_address(dtype, features):
    from flashlight_b200 import functions as F
    features = min(features, 32 * 8 * (16 // torch.empty(0, dtype=dtype).element_size()))
    x, dy = randn(37, features, seed=1).cuda().to(dtype), randn(37, features, seed=2).cuda().to(dtype)
    w, b = randn(features, seed=3).cuda(), randn(features, seed=4).cuda()
    odd = lambda t: torch.cat([t.new_zeros(1), t])[1:]
    assert odd(w).data_ptr() % 16 == 4
    want = F.layernorm(x, w, b, 1e-5)
    got = F.layernorm(x, odd(w), odd(b), 1e-5)
    assert all(torch.equal(p, q) for p, q in zip(want, got))
    gw = F.layernorm_backward(dy, want[1], w, want[2], True, True)
    go = F.layernorm_backward(dy, want[1], odd(w), want[2], True, True)
    assert all(torch.equal(p, q) for p, q in zip(gw, go))
