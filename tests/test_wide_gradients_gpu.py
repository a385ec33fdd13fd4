"""fp32 gradients of bf16 contractions (flb200_matmul_wide) at tile edges and split sums, and the
gradients of a packed projection whether its parts arrive in one buffer or not."""
import pytest
import torch

from tests.parity import assert_close, randn

pytestmark = pytest.mark.gpu


# m, n, k: single tiles with tails, pairs, few tiles of a long K (split, reduced by a second kernel;
# many splits of a small result, which share a CTA there)
@pytest.mark.parametrize("mnk", [(8, 8, 8), (72, 40, 200), (512, 1536, 600), (768, 768, 4096), (136, 264, 8200), (8, 32, 20000),
                                 (72, 40, 12544)])
def test_matmul_wide(mnk):
    from flashlight_b200 import functions as F
    m, n, k = mnk
    a, b = randn(k, m, seed=1).bfloat16(), randn(k, n, seed=2).bfloat16()
    got = F.matmul(a.cuda(), b.cuda(), m=m, n=n, k=k, a_strides=(1, m), b_strides=(n, 1), wide=True)
    assert got.dtype == torch.float32
    assert_close(got, a.double().t() @ b.double(), 1e-4, "wide product")


@pytest.mark.parametrize("one_buffer", [True, False])
def test_unbind_gradients(one_buffer):
    from flashlight_b200 import autograd as A
    x = A.Variable(randn(6, 12, seed=3).cuda(), True)
    parts = A.unbind(x, lambda t: t.reshape(6, 3, 4).permute(1, 0, 2).contiguous(),
                     lambda g: g.permute(1, 0, 2).reshape(6, 12), 3)
    g = randn(3, 6, 4, seed=4).cuda()
    for i in (1, 0, 2):
        parts[i].grad_func(parts[i].inputs, g[i] if one_buffer else g[i].clone())
    assert torch.equal(x.grad, g.permute(1, 0, 2).reshape(6, 12))


def test_wide_and_plain_contributions_add_up():
    from flashlight_b200 import autograd as A
    w = A.Variable(randn(4, 4, seed=5).bfloat16().cuda(), True)
    a, b = randn(4, 4, seed=6).cuda(), randn(4, 4, seed=7).bfloat16().cuda()
    w.addGrad(a)
    w.addGrad(b)
    assert torch.equal(w.grad, a + b.float())


def test_add_grad_refuses_gradients_of_unrelated_types():
    """Two types meet in one gradient only where one is the tensor's and the other fp32."""
    from flashlight_b200.autograd import Variable
    for own, first, second in ((torch.bfloat16, torch.bfloat16, torch.float16),
                               (torch.float16, torch.float32, torch.bfloat16),
                               (torch.float32, torch.float32, torch.bfloat16)):
        v = Variable(torch.zeros(4, dtype=own, device="cuda"), True)
        v.addGrad(torch.ones(4, dtype=first, device="cuda"))
        with pytest.raises(ValueError):
            v.addGrad(torch.ones(4, dtype=second, device="cuda"))
