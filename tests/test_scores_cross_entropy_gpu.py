"""The loss taken straight from the class scores against the chain cast, logSoftmax, cross entropy and its
fused gradient: the same arithmetic in the same order, so the same bits."""
import pytest
import torch

from tests.parity import randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("C,X", [(1028, 3), (4100, 37), (32000, 5), (1027, 4), (1024, 4)])  # last two: the chain
@pytest.mark.parametrize("reduction", ["mean", "sum", "none"])
def test_scores_cross_entropy(dtype, C, X, reduction):
    from flashlight_b200 import _lib as L
    from flashlight_b200 import autograd as A
    from flashlight_b200 import functions as F
    from flashlight_b200.autograd import Variable
    red = {"mean": L.REDUCE_MEAN, "sum": L.REDUCE_SUM, "none": L.REDUCE_NONE}[reduction]
    x = (randn(X, C, seed=1) * 4).cuda().to(dtype)
    x[0, :-8] = float("-inf")  # a thread's first vectors, and all of most threads', weigh nothing
    t = torch.arange(X, dtype=torch.int32).cuda() * 17 % C
    t[0], t[1] = C - 3, -1  # ignored
    gl = randn(X if reduction == "none" else 1, seed=2).cuda()

    xv = Variable(x, True)
    loss = A.log_softmax_cross_entropy(xv, t, red, -1, wide=True)
    loss.backward(gl)
    y = F.log_softmax(x.float())
    want, state = F.categorical_cross_entropy(y, t, red, -1)
    grad = F.log_softmax_cross_entropy_backward(y, gl, state).to(dtype)
    assert bool(torch.isfinite(want).all())
    assert torch.equal(loss.tensor, want)
    assert xv.grad.dtype == dtype and torch.equal(xv.grad, grad)
