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


def both(x, t):
    """(loss, gradient, state) from the scores, and of the chain."""
    from flashlight_b200 import _lib as L
    from flashlight_b200 import functions as F
    red, gl = L.REDUCE_NONE, torch.ones(x.shape[0], device="cuda")
    got = F.scores_cross_entropy(x, t, red, -1)
    assert got is not None
    loss, state, lse = got
    g = F.scores_cross_entropy_backward(x, lse, gl, state)
    y = F.log_softmax(x.float())
    want, wstate = F.categorical_cross_entropy(y, t, red, -1)
    wg = F.log_softmax_cross_entropy_backward(y, gl, wstate).to(x.dtype)
    return (loss, g, state), (want, wg, wstate)


def same(a, b):
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(), b.nan_to_num())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_special_scores(dtype):
    """Rows of -inf alone, with a NaN, with +inf, of the type's lowest value, and targets out of range."""
    from flashlight_b200 import _lib as L
    from flashlight_b200 import autograd as A
    from flashlight_b200 import functions as F
    from flashlight_b200.autograd import Variable
    C, X = 2052, 7
    x = randn(X, C, seed=3).cuda().to(dtype)
    x[0] = float("-inf")
    x[1, 1500] = float("nan")
    x[2, 7] = float("inf")
    x[3] = torch.finfo(dtype).min
    x[4, :-1], x[4, -1] = float("-inf"), float("nan")
    t = torch.tensor([3, 4, 5, 6, 7, C, 8], dtype=torch.int32, device="cuda")  # row 5: out of range
    (loss, g, state), (want, wg, wstate) = both(x, t)
    assert same(loss, want) and same(g, wg)
    assert bool(torch.isnan(loss[[0, 1, 2, 4]]).all()) and bool(torch.isfinite(loss[[3, 5, 6]]).all())
    assert int(state.count[1]) == int(wstate.count[1]) == 1
    with pytest.raises(ValueError):
        F.check_targets(state)
    # the operator of the tape takes this path: the rows' lse, the loss, its sum, the gradient
    n = L.kernel_launches()
    xv = Variable(x, True)
    A.log_softmax_cross_entropy(xv, t, L.REDUCE_NONE, -1, wide=True).backward()
    assert L.kernel_launches() - n == 4 and same(xv.grad, wg)


def test_rows_without_a_kernel():
    """Where the rows are too many, not aligned or of other lengths the chain takes over."""
    from flashlight_b200 import autograd as A
    from flashlight_b200 import functions as F
    from flashlight_b200.autograd import Variable
    C = 1028
    wide = randn(65536, C, seed=4).cuda()
    flat = randn(3 * C + 1, seed=5).cuda()
    for x in (wide, flat[1:].view(3, C), randn(3, 1024, seed=6).cuda(), randn(3, 1030, seed=7).cuda()):
        t = torch.arange(x.shape[0], dtype=torch.int32, device="cuda") % x.shape[1]
        if x is wide:
            assert F.scores_cross_entropy(x[:65535], t[:65535]) is not None
        assert F.scores_cross_entropy(x, t) is None
        xv = Variable(x, True)
        loss = A.log_softmax_cross_entropy(xv, t, wide=True)
        loss.backward()
        y = F.log_softmax(x)
        want, state = F.categorical_cross_entropy(y, t)
        assert torch.equal(loss.tensor, want)
        gl = torch.ones(1, device="cuda")
        assert torch.equal(xv.grad, F.log_softmax_cross_entropy_backward(y, gl, state))
