"""relu(batch-norm) whose output has two consumers, or whose input takes no gradient: the gradients are
those of the operator chain (the consumers' gradients added by F.add first) bit for bit."""
import pytest
import torch

from tests.parity import randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    (3, 8, 5, 7),      # 105 rows: whole groups of rows and a remainder
    (2, 264, 3, 3),    # more vectors than a CTA has columns, fewer rows than it has lanes
    (40, 64, 29, 31),  # many splits
    (2, 12, 6, 6),     # no whole 16-bit vectors
])
@pytest.mark.parametrize("need_x", [False, True])
def test_two_consumers(shape, dtype, need_x):
    from flashlight_b200 import autograd as A
    from flashlight_b200 import functions as F
    from flashlight_b200.autograd import Variable
    cl = lambda seed, s=1.0: (randn(*shape, seed=seed) * s).cuda().to(dtype).contiguous(
        memory_format=torch.channels_last)
    C = shape[1]
    x, ga, gb = cl(1), cl(2, 0.1), cl(3, 0.1)
    w, b = (randn(C, seed=4).abs() + 0.5).cuda(), randn(C, seed=5).cuda()

    def run(second, need, retain=False):
        xv, wv, bv = Variable(x, need), Variable(w, True), Variable(b, True)
        y = A.batchnorm(xv, wv, bv, None, None, [2], True, 0.1, 1e-5, relu=True)
        if second:
            y.addGrad(ga)
            y.backward(gb, retain_graph=retain)
        else:
            y.backward(F.add(ga, gb), retain_graph=retain)
        return xv.grad, wv.grad, bv.grad, y.grad

    got, want = run(True, need_x), run(False, True)
    assert (got[0] is not None) == need_x
    if need_x:
        assert torch.equal(got[0], want[0])
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # a graph that is kept keeps the sum as the output's gradient
    kept = run(True, need_x, retain=True)
    assert torch.equal(kept[3], F.add(ga, gb)) and torch.equal(kept[1], want[1])


def block(x, g1, g2, need_x=True, hook=None):
    """Gradients of relu(batch-norm) of x and the launches they took."""
    from flashlight_b200 import _lib as L
    from flashlight_b200 import autograd as A
    from flashlight_b200.autograd import Variable
    C = x.shape[1]
    xv = Variable(x, need_x)
    wv = Variable((randn(C, seed=4).abs() + 0.5).cuda(), True)
    bv = Variable(randn(C, seed=5).cuda(), True)
    y = A.batchnorm(xv, wv, bv, None, None, [2], True, 0.1, 1e-5, relu=True)
    if hook is not None:
        y.registerGradHook(hook)
    n = L.kernel_launches()
    if g2 is not None:
        y.addGrad(g2)
    y.backward(g1)
    return [xv.grad, wv.grad, bv.grad], L.kernel_launches() - n


def test_the_sum_is_fused():
    """One launch less than the addition and the gradient of the sum; none for a gradient nobody takes."""
    from flashlight_b200 import functions as F
    cl = lambda seed: randn(3, 8, 5, 7, seed=seed).cuda().contiguous(memory_format=torch.channels_last)
    x, ga, gb = cl(1), cl(2), cl(3)
    _, two = block(x, gb, ga)
    _, one = block(x, F.add(ga, gb), None)
    _, none = block(x, gb, ga, need_x=False)
    assert (two, none) == (one, one - 1)


@pytest.mark.parametrize("kind", ["fl_order", "fl_order_odd", "layout", "hook"])
def test_other_consumers(kind):
    """Without channels last, with a gradient in another layout, with a hook: the chain's results."""
    from flashlight_b200 import functions as F
    shape = (3, 8, 5, 7) if kind == "fl_order_odd" else (4, 16, 6, 8)
    x, ga, gb = (randn(*shape, seed=s).cuda() for s in (1, 2, 3))
    seen = []
    hook = (lambda v: seen.append(v.grad.clone())) if kind == "hook" else None
    if kind in ("layout", "hook"):
        x, ga = (v.contiguous(memory_format=torch.channels_last) for v in (x, ga))
        if kind == "hook":
            gb = gb.contiguous(memory_format=torch.channels_last)
    total = F.add(ga.contiguous(), gb.contiguous())
    if kind in ("layout", "hook"):
        total = total.contiguous(memory_format=torch.channels_last)
    want, _ = block(x, total, None)
    if kind == "layout":
        with pytest.raises(ValueError):  # as the addition of the two does
            block(x, gb, ga)
    else:
        got, _ = block(x, gb, ga, hook=hook)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    if kind == "hook":
        assert len(seen) == 1 and torch.equal(seen[0], total)
    got, _ = block(x, total, None, need_x=False)
    assert got[0] is None and all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
