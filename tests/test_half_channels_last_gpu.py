"""f16 / bf16 channels-last tensors where the 16-byte rules of the kernels begin and end, against
fp64 results of the oracle on the rounded operands."""
import pytest
import torch

from oracle import flref as R
from tests.parity import assert_close_scaled, randn

pytestmark = pytest.mark.gpu

TOL = {torch.float16: 3e-3, torch.bfloat16: 1.6e-2}


def cl(t):
    return t.cuda().contiguous(memory_format=torch.channels_last)


# channels: one vector, a tile's tail, several CTAs; 12 is no multiple of 8 (element kernels, the
# block's tail runs as separate operators)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(2, 8, 3, 5), (3, 72, 7, 7), (2, 2056, 2, 3), (5, 64, 28, 28), (2, 12, 4, 4)])
def test_batchnorm_16bit_channels_last(dtype, shape):
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import B200AutogradExtension
    ext, tol = B200AutogradExtension(math_mode=L.MATH_TF32), TOL[dtype]
    ch = shape[1]
    x, s = (randn(*shape, seed=91) * 1.7 + 0.4).to(dtype), randn(*shape, seed=92).to(dtype)
    w, b = randn(ch, seed=93).abs() + 0.5, randn(ch, seed=94)
    rm, rv = randn(ch, seed=95), randn(ch, seed=96).abs() + 0.3
    y, sm, sv = ext.batchnorm(cl(x), w.cuda(), b.cuda(), None, None, [2], True, 0.0, 1e-5)
    wy = R.batchnorm(x.double(), w.double(), b.double(), None, None, [2], True, 0.0, 1e-5)[0]
    assert_close_scaled(y.float(), wy, tol, "bn y")
    ye = ext.batchnorm(cl(x), w.cuda(), b.cuda(), rm.cuda(), rv.cuda(), [2], False, 0.0, 1e-5, relu=True)[0]
    we = R.batchnorm(x.double(), w.double(), b.double(), rm.double(), rv.double(), [2], False, 0.0, 1e-5)[0]
    assert_close_scaled(ye.float(), torch.relu(we), tol, "bn evaluation")
    gy = randn(*shape, seed=97).to(dtype)
    got = ext.batchnormBackward(cl(gy), sm, sv, cl(x), w.cuda(), [2], True, 1e-5)
    for g, want in zip(got, R.batchnorm_backward(gy.double(), x.double(), w.double(), [2], 1e-5)):
        assert_close_scaled(g.float(), want, tol, "bn gradient")
    assert ext.batchnormAddReluSupported(cl(x), cl(s), [2]) == (ch % 8 == 0)
    if ch % 8:
        return
    y, mask, sm, sv = ext.batchnormAddRelu(cl(x), cl(s), w.cuda(), b.cuda(), None, None, [2], True, 0.0, 1e-5)
    assert_close_scaled(y.float(), torch.relu(wy + s.double()), tol, "tail y")
    ga, gb = randn(*shape, seed=98).to(dtype), randn(*shape, seed=99).to(dtype)
    for second in (gb, None):
        got = ext.batchnormAddReluBackward(mask, cl(ga), None if second is None else cl(second), sm, sv, cl(x),
                                           w.cuda(), [2], True, 1e-5)
        tot = ga.double() + (0.0 if second is None else second.double())
        gz = tot * (y.detach().cpu().double() > 0)
        for g, want in zip(got, (gz,) + tuple(R.batchnorm_backward(gz, x.double(), w.double(), [2], 1e-5))):
            assert_close_scaled(g.float(), want, tol, "tail gradient")
