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
    from flashlight_b200 import functions as F
    chain = F.relu(F.add(ext.batchnorm(cl(x), w.cuda(), b.cuda(), None, None, [2], True, 0.0, 1e-5)[0], cl(s)))
    assert torch.equal(y, chain)  # the same values, so the same relu predicate, as the operators
    ga, gb = randn(*shape, seed=98).to(dtype), randn(*shape, seed=99).to(dtype)
    for second in (gb, None):
        got = ext.batchnormAddReluBackward(mask, cl(ga), None if second is None else cl(second), sm, sv, cl(x),
                                           w.cuda(), [2], True, 1e-5)
        tot = ga.double() + (0.0 if second is None else second.double())
        gz = tot * (y.detach().cpu().double() > 0)
        for g, want in zip(got, (gz,) + tuple(R.batchnorm_backward(gz, x.double(), w.double(), [2], 1e-5))):
            assert_close_scaled(g.float(), want, tol, "tail gradient")


# N, C, H, W, Cout, k, stride, pad, dilation: 1 x 1 GEMM with K and N tails; one 64-channel stage and
# one past it; fewer than 64 channels; 72 channels (the filter gradient widens); strided 1 x 1 and
# 3 x 3 (classes of backward-data); more taps than a filter-gradient tile; a pixel count past the
# patch; all tile widths
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", [(2, 8, 5, 5, 32, 1, 1, 0, 1), (3, 64, 9, 9, 256, 1, 1, 0, 1),
                                  (2, 128, 14, 14, 64, 3, 1, 1, 1), (2, 40, 13, 11, 24, 3, 1, 1, 1),
                                  (2, 72, 7, 7, 136, 3, 1, 1, 1), (2, 128, 15, 14, 192, 1, 2, 0, 1),
                                  (3, 64, 17, 18, 64, 3, 2, 1, 1), (2, 16, 12, 12, 32, 5, 1, 2, 1),
                                  (4, 64, 33, 40, 128, 3, 1, 2, 2), (40, 256, 14, 14, 256, 3, 1, 1, 1),
                                  (9, 512, 7, 7, 512, 3, 1, 1, 1)])
def test_conv_16bit_channels_last(dtype, case):
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import B200AutogradExtension
    N, C, H, W, Co, k, s, p, d = case
    ext, tol = B200AutogradExtension(math_mode=L.MATH_TF32), TOL[dtype]
    x = randn(N, C, H, W, seed=80).to(dtype)
    w = (randn(Co, C, k, k, seed=81) * (1.0 / (C * k * k) ** 0.5)).to(dtype)
    b = randn(Co, seed=82).to(dtype)
    args = (s, s, p, p, d, d, 1)
    stats = []
    y = ext.conv2d(cl(x), w.cuda(), b.cuda(), *args, stats_out=stats)
    want = R.conv2d(x.double(), w.double(), b.double(), *args)
    assert y.dtype == dtype
    assert_close_scaled(y.float(), want, tol, "conv y")
    if stats:  # statistics of the stored values, taken in the epilogue
        weight, bias = randn(Co, seed=84).abs() + 0.5, randn(Co, seed=85)
        z = ext.batchnorm(y, weight.cuda(), bias.cuda(), None, None, [2], True, 0.0, 1e-5, conv_stats=stats[0])[0]
        wz = R.batchnorm(y.cpu().double(), weight.double(), bias.double(), None, None, [2], True, 0.0, 1e-5)[0]
        assert_close_scaled(z.float(), wz, tol, "bn from conv statistics")
    gy = randn(*want.shape, seed=83).to(dtype)
    gx = ext.conv2dBackwardData(cl(gy), cl(x), w.cuda(), *args)
    assert_close_scaled(gx.float(), R.conv2d_backward_data(gy.double(), x.shape, w.double(), *args), tol, "conv dx")
    gw, gb = ext.conv2dBackwardFilterBias(cl(gy), cl(x), w.cuda(), b.cuda(), *args)
    wgw, wgb = R.conv2d_backward_filter_bias(gy.double(), x.double(), w.shape, True, *args)
    assert_close_scaled(gw.float(), wgw, tol, "conv dw")
    assert_close_scaled(gb.float(), wgb, tol, "conv db")


# channels off the vectors: a thread keeps to one channel, unless there are more channels than threads
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("shape", [(3, 30, 20, 21), (1, 5, 2, 1), (1, 2051, 1, 2), (64, 33, 30, 30)])
def test_batchnorm_element_kernels(dtype, shape):
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import B200AutogradExtension
    ext, tol = B200AutogradExtension(math_mode=L.MATH_TF32), TOL.get(dtype, 1e-4)
    ch = shape[1]
    x, gy = (randn(*shape, seed=191) * 1.7 + 0.4).to(dtype), randn(*shape, seed=192).to(dtype)
    w, b = randn(ch, seed=193).abs() + 0.5, randn(ch, seed=194)
    rm, rv = randn(ch, seed=195), randn(ch, seed=196).abs() + 0.3
    y = ext.batchnorm(cl(x), w.cuda(), b.cuda(), rm.cuda(), rv.cuda(), [2], False, 0.0, 1e-5)[0]
    want = R.batchnorm(x.double(), w.double(), b.double(), rm.double(), rv.double(), [2], False, 0.0, 1e-5)[0]
    assert_close_scaled(y.float(), want, tol, "bn evaluation")
    if x.numel() < 64 * ch:  # the gradient of two rows per channel is what their cancellation leaves
        return
    _, sm, sv = ext.batchnorm(cl(x), w.cuda(), b.cuda(), None, None, [2], True, 0.0, 1e-5)
    got = ext.batchnormBackward(cl(gy), sm, sv, cl(x), w.cuda(), [2], True, 1e-5)
    for g, v in zip(got, R.batchnorm_backward(gy.double(), x.double(), w.double(), [2], 1e-5)):
        assert_close_scaled(g.float(), v, tol, "bn gradient")
