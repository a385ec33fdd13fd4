"""The fp32-FMA contraction kernel at the edges of its tiles, splits and operand loaders, against
fp64 products and the CPU oracle (strict bound)."""
import pytest
import torch

from oracle import flref as R
from tests.parity import STRICT_TOL, assert_close, randn

pytestmark = pytest.mark.gpu


# (m, n, k): one element; below, at and past the 32 / 64 / 128 tiles; K below a stage, with a tail,
# split over a cluster of CTAs, and over clusters and scratch
@pytest.mark.parametrize("mnk", [(1, 1, 1), (31, 33, 15), (64, 64, 16), (129, 65, 36), (1, 1024, 3136),
                                 (130, 260, 20), (32, 28, 20000), (3000, 30, 72), (257, 128, 516)])
@pytest.mark.parametrize("a_k", [True, False])
@pytest.mark.parametrize("b_k", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_matmul_strict_loaders(mnk, a_k, b_k, offset):
    """a_k / b_k: k contiguous (else the rows); offset 1: base not 16-byte aligned, so that the
    element loaders read what the vector loaders would."""
    from flashlight_b200 import _lib as L
    from flashlight_b200 import functions as F
    m, n, k = mnk
    a, b = randn(m, k, seed=1), randn(k, n, seed=2)
    store = lambda t: torch.cat([torch.zeros(offset), t.reshape(-1)]).cuda()[offset:]
    ad, bd = store(a if a_k else a.t().contiguous()), store(b.t().contiguous() if b_k else b)
    c = F.matmul(ad, bd, m=m, n=n, k=k, a_strides=(k, 1) if a_k else (1, m),
                 b_strides=(1, k) if b_k else (n, 1), math_mode=L.MATH_STRICT_F32)
    assert_close(c, a.double() @ b.double(), STRICT_TOL, f"matmul {mnk}")


# results stored along their rows (four at a time where m and the strides allow it), with and without
# a split of K, and added to
@pytest.mark.parametrize("mnk", [(64, 33, 40), (36, 5, 2100), (130, 70, 100), (33, 20, 3000), (1, 40, 17), (128, 64, 20000)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_matmul_strict_transposed_result(mnk, beta):
    from flashlight_b200 import _lib as L
    from flashlight_b200 import functions as F
    m, n, k = mnk
    a, b, c = randn(m, k, seed=14), randn(k, n, seed=15), randn(n, m, seed=16)
    got = c.cuda()
    F.matmul(a.cuda(), b.cuda(), got, m=m, n=n, k=k, a_strides=(k, 1), b_strides=(n, 1), c_strides=(1, m), beta=beta,
             math_mode=L.MATH_STRICT_F32)
    assert_close(got, (a.double() @ b.double()).t() + beta * c.double(), STRICT_TOL, f"matmul {mnk}")


# batches that fill grid z with and without a split of K beside them (65535 is the most)
@pytest.mark.parametrize("zmnk", [(8192, 4, 4, 512), (9000, 5, 3, 1024), (40000, 1, 2, 128), (65535, 1, 1, 256)])
def test_matmul_strict_many_batches(zmnk):
    from flashlight_b200 import _lib as L
    from flashlight_b200 import functions as F
    z, m, n, k = zmnk
    a, b = randn(z, m, k, seed=8), randn(z, k, n, seed=9)
    c = F.matmul(a.cuda(), b.cuda(), m=m, n=n, k=k, batch=z, a_strides=(k, 1), b_strides=(n, 1),
                 batch_strides=(m * k, k * n, 0), math_mode=L.MATH_STRICT_F32)
    assert_close(c, a.double() @ b.double(), STRICT_TOL, f"batched matmul {zmnk}")


def test_matmul_strict_k_past_32_bits():
    """2^31 + 37 products of 2 and 0.5 (strides of 0 read one element of each): all partial sums are
    whole numbers below 2^24 or sums of a few of them."""
    from flashlight_b200 import _lib as L
    from flashlight_b200 import functions as F
    k = 2 ** 31 + 37
    c = F.matmul(torch.full((4,), 2.0).cuda(), torch.full((4,), 0.5).cuda(), m=1, n=1, k=k, a_strides=(1, 0),
                 b_strides=(0, 1), math_mode=L.MATH_STRICT_F32)
    assert abs(float(c) / k - 1.0) <= 1e-6


def test_conv_strict_filter_gradient_of_many_pixels():
    """More output pixels than one sum takes: 1025 images of 2^20, every product 0.5."""
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import B200AutogradExtension
    ext = B200AutogradExtension(math_mode=L.MATH_STRICT_F32)
    x, gy = torch.ones(1025, 1, 1024, 1024, device="cuda"), torch.full((1025, 1, 1024, 1024), 0.5, device="cuda")
    gw, _ = ext.conv2dBackwardFilterBias(gy, x, torch.ones(1, 1, 1, 1, device="cuda"), None, 1, 1, 0, 0, 1, 1, 1)
    assert float(gw) == 1025 * 2.0 ** 19


# N, C, H, W, Cout, kH, kW, stride, pad, groups: element loaders; repacked filter and channels-last
# copy; channels not a multiple of 4; groups; a filter of many taps; stride with empty classes;
# filters whose repacking needs more than the default shared memory, and more than there is; more
# images than a grid's third extent; a channel per group; long sums of few pixels, in whole quads and
# not; one output channel
@pytest.mark.parametrize("case", [(2, 1, 9, 9, 8, 5, 5, 1, 2, 1), (16, 32, 14, 14, 64, 5, 5, 1, 2, 1),
                                  (8, 36, 13, 15, 44, 3, 3, 2, 1, 1), (16, 30, 14, 14, 66, 3, 3, 1, 1, 1),
                                  (16, 64, 12, 12, 64, 3, 3, 1, 1, 4), (2, 16, 1, 70, 24, 1, 13, 1, 0, 1),
                                  (40, 64, 17, 17, 256, 1, 1, 2, 0, 1), (8, 64, 30, 30, 64, 1, 1, 1, 0, 1),
                                  (2, 8, 1, 900, 16, 1, 401, 1, 0, 1), (2, 4, 1, 2500, 8, 1, 2001, 1, 0, 1),
                                  (70000, 8, 1, 6, 16, 1, 3, 1, 0, 1), (3, 24, 9, 11, 24, 3, 3, 1, 1, 24),
                                  (5, 6, 17, 19, 6, 5, 5, 2, 2, 6), (1, 256, 4, 4, 64, 3, 3, 1, 1, 1),
                                  (1, 130, 5, 3, 70, 3, 3, 1, 1, 1), (2, 20, 33, 31, 1, 3, 3, 1, 1, 1)])
@pytest.mark.parametrize("channels_last", [False, True])
def test_conv_strict_routes(case, channels_last):
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import B200AutogradExtension
    N, C, H, W, Co, kH, kW, s, p, groups = case
    if channels_last and C == 1:
        pytest.skip("one channel has one layout")
    ext = B200AutogradExtension(math_mode=L.MATH_STRICT_F32)
    x = randn(N, C, H, W, seed=3)
    w = randn(Co, C // groups, kH, kW, seed=4) * (1.0 / (C // groups * kH * kW) ** 0.5)
    b = randn(Co, seed=5)
    args = (s, s, p, p, 1, 1, groups)
    put = lambda t: t.cuda().contiguous(memory_format=torch.channels_last) if channels_last else t.cuda()
    y = ext.conv2d(put(x), w.cuda(), b.cuda(), *args)
    want = R.conv2d(x.double(), w.double(), b.double(), *args)
    assert_close(y, want, STRICT_TOL, "conv forward")
    gy = randn(*want.shape, seed=6)
    gx = ext.conv2dBackwardData(put(gy), put(x), w.cuda(), *args)
    assert_close(gx, R.conv2d_backward_data(gy.double(), x.shape, w.double(), *args), STRICT_TOL, "conv dx")
    gw, gb = ext.conv2dBackwardFilterBias(put(gy), put(x), w.cuda(), b.cuda(), *args)
    wgw, wgb = R.conv2d_backward_filter_bias(gy.double(), x.double(), w.shape, True, *args)
    assert_close(gw, wgw, STRICT_TOL, "conv dw")
    assert_close(gb, wgb, STRICT_TOL, "conv db")


def test_conv_strict_groups_launch_once():
    """The filters of all groups are repacked by one launch, and the results are those of the groups
    one by one."""
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import B200AutogradExtension
    ext = B200AutogradExtension(math_mode=L.MATH_STRICT_F32)
    N, C, H, groups = 8, 256, 20, 64
    args = (1, 1, 1, 1, 1, 1, groups)
    x, w = randn(N, C, H, H, seed=21), randn(C, C // groups, 3, 3, seed=22) / 6
    gy = randn(N, C, H, H, seed=23)
    before = L.kernel_launches()
    y = ext.conv2d(x.cuda(), w.cuda(), None, *args)
    gx = ext.conv2dBackwardData(gy.cuda(), x.cuda(), w.cuda(), *args)
    assert L.kernel_launches() - before <= 8
    assert_close(y, R.conv2d(x.double(), w.double(), None, *args), STRICT_TOL, "conv forward")
    assert_close(gx, R.conv2d_backward_data(gy.double(), x.shape, w.double(), *args), STRICT_TOL, "conv dx")
