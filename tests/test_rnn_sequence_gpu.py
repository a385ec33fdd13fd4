"""The persistent recurrences at the edges of their tiles: hidden sizes below, at and past the unit,
k-slice and output tiles, batches of one row, past one job and past two, one and two directions."""
import pytest
import torch

from oracle import flref as R
from tests.parity import assert_close_scaled, randn

pytestmark = pytest.mark.gpu


# hidden, batch, steps, both directions
@pytest.mark.parametrize("dims", [(4, 1, 1, False), (36, 3, 5, True), (128, 48, 4, True), (132, 33, 6, False),
                                  (320, 5, 7, True), (516, 49, 4, True), (768, 32, 5, True), (900, 48, 4, False),
                                  (1000, 70, 4, True), (1024, 48, 4, True)])
@pytest.mark.parametrize("mode", [R.RNN_LSTM, R.RNN_GRU, R.RNN_TANH])
def test_recurrence_edges(dims, mode):
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import AutogradPayload, B200AutogradExtension, RNNGradData
    H, B, T, both = dims
    dirs, I, layers = 2 if both else 1, 24, 1
    ext = B200AutogradExtension(math_mode=L.MATH_TF32)
    w = randn(R.rnn_num_params(I, H, layers, mode, both), seed=40) * (0.5 / H ** 0.5)
    x, gy = randn(T, B, I, seed=41), randn(T, B, dirs * H, seed=44)
    hx = randn(dirs, B, H, seed=42) * 0.5
    cx = randn(dirs, B, H, seed=43) * 0.5 if mode == R.RNN_LSTM else None
    dev = lambda t: None if t is None else t.cuda()
    f64 = lambda t: None if t is None else t.double()
    payload = AutogradPayload()
    before = L.kernel_launches()
    y, hy, cy = ext.rnn(x.cuda(), hx.cuda(), dev(cx), w.cuda(), H, layers, mode, both, 0.0, payload)
    assert L.kernel_launches() - before <= 12 * dirs
    wy, why, wcy = R.rnn(x.double(), hx.double(), f64(cx), w.double(), H, layers, mode, both)
    assert_close_scaled(y, wy, 5e-3, "y")
    assert_close_scaled(hy, why, 5e-3, "hy")
    got = ext.rnnBackward(x.cuda(), hx.cuda(), dev(cx), w.cuda(), RNNGradData(gy.cuda(), None, None), y, layers,
                          H, mode, both, 0.0, payload)
    want = R.rnn_backward(x.double(), hx.double(), f64(cx), w.double(), H, layers, mode, both, gy.double(), None, None)
    for g, v, what in zip(got, want, ("dx", "dhx", "dcx", "dw")):
        if v is not None and (what != "dcx" or mode == R.RNN_LSTM):
            assert_close_scaled(g, v, 5e-3, what)


# few rows: warps of the kernels that have no tile, row or pair of their own; with gradients of the
# final states
@pytest.mark.parametrize("dims", [(36, 2, 1200), (132, 5, 700), (320, 5, 700)])
@pytest.mark.parametrize("mode", [R.RNN_LSTM, R.RNN_GRU, R.RNN_TANH])
def test_recurrence_many_steps(dims, mode):
    """Hundreds of steps in as many launches as one: no kernel per step, forward or backward."""
    from flashlight_b200 import _lib as L
    from flashlight_b200.extension import AutogradPayload, B200AutogradExtension, RNNGradData
    H, B, T = dims
    I = 24
    ext = B200AutogradExtension(math_mode=L.MATH_TF32)
    w = randn(R.rnn_num_params(I, H, 1, mode, False), seed=50) * (0.5 / H ** 0.5)
    hx = randn(1, B, H, seed=51) * 0.5
    cx = randn(1, B, H, seed=52) * 0.5 if mode == R.RNN_LSTM else None
    dhy, dcy = randn(1, B, H, seed=53), randn(1, B, H, seed=54) if mode == R.RNN_LSTM else None
    dev = lambda t: None if t is None else t.cuda()
    f64 = lambda t: None if t is None else t.double()
    counts = []
    for steps in (1, T):
        x, gy = randn(steps, B, I, seed=55), randn(steps, B, H, seed=56)
        payload = AutogradPayload()
        before = L.kernel_launches()
        y, hy, _ = ext.rnn(x.cuda(), hx.cuda(), dev(cx), w.cuda(), H, 1, mode, False, 0.0, payload)
        middle = L.kernel_launches()
        got = ext.rnnBackward(x.cuda(), hx.cuda(), dev(cx), w.cuda(), RNNGradData(gy.cuda(), dhy.cuda(), dev(dcy)), y,
                              1, H, mode, False, 0.0, payload)
        counts.append((middle - before, L.kernel_launches() - middle))
    torch.cuda.synchronize()
    L.check(L.lib.flb200_tc_poll_status(torch.cuda.current_stream().cuda_stream))
    assert counts[1][0] <= counts[0][0] + 2 and counts[1][1] <= counts[0][1] + 6, counts
    wy, why, _ = R.rnn(x.double(), hx.double(), f64(cx), w.double(), H, 1, mode, False)
    assert_close_scaled(y, wy, 5e-3, "y")
    assert_close_scaled(hy, why, 5e-3, "hy")
    want = R.rnn_backward(x.double(), hx.double(), f64(cx), w.double(), H, 1, mode, False, gy.double(), dhy.double(),
                          f64(dcy))
    for g, v, what in zip(got, want, ("dx", "dhx", "dcx", "dw")):
        if v is not None and (what != "dcx" or mode == R.RNN_LSTM):
            assert_close_scaled(g, v, 5e-3, what)
