"""Fused attention on the packed projection at the edges of its 128-position blocks, against the fp64
chain on the rounded operands."""
import pytest
import torch

from tests.parity import assert_close_scaled, randn

pytestmark = pytest.mark.gpu


# below, at and past one block; several blocks with a tail
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 40, 3), (1, 128, 2), (3, 129, 2), (2, 200, 8), (1, 512, 4), (2, 700, 1)])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_packed(shape, causal):
    from flashlight_b200 import functions as F
    B, T, h = shape
    scale = 0.125
    qkv = (randn(B * T, 3 * h * 64, seed=1) * 1.5).bfloat16()
    go = randn(B * T, h * 64, seed=2).bfloat16()
    out, lse = F.attention_packed(qkv.cuda(), B, T, h, scale, causal)
    g = F.attention_packed_backward(qkv.cuda(), out, go.cuda(), lse, B, T, h, scale, causal)

    ref = qkv.double().requires_grad_(True)
    q, k, v = ref.reshape(B, T, 3, h, 64).permute(2, 0, 3, 1, 4)
    s = scale * q @ k.transpose(-1, -2)
    if causal:
        s = s.masked_fill(torch.ones(T, T).triu(1).bool(), float("-inf"))
    want = (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3).reshape(B * T, h * 64)
    want.backward(go.double())
    assert_close_scaled(out.float(), want.detach(), 1.2e-2, "attention output")
    assert_close_scaled(lse.reshape(B, h, T), torch.logsumexp(s.detach(), -1), 1e-3, "attention lse")
    assert_close_scaled(g.float(), ref.grad, 1.6e-2, "attention gradient")


@pytest.mark.parametrize("causal", [True, False])
def test_attention_packed_infinite_scores(causal):
    """Keys of score -inf weigh nothing, even where they fill the first blocks of a row; rows that see
    no other keys are NaN, as softmax makes them."""
    from flashlight_b200 import functions as F
    B, T, h, lead = 1, 400, 2, 260
    qkv = randn(B * T, 3, h, 64, seed=3).bfloat16()
    qkv[:, 0, :, 0] = 1.0
    qkv[:lead, 1, :, 0] = float("-inf")
    out, lse = F.attention_packed(qkv.reshape(B * T, 3 * h * 64).cuda(), B, T, h, 0.125, causal)
    q, k, v = qkv.double().reshape(B, T, 3, h, 64).permute(2, 0, 3, 1, 4)
    s = 0.125 * q @ k.transpose(-1, -2)
    if causal:
        s = s.masked_fill(torch.ones(T, T).triu(1).bool(), float("-inf"))
    want = (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3).reshape(B * T, h * 64)
    first = lead if causal else 0
    assert out[:first].isnan().all()
    assert_close_scaled(out[first:].float(), want[first:], 1.2e-2, "attention output")
    assert_close_scaled(lse.reshape(B, h, T)[:, :, first:], torch.logsumexp(s, -1)[:, :, first:], 1e-3, "attention lse")


def test_attention_packed_large_scores():
    """The softmax of a single key is 1 and its lse the score, whatever the score: 0.125 * 64 * 110 * 111 = 97680,
    exact in every step, and nothing between the score and its exponential may round by the score's size."""
    from flashlight_b200 import functions as F
    B, T, h = 3, 1, 2
    qkv = randn(B, 3, h, 64, seed=4).bfloat16()
    qkv[:, 0], qkv[:, 1] = 110.0, 111.0
    qkv = qkv.reshape(B, 3 * h * 64).cuda()
    go = randn(B, h * 64, seed=5).bfloat16().cuda()
    out, lse = F.attention_packed(qkv, B, T, h, 0.125, True)
    g = F.attention_packed_backward(qkv, out, go, lse, B, T, h, 0.125, True)
    assert torch.equal(lse, torch.full_like(lse, 97680.0))
    assert torch.equal(out, qkv.reshape(B, 3, h * 64)[:, 2])
    assert torch.equal(g.reshape(B, 3, h * 64)[:, 2], go)


def test_attention_packed_declines_what_it_is_not_built_for():
    from flashlight_b200 import functions as F
    assert F.attention_packed(randn(8, 96, seed=1).bfloat16().cuda(), 1, 8, 1, 1.0, True) is None
    assert F.attention_packed(randn(8, 192, seed=1).cuda(), 1, 8, 1, 1.0, True) is None
