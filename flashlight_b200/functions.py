"""Fused forward / gradient kernels for the tensor-op chains of Flashlight's
autograd functions that are NOT behind fl::AutogradExtension
(flashlight/fl/autograd/Functions.cpp): relu, gelu, tanh, dropout, linear,
logSoftmax, categoricalCrossEntropy, bias tile/sumAs and gradient accumulation.

Tensor convention as in extension.py: torch shape = reversed fl shape, None for
an absent tensor.  Every function launches flb200 kernels through the C ABI on
torch's current stream; nothing is computed by torch itself.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib as L
from ._native import native as N
from .extension import default_math_mode, dtype_code, ptr, stream_handle, workspace

# operator numbers of native.unary / native.binary
_RELU, _GELU, _TANH, _ADD = range(4)


def relu(x):
    """fl::relu = max(x, 0) (Functions.cpp:1787-1789)."""
    return N.unary(_RELU, x)


def relu_backward(x, grad_y):
    """(x > 0) * dy (Functions.cpp:329-338).  Passing the output y instead of x gives the same mask."""
    return N.binary(_RELU, x, grad_y, None)


def relu_with_mask(x):
    """relu that also returns the predicate x > 0 packed 8 elements per byte."""
    return N.relu_mask(x, None)


def relu_backward_mask(mask, grad_y):
    return N.relu_mask_backward(mask, grad_y, None)


def add_relu_with_mask(a, b):
    """relu(a + b) in one pass, with the predicate (a + b) > 0 packed 8 elements per byte."""
    return N.relu_mask(a, b)


def relu_backward_mask_sum(mask, grad_a, grad_b):
    """mask ? grad_a + grad_b : 0 — the relu gradient of an output with two consumers."""
    return N.relu_mask_backward(mask, grad_a, grad_b)


def gelu(x):
    """fl::gelu, tanh form (Functions.cpp:1791-1796)."""
    return N.unary(_GELU, x)


def gelu_backward(x, grad_y):
    return N.binary(_GELU, x, grad_y, None)


def tanh(x):
    return N.unary(_TANH, x)


def tanh_backward(y, grad_y):
    """(1 - y^2) * dy from the saved output (Functions.cpp:454-463)."""
    return N.binary(_TANH, y, grad_y, None)


def dropout_apply(x, mask, p: float):
    """x * mask / (1 - p): forward with x, gradient with dy (Functions.cpp:1777-1785)."""
    return N.dropout_apply(x, mask, 1.0 / (1.0 - p))


def add(a, b, out=None):
    """Gradient fan-in accumulation of Variable::addGrad (Variable.cpp:205-211)."""
    return N.binary(_ADD, a, b, out)


_ASTYPE_CODES = {torch.float32: L.F32, torch.float16: L.F16, torch.bfloat16: L.BF16}


def astype(x, dtype):
    """x.to(dtype) between float32 and float16 / bfloat16 through flb200_astype (contiguous
    tensors); None for anything else (the caller then lets torch convert)."""
    src, dst = _ASTYPE_CODES.get(x.dtype), _ASTYPE_CODES.get(dtype)
    if src is None or dst is None or not x.is_cuda or not x.is_contiguous():
        return None
    if src != dst and L.F32 not in (src, dst):
        return None
    return N.astype(x, dst)


def reorder(x, shape, perm):
    """`x.reshape(shape).permute(perm).contiguous()` through flb200_reorder: `shape` has up to five
    extents, `perm` keeps the last one in place (the contiguous run).  Returns the permuted,
    contiguous tensor; None where the kernel's 16-byte rules do not hold (the caller then uses
    the torch copy)."""
    return N.reorder(x, tuple(shape), tuple(perm))


def channel_sum(x, outer: int, channels: int, inner: int):
    """out[c] = sum_{o,i} x[o][c][i] (conv bias gradient; detail::sumAs onto a bias)."""
    return N.channel_sum(x, outer, channels, inner)


def channel_bias_add(x, bias, outer: int, channels: int, inner: int, out=None):
    return N.channel_bias_add(x, bias, outer, channels, inner, out)


def layernorm_affine(xhat, weight, bias):
    """y = xhat * weight + bias over rows of features (the affine part of fl::LayerNorm);
    weight / bias are fp32 parameter vectors of the last dimension's length."""
    feat = xhat.shape[-1]
    xh = xhat.contiguous()
    y = torch.empty_like(xh)
    L.check(L.lib.flb200_layernorm_affine_forward(ptr(xh), ptr(weight), ptr(bias), ptr(y),
                                                  xh.numel() // feat, feat, dtype_code(xh),
                                                  stream_handle()))
    return y


def layernorm(x, weight, bias, eps: float):
    """fl::LayerNorm over the last dimension in one kernel: returns (y, xhat, invstd)."""
    return N.layernorm(x.contiguous(), weight, bias, eps)


def layernorm_backward(grad_y, xhat, weight, invstd, need_input_grad=True, need_param_grads=True):
    """Returns (grad_x, grad_weight, grad_bias); the parameter gradients are fp32."""
    return N.layernorm_backward(grad_y.contiguous(), xhat, weight, invstd, need_input_grad,
                                need_param_grads)


def layernorm_affine_backward(grad_y, xhat, weight, need_input_grad=True, need_param_grads=True):
    """Returns (grad_xhat, grad_weight, grad_bias); the parameter gradients are fp32."""
    feat = xhat.shape[-1]
    rows = xhat.numel() // feat
    gy, xh = grad_y.contiguous(), xhat.contiguous()
    gx = torch.empty_like(xh) if need_input_grad else None
    gw = gb = None
    if need_param_grads:
        gw = torch.empty(feat, dtype=torch.float32, device=xh.device)
        gb = torch.empty(feat, dtype=torch.float32, device=xh.device)
    nbytes = L.lib.flb200_layernorm_affine_workspace_bytes(rows, feat)
    ws = workspace(nbytes, xh)
    L.check(L.lib.flb200_layernorm_affine_backward(ptr(gy), ptr(xh), ptr(weight), ptr(gx), ptr(gw),
                                                   ptr(gb), rows, feat, dtype_code(xh), ptr(ws),
                                                   nbytes, stream_handle()))
    return gx, gw, gb


# ------------------------------------------------------------------ linear
def linear(x, weight, bias=None, math_mode: Optional[int] = None):
    """fl::linear forward (Functions.cpp:1255-1275): fl weight [O,I] (torch (I,O)), x fl [I,...]."""
    return N.linear(x, weight, bias, default_math_mode() if math_mode is None else math_mode)


def linear_bias_act(x, weight, bias, gelu: bool = False, math_mode: Optional[int] = None):
    """y = act(x W + bias) in one kernel (flb200_linear_bias_act_forward): returns (y, pre) with
    pre = x W + bias when gelu is on (None otherwise), or None where the tensor-core path does
    not cover the call and the operators have to run one by one."""
    return N.linear_bias_act(x, weight, bias, gelu,
                             default_math_mode() if math_mode is None else math_mode)


def linear_backward(x, weight, grad_y, has_bias: bool, need_input_grad=True, need_weight_grad=True,
                    math_mode: Optional[int] = None):
    """The linear gradFunc (Functions.cpp:1277-1305): returns (grad_x, grad_weight, grad_bias)."""
    return N.linear_backward(x, weight, grad_y, has_bias, need_input_grad, need_weight_grad,
                             default_math_mode() if math_mode is None else math_mode)


def matmul(a, b, c=None, *, m, n, k, a_strides, b_strides, c_strides=None, batch=1,
           batch_strides=(0, 0, 0), alpha=1.0, beta=0.0, math_mode: Optional[int] = None,
           wide: bool = False):
    """C[m,n] = alpha * A(m,k) B(k,n) + beta * C on strided row-major views (flb200_matmul); wide: an
    f32 result whatever the operands' type."""
    c_row, c_col = c_strides if c is not None else (0, 0)
    return N.matmul(a, b, c, m, n, k, a_strides[0], a_strides[1], b_strides[0], b_strides[1], c_row,
                    c_col, batch, batch_strides[0], batch_strides[1], batch_strides[2], alpha, beta,
                    default_math_mode() if math_mode is None else math_mode, wide)


# --------------------------------------------------- logSoftmax and CE loss
def log_softmax(x):
    """fl::logSoftmax(input, 0) (Functions.cpp:1044-1060): over fl dim 0 = torch's last dim."""
    return N.log_softmax(x)


def log_softmax_backward(y, grad_y):
    return N.log_softmax_backward(y, grad_y)


class CrossEntropyState:
    """What the categoricalCrossEntropy gradFunc captures: targets, kept-target count, mode."""

    def __init__(self, targets, count, reduction, ignore_index):
        self.targets, self.count, self.reduction, self.ignore_index = (
            targets, count, reduction, ignore_index)


def categorical_cross_entropy(logp, targets, reduction: int = L.REDUCE_MEAN, ignore_index: int = -1):
    """fl::categoricalCrossEntropy (Functions.cpp:1078-1154).  Returns (loss, state).
    Raises ValueError when a target lies outside [0, C) and is not ignore_index."""
    if targets.numel() * logp.shape[-1] != logp.numel():
        raise ValueError("dimension mismatch in categorical cross entropy")
    if targets.dtype != torch.int32:
        targets = targets.to(torch.int32)
    loss, meta = N.cce_forward(logp, targets, reduction, ignore_index)
    return loss, CrossEntropyState(targets, meta, reduction, ignore_index)


def check_targets(state: CrossEntropyState) -> None:
    """Host-side read of the bad-target flag (one synchronising copy); the
    reference performs the same check eagerly (Functions.cpp:1100-1107)."""
    if int(state.count[1].item()) != 0:
        raise ValueError("target contains elements out of valid range [0, num_categories) "
                         "in categorical cross entropy")


def categorical_cross_entropy_backward(grad_loss, state: CrossEntropyState, C_classes: int, like):
    return N.cce_backward(grad_loss, state.targets, state.count, C_classes, state.reduction,
                          state.ignore_index, like)


def log_softmax_cross_entropy_backward(y, grad_loss, state: CrossEntropyState):
    """Gradient of categoricalCrossEntropy(logSoftmax(x)) w.r.t. x in one pass."""
    return N.log_softmax_cce_backward(y, grad_loss, state.targets, state.count, state.reduction,
                                      state.ignore_index)


def scores_cross_entropy(x, targets, reduction: int = L.REDUCE_MEAN, ignore_index: int = -1):
    """categoricalCrossEntropy(logSoftmax(x)) in fp32 arithmetic whatever the type of the scores, without
    the log-probabilities in memory.  Returns (loss, state, lse), or None where the library has no kernel
    for the rows (see flb200_scores_cce_forward)."""
    if targets.numel() * x.shape[-1] != x.numel():
        raise ValueError("dimension mismatch in categorical cross entropy")
    if targets.dtype != torch.int32:
        targets = targets.to(torch.int32)
    out = N.scores_cce_forward(x, targets, reduction, ignore_index)
    if out is None:
        return None
    return out[0], CrossEntropyState(targets, out[1], reduction, ignore_index), out[2]


def scores_cross_entropy_backward(x, lse, grad_loss, state: CrossEntropyState):
    return N.scores_cce_backward(x, lse, grad_loss, state.targets, state.count, state.reduction,
                                 state.ignore_index)


# ------------------------------------------------------------------ embedding
def embedding(table, ids):
    """fl::embedding forward: rows of `table` (vocab, dim) picked by `ids` (any shape)."""
    return N.embedding(table, ids.contiguous())


def embedding_backward(grad_out, ids, vocab: int):
    """Gradient of the table (f32, (vocab, dim)), summed in position order without atomics."""
    return N.embedding_backward(grad_out.contiguous(), ids.contiguous(), vocab)


# ------------------------------------------------------------------ attention softmax
def softmax(x, scale: float = 1.0, causal_period: int = 0):
    """softmax over the last dim of scale * x, optionally with the causal mask of stacked
    (period x cols) score matrices folded in."""
    return N.softmax(x, scale, causal_period, False)


def softmax_lse(x, scale: float = 1.0, causal_period: int = 0):
    """softmax as above plus lse[row] = log sum exp(scale * x[row]) (fp32), the only thing the
    fused attention gradient keeps of the scores."""
    return N.softmax(x, scale, causal_period, True)


def attention_backward_supported(q) -> bool:
    return bool(L.lib.flb200_attention_backward_supported(q.shape[1], q.shape[2], dtype_code(q)))


def attention_backward(q, k, v, o, grad_o, lse, scale: float, causal: bool):
    """(dq, dk, dv) of o = softmax(scale * q k^T [+ causal mask]) v in one flash-style kernel;
    q, k, v, o, grad_o (batch * heads, T, head dim) dense, lse (batch * heads * T,) fp32."""
    return N.attention_backward(q, k, v, o, grad_o, lse, scale, causal)


def attention_packed(qkv, B: int, T: int, heads: int, scale: float, causal: bool):
    """softmax(scale * q k^T [+ causal mask]) v from the packed projection (B * T, 3 * heads * head
    dim) in one kernel: returns (out (B * T, heads * head dim), lse), or None where it is not built
    (bf16 tensors of head dimension 64 only)."""
    return N.attention_packed(qkv, B, T, heads, scale, causal)


def attention_packed_backward(qkv, out, grad_out, lse, B: int, T: int, heads: int, scale: float, causal: bool):
    """Gradient of attention_packed with respect to the packed projection."""
    return N.attention_packed_backward(qkv, out, grad_out, lse, B, T, heads, scale, causal)


def softmax_backward(y, grad_y, scale: float = 1.0):
    return N.softmax_backward(y, grad_y, scale)
