"""Host-side mirror of fl::AutogradExtension over the flb200 C ABI.

`B200AutogradExtension` has the nine operator methods of the reference
interface (flashlight/fl/autograd/tensor/AutogradExtension.h:46-180) with the
same names, argument order and argument meaning; the C++ class of the same
name (csrc/fl/B200AutogradExtension.cpp) is the one a Flashlight build links.
This Python class exists so that the parity tests and the benchmark drive the
very same C entry points from device buffers that torch owns.

Tensor convention: a torch CUDA tensor of shape (d_{k-1}, ..., d_0), contiguous,
stands for the fl tensor [d_0, ..., d_{k-1}] — fl is column-major, so the bytes
are identical.  An image batch fl [W,H,C,N] is torch (N,C,H,W); `axes` and every
other dimension index are fl indices (0 = fastest).  An absent (empty) fl tensor
is None.  Out-parameters of the reference (saveMean, saveVar) are returned.

Channels-last storage: an image batch may also be a torch tensor in
torch.channels_last memory format (same logical (N,C,H,W) indexing, bytes laid out
[N][H][W][C]).  conv2d, pool2d and batchnorm over the channel axis take such tensors
as they are (FLB200_LAYOUT_NHWC), return their results in the same format, and the
element-wise functions work on any two tensors of equal layout, so a network whose
first convolution is called with channels_last_out=True keeps every activation in
the layout the tensor-core convolutions read natively and no layout copy is made.
"""
from __future__ import annotations

import ctypes as C
import os
from dataclasses import dataclass, field
from typing import Optional, Sequence

import torch

from . import _lib as L
from ._native import native as N

_DTYPES = {torch.float32: L.F32, torch.float16: L.F16, torch.bfloat16: L.BF16}


def dtype_code(t: torch.Tensor) -> int:
    try:
        return _DTYPES[t.dtype]
    except KeyError:
        raise ValueError(f"dtype {t.dtype} is not supported by the B200 autograd extension") from None


def ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    if t is None:
        return None
    if not t.is_cuda:
        raise ValueError("the B200 autograd extension needs device (CUDA) tensors")
    if not is_dense(t):
        # fl::DevicePtr also refuses non-contiguous tensors (flashlight/fl/common/DevicePtr.cpp:16-33)
        raise ValueError("can't get device pointer of non-contiguous tensor")
    return t.data_ptr()


def is_channels_last(t: Optional[torch.Tensor]) -> bool:
    """True for a 4-d tensor stored [N][H][W][C] whose bytes differ from the [N][C][H][W] order
    (with one channel or 1x1 planes the two orders coincide and the tensor counts as the latter)."""
    return (t is not None and t.dim() == 4 and not t.is_contiguous()
            and t.is_contiguous(memory_format=torch.channels_last))


def is_dense(t: torch.Tensor) -> bool:
    """Contiguous in fl's order or in channels-last order."""
    return t.is_contiguous() or is_channels_last(t)


def same_layout(a: torch.Tensor, b: torch.Tensor) -> bool:
    return a.shape == b.shape and is_channels_last(a) == is_channels_last(b)


def stream_handle() -> int:
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


_mask_offset = 0


def bernoulli_mask(shape, keep_prob: float, device, dtype=torch.float32, seed: Optional[int] = None,
                   offset: Optional[int] = None) -> torch.Tensor:
    """A 0 / 1 mask with P(1) = keep_prob from the library's counter-based generator
    (flb200_bernoulli_mask).  Without an explicit (seed, offset) the stream continues from the
    last call, seeded by torch's CUDA generator seed."""
    global _mask_offset
    out = torch.empty(shape, dtype=dtype, device=device)
    if seed is None:
        seed = torch.cuda.initial_seed() & ((1 << 64) - 1)
    if offset is None:
        offset = _mask_offset
        _mask_offset += (out.numel() + 3) // 4
    N.bernoulli_mask(out, keep_prob, seed, offset)
    return out


def workspace(nbytes: int, like: torch.Tensor) -> Optional[torch.Tensor]:
    if nbytes <= 0:
        return None
    return torch.empty(int(nbytes), dtype=torch.uint8, device=like.device)


class _ConvLayoutCache:
    """flb200_conv2d_cache plus the tensors behind it.  A copy is only trusted for the very
    tensor it was made from: same storage address and same version counter."""

    def __init__(self, x_bytes: int, gy_bytes: int, like: torch.Tensor):
        self.c = L.Conv2dCache()
        self.x_bytes, self.gy_bytes, self.device = int(x_bytes), int(gy_bytes), like.device
        self.x_buf = self.gy_buf = None
        self.x_key = self.gy_key = None

    @staticmethod
    def _key(t: torch.Tensor):
        return (t.data_ptr(), t._version, tuple(t.shape))

    def bind_x(self, x: torch.Tensor) -> None:
        if self.x_bytes and self.x_buf is None:
            self.x_buf = torch.empty(self.x_bytes, dtype=torch.uint8, device=self.device)
            self.c.x_cl, self.c.x_cl_bytes = self.x_buf.data_ptr(), self.x_bytes
        self.c.x_cl_valid = 0
        self.x_key = self._key(x)

    def check_x(self, x: torch.Tensor) -> None:
        if self.x_key != self._key(x):
            self.bind_x(x)

    def bind_gy(self, gy: torch.Tensor) -> None:
        if self.gy_bytes and self.gy_buf is None:
            self.gy_buf = torch.empty(self.gy_bytes, dtype=torch.uint8, device=self.device)
            self.c.gy_cl, self.c.gy_cl_bytes = self.gy_buf.data_ptr(), self.gy_bytes
        self.c.gy_cl_valid = 0
        self.gy_key = self._key(gy)

    def check_gy(self, gy: torch.Tensor) -> None:
        if self.gy_key != self._key(gy):
            self.c.gy_cl_valid = 0

    def release_gy(self) -> None:
        """The copy of grad_y is dead after backward-filter; give its memory back."""
        self.gy_buf = None
        self.gy_key = None
        self.c.gy_cl, self.c.gy_cl_bytes, self.c.gy_cl_valid = None, 0, 0

    def address(self) -> int:
        return C.addressof(self.c)


class AutogradPayload:
    """detail::AutogradPayload: a nullable slot that forward fills and backward reads."""

    def __init__(self):
        self.data = None


@dataclass
class RNNGradData:
    """detail::RNNGradData (flashlight/fl/autograd/tensor/AutogradOps.h:356-360)."""
    dy: Optional[torch.Tensor] = None
    dhy: Optional[torch.Tensor] = None
    dcy: Optional[torch.Tensor] = None


@dataclass
class _PoolPayload:
    argmax: torch.Tensor


@dataclass
class _RnnPayload:
    reserve: torch.Tensor
    dropout_mask: Optional[torch.Tensor] = None


def _shape4(t: torch.Tensor):
    """torch (.., N, C, H, W) with missing leading dims = 1 -> (W, H, C, N)."""
    if t.dim() > 4:
        raise ValueError("expected at most 4 dimensions")
    s = (1,) * (4 - t.dim()) + tuple(t.shape)
    return s[3], s[2], s[1], s[0]


def default_math_mode() -> int:
    """FLB200_TF32=1 selects the tensor-core (TF32) kernels, FLB200_TF32=0 strict fp32."""
    if os.environ.get("FLB200_MATH", "") in L.MATH_BY_NAME:  # strict | tf32 | f32x3
        return L.MATH_BY_NAME[os.environ["FLB200_MATH"]]
    return L.MATH_TF32 if os.environ.get("FLB200_TF32", "0") not in ("0", "", "false") else L.MATH_STRICT_F32


class DynamicBenchmark:
    """fl::DynamicBenchmark with DynamicBenchmarkOptions<KernelMode>
    (flashlight/fl/common/DynamicBenchmark.h:60-263): while the class-wide benchmark mode is on,
    audit() times the call under the current option (device synchronised on both sides, as
    fl::sync() does there); every option is timed `count` times, then the fastest is kept."""

    _benchmark_mode = False

    def __init__(self, options: Sequence[int], count: int = 10):
        if not options:
            raise ValueError("Options must be passed vector with at least one element")
        self.options, self.count = list(options), int(count)
        self.reset()

    def reset(self) -> None:
        self.times = [0.0] * len(self.options)
        self.counts = [0] * len(self.options)
        self._complete, self._idx = False, 0

    @classmethod
    def setBenchmarkMode(cls, mode: bool) -> None:
        cls._benchmark_mode = bool(mode)

    @classmethod
    def getBenchmarkMode(cls) -> bool:
        return cls._benchmark_mode

    def _update(self) -> None:
        if self._complete:
            return
        for i, c in enumerate(self.counts):
            if c < self.count:
                self._idx = i
                return
        self._complete = True
        self._idx = min(range(len(self.options)), key=lambda i: self.times[i])

    def currentOption(self) -> int:
        self._update()
        return self.options[self._idx]

    def timingsComplete(self) -> bool:
        self._update()
        return self._complete

    def audit(self, function, incrementCount: bool = True):
        if self.timingsComplete() or not self._benchmark_mode:
            return function()
        import time
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        out = function()
        torch.cuda.synchronize()
        self.times[self._idx] += time.perf_counter() - t0
        if incrementCount:
            self.counts[self._idx] += 1
        return out


class B200AutogradExtension:
    """sm_100a implementation of the Flashlight autograd extension interface."""

    def __init__(self, math_mode: Optional[int] = None, cache_layouts: Optional[bool] = None):
        self.math_mode = default_math_mode() if math_mode is None else math_mode
        # Keep the channels-last copies of x and grad_y in the payload of each conv2d call
        # site (forward -> backward-filter, backward-data -> backward-filter).  Costs one
        # extra copy of x per convolution that uses one; FLB200_CACHE_LAYOUTS=0 turns it off.
        if cache_layouts is None:
            cache_layouts = os.environ.get("FLB200_CACHE_LAYOUTS", "1") != "0"
        self.cache_layouts = cache_layouts

    # ------------------------------------------------------------ registry
    def isDataTypeSupported(self, dtype) -> bool:
        """TensorExtension::isDataTypeSupported (flashlight/fl/tensor/TensorExtension.h:34)."""
        return dtype in _DTYPES

    def createBenchmarkOptions(self) -> DynamicBenchmark:
        """Options of a Conv2D module's run-time autotune: fp32 FMA, TF32 ("allow conversion")
        and the three-pass split, tried in that order (the counterpart of
        backend/cudnn/CudnnAutogradExtension.cpp:16-25)."""
        return DynamicBenchmark([L.MATH_STRICT_F32, L.MATH_TF32, L.MATH_F32X3])

    def _audited(self, bench: Optional[DynamicBenchmark], run):
        """run(math_mode) under the benchmark's current option while tuning is on, else in the
        configured mode (backend/cudnn/Conv2D.cpp:401-405,466-535)."""
        if bench is None or not DynamicBenchmark.getBenchmarkMode():
            return run(self.math_mode)
        mode = bench.currentOption()
        return bench.audit(lambda: run(mode))

    # --------------------------------------------------------------- conv2d
    def _conv_desc(self, input, weights, sx, sy, px, py, dx, dy, groups,
                   output_channels_last: Optional[bool] = None) -> L.Conv2dDesc:
        """output_channels_last: layout of y / grad_y; None = that of the input."""
        if input.dtype not in _DTYPES or weights.dtype != input.dtype:
            raise ValueError("conv2d: input and weights must share one of f32 / f16 / bf16")
        x_cl = is_channels_last(input)
        y_cl = x_cl if output_channels_last is None else bool(output_channels_last)
        if x_cl and not y_cl:
            raise ValueError("conv2d: a channels-last input gives a channels-last output")
        layout = L.LAYOUT_NHWC if x_cl else (L.LAYOUT_NCHW_IN_NHWC_OUT if y_cl else L.LAYOUT_NCHW)
        W, H, Cin, N = _shape4(input)
        kW, kH, Cg, Cout = _shape4(weights)
        if Cg * groups != Cin:
            raise ValueError(
                f"conv2d: weight has {Cg} input channels per group x {groups} groups, input has {Cin}")
        return L.Conv2dDesc(W, H, Cin, N, kW, kH, Cout, sx, sy, px, py, dx, dy, groups,
                            dtype_code(input), self.math_mode, layout)

    def _conv_cache(self, payload, input, weights, args, y_cl, mode) -> Optional["_ConvLayoutCache"]:
        """The layout cache kept in the payload of one conv2d call site (None when the route
        keeps no channels-last copies, when there is no payload, or when caching is off)."""
        if payload is None or not self.cache_layouts:
            return None
        if isinstance(payload.data, _ConvLayoutCache):
            return payload.data
        if mode == L.MATH_STRICT_F32:  # the fp32 kernels read either layout in place
            return None
        nx, ng = N.conv2d_cache_bytes(input, weights, *args, y_cl, mode)
        if nx == 0 and ng == 0:
            return None
        payload.data = _ConvLayoutCache(nx, ng, input)
        return payload.data

    def conv2d(self, input, weights, bias, sx, sy, px, py, dx, dy, groups, payload=None,
               channels_last_out: Optional[bool] = None, stats_out: Optional[list] = None):
        """channels_last_out=True on an input in fl's order: the output (and from there the whole
        network) is stored channels-last; a channels-last input always gives such an output.
        stats_out: a list that receives (matrix, groups) — the batch-norm statistics of the result,
        taken in the convolution's epilogue (flb200_conv2d_forward_stats), for
        batchnorm(..., conv_stats=...) — where the library can do that; it stays empty otherwise."""
        args = (sx, sy, px, py, dx, dy, groups)
        y_cl = -1 if channels_last_out is None else int(bool(channels_last_out))
        cache = self._conv_cache(payload, input, weights, args, y_cl, self.math_mode)
        if cache is not None:
            cache.bind_x(input)
        out, stats, stat_groups = N.conv2d(input, weights, bias, *args, y_cl, self.math_mode,
                                           cache.address() if cache is not None else None,
                                           stats_out is not None)
        if stats is not None:
            stats_out.append((stats, stat_groups))
        return out

    def conv2dBackwardData(self, gradOutput, input, weight, sx, sy, px, py, dx, dy, groups,
                           dataGradBenchmark=None, payload=None):
        args = (sx, sy, px, py, dx, dy, groups)

        def run(mode):
            cache = self._conv_cache(payload, input, weight, args, self._y_cl(gradOutput, input), mode)
            if cache is not None:
                cache.bind_gy(gradOutput)
            return N.conv2d_backward_data(gradOutput, input, weight, *args, mode,
                                          cache.address() if cache is not None else None)

        return self._audited(dataGradBenchmark, run)

    @staticmethod
    def _y_cl(gradOutput, input) -> int:
        return int(is_channels_last(gradOutput) or is_channels_last(input))

    def conv2dBackwardFilterBias(self, gradOutput, input, weights, bias, sx, sy, px, py, dx, dy,
                                 groups, filterBench=None, biasBench=None, autogradPayload=None):
        args = (sx, sy, px, py, dx, dy, groups)

        def run(mode):
            cache = self._conv_cache(autogradPayload, input, weights, args,
                                     self._y_cl(gradOutput, input), mode)
            if cache is not None:
                cache.check_x(input)
                cache.check_gy(gradOutput)
            grads = N.conv2d_backward_filter_bias(gradOutput, input, weights, bias, *args, mode,
                                                  cache.address() if cache is not None else None)
            if cache is not None:
                cache.release_gy()
            return grads

        # the bias gradient is a reduction: nothing to choose
        return self._audited(filterBench, run)

    # --------------------------------------------------------------- pool2d
    def pool2d(self, input, wx, wy, sx, sy, px, py, mode, payload=None):
        out, argmax = N.pool2d(input, wx, wy, sx, sy, px, py, int(mode), payload is not None)
        if argmax is not None:
            payload.data = _PoolPayload(argmax)
        return out

    def pool2dBackward(self, gradOutput, input, poolOutput, wx, wy, sx, sy, px, py, mode,
                       payload=None):
        argmax = payload.data.argmax if payload is not None and payload.data is not None else None
        return N.pool2d_backward(gradOutput, input, argmax, wx, wy, sx, sy, px, py, int(mode))

    # ------------------------------------------------------------ batchnorm
    def batchnorm(self, input, weight, bias, runningMean, runningVar, axes, train, momentum,
                  epsilon, payload=None, relu=False, conv_stats=None):
        """Returns (output, saveMean, saveVar).  saveVar holds 1/sqrt(var + eps).
        runningMean / runningVar are updated in place when given.  relu=True returns
        relu(batchnorm(x)) from the same two passes (pair it with batchnormReluBackward)."""
        stats, groups = conv_stats if conv_stats is not None else (None, 0)
        return N.batchnorm(input, weight, bias, runningMean, runningVar, axes, train, momentum, epsilon,
                           relu, stats, groups)

    def batchnormBackward(self, gradOutput, saveMean, saveVar, input, weight, axes, train, epsilon,
                          payload=None):
        if not train:
            # cudnn/BatchNorm.cpp:196-199
            raise RuntimeError("can't compute batchnorm grad when train was not specified")
        return N.batchnorm_backward(gradOutput, saveMean, saveVar, input, weight, None, axes, False)

    def batchnormAddReluSupported(self, input, addend, axes) -> bool:
        return N.batchnorm_add_relu_supported(input, addend, axes)

    def batchnormAddRelu(self, input, addend, weight, bias, runningMean, runningVar, axes, train,
                         momentum, epsilon, payload=None, conv_stats=None):
        """relu(batchnorm(input) + addend) with the predicate's bit mask: returns
        (output, mask, saveMean, saveVar).  Check batchnormAddReluSupported first."""
        stats, groups = conv_stats if conv_stats is not None else (None, 0)
        return N.batchnorm_add_relu(input, addend, weight, bias, runningMean, runningVar, axes, train,
                                    momentum, epsilon, stats, groups)

    def batchnormAddReluBackward(self, mask, gradA, gradB, saveMean, saveVar, input, weight, axes,
                                 train, epsilon, payload=None):
        """Gradient of batchnormAddRelu: returns (gradSum, gradInput, gradWeight, gradBias) where
        gradSum = mask ? gradA + gradB : 0 is the addend's gradient (gradB may be None)."""
        if not train:
            raise RuntimeError("can't compute batchnorm grad when train was not specified")
        return N.batchnorm_add_relu_backward(mask, gradA, gradB, saveMean, saveVar, input, weight, axes)

    @staticmethod
    def batchnormSumSupported(input, gradA, gradB, axes) -> bool:
        """Whether batchnormReluBackward adds two gradients itself."""
        return (list(axes) == [2] and is_channels_last(input) and gradA.dtype == input.dtype and
                gradB.dtype == input.dtype and same_layout(gradA, input) and same_layout(gradB, input) and
                input.shape[1] * input.element_size() % 16 == 0 and
                not (input.data_ptr() | gradA.data_ptr() | gradB.data_ptr()) & 15)

    def batchnormReluBackward(self, gradOutput, saveMean, saveVar, input, weight, bias, axes, train,
                              epsilon, payload=None, gradOutput2=None, needInput=True):
        """Gradient of relu(batchnorm(x)) given the gradient of the relu output: the predicate
        is rebuilt from the input, so no output tensor or mask is needed.  gradOutput2: a second
        consumer's gradient, added where the first is read (check batchnormSumSupported);
        needInput=False: None in the place of the input's gradient."""
        if not train:
            raise RuntimeError("can't compute batchnorm grad when train was not specified")
        if gradOutput2 is not None or not needInput:
            return N.batchnorm_relu_backward_sum(gradOutput, gradOutput2, saveMean, saveVar, input, weight,
                                                 bias, axes, needInput)
        return N.batchnorm_backward(gradOutput, saveMean, saveVar, input, weight, bias, axes, True)

    # ------------------------------------------------------------------ rnn
    def _rnn_desc(self, input, hiddenSize, numLayers, mode, bidirectional) -> L.RnnDesc:
        if input.dtype != torch.float32:
            raise ValueError("rnn: only f32 tensors are supported")
        if input.dim() != 3:
            raise ValueError("rnn: input must be [inputSize, batch, seqLen]")
        T, B, I = input.shape
        return L.RnnDesc(I, hiddenSize, numLayers, B, T, int(mode), 1 if bidirectional else 0, L.F32,
                         self.math_mode)

    def rnn(self, input, hiddenState, cellState, weights, hiddenSize, numLayers, mode,
            bidirectional, dropout, payload=None, dropout_mask=None):
        """Returns (y, hy, cy); cy is None unless mode is LSTM.  dropout > 0 applies inter-layer
        dropout (backend/cudnn/RNN.cpp:83-85): the mask [numLayers - 1, T, B, H * dirs] of 0 / 1
        is drawn here (`bernoulli_mask`, a counter-based generator seeded from torch's) unless the
        caller supplies one, and is kept in the payload for the backward pass."""
        if not 0.0 <= dropout < 1.0:
            raise ValueError("rnn: dropout must be in [0, 1)")
        d = self._rnn_desc(input, hiddenSize, numLayers, mode, bidirectional)
        nparams = L.lib.flb200_rnn_num_params(C.byref(d))
        if weights.numel() != nparams:
            raise ValueError(f"rnn: weights has {weights.numel()} elements, expected {nparams}")
        dirs = 2 if bidirectional else 1
        T, B, _ = input.shape
        dev = input.device
        use_dropout = (dropout > 0.0 or dropout_mask is not None) and numLayers > 1
        mask = None
        if use_dropout:
            shape = (numLayers - 1, T, B, hiddenSize * dirs)
            if dropout_mask is not None:
                mask = dropout_mask
                if tuple(mask.shape) != shape or mask.dtype != torch.float32 or not mask.is_contiguous():
                    raise ValueError(f"rnn: dropout mask must be a dense float32 tensor {shape}")
            else:
                mask = bernoulli_mask(shape, 1.0 - dropout, dev)
        y = torch.empty((T, B, hiddenSize * dirs), dtype=torch.float32, device=dev)
        hy = torch.empty((numLayers * dirs, B, hiddenSize), dtype=torch.float32, device=dev)
        cy = torch.empty_like(hy) if int(mode) == L.RNN_LSTM else None
        reserve = None
        rbytes = 0
        if payload is not None:
            rbytes = (L.lib.flb200_rnn_reserve_bytes_dropout(C.byref(d)) if use_dropout
                      else L.lib.flb200_rnn_reserve_bytes(C.byref(d)))
            reserve = workspace(rbytes, input)
            payload.data = _RnnPayload(reserve)
            payload.data.dropout_mask = mask
        wbytes = L.lib.flb200_rnn_workspace_bytes(C.byref(d), 0 if reserve is not None else 2)
        if reserve is None and use_dropout:
            wbytes += L.lib.flb200_rnn_reserve_bytes_dropout(C.byref(d))
        ws = workspace(wbytes, input)
        if use_dropout:
            L.check(L.lib.flb200_rnn_forward_dropout(
                C.byref(d), ptr(input), ptr(hiddenState), ptr(cellState), ptr(weights), ptr(mask),
                float(dropout), ptr(y), ptr(hy), ptr(cy), ptr(reserve), rbytes, ptr(ws), wbytes,
                stream_handle()))
        else:
            L.check(L.lib.flb200_rnn_forward(
                C.byref(d), ptr(input), ptr(hiddenState), ptr(cellState), ptr(weights), ptr(y),
                ptr(hy), ptr(cy), ptr(reserve), rbytes, ptr(ws), wbytes, stream_handle()))
        return y, hy, cy

    def rnnBackward(self, input, hiddenState, cellState, weights, gradData: RNNGradData, output,
                    numLayers, hiddenSize, mode, bidirectional, dropProb, payload=None):
        """Returns (dx, dhx, dcx, dw)."""
        if payload is None or payload.data is None:
            raise ValueError("B200AutogradExtension::rnnBackward given null detail::AutogradPayload")
        d = self._rnn_desc(input, hiddenSize, numLayers, mode, bidirectional)
        reserve = payload.data.reserve
        mask = getattr(payload.data, "dropout_mask", None)
        dx = torch.empty_like(input)
        dirs = 2 if bidirectional else 1
        B = input.shape[1]
        dhx = torch.empty((numLayers * dirs, B, hiddenSize), dtype=torch.float32, device=input.device)
        dcx = torch.empty_like(dhx) if int(mode) == L.RNN_LSTM else None
        dw = torch.empty_like(weights)
        wbytes = L.lib.flb200_rnn_workspace_bytes(C.byref(d), 1)
        ws = workspace(wbytes, input)
        if mask is not None:
            L.check(L.lib.flb200_rnn_backward_dropout(
                C.byref(d), ptr(input), ptr(hiddenState), ptr(cellState), ptr(weights), ptr(mask),
                float(dropProb), ptr(output), ptr(gradData.dy), ptr(gradData.dhy),
                ptr(gradData.dcy), ptr(dx), ptr(dhx), ptr(dcx), ptr(dw), ptr(reserve),
                reserve.numel(), ptr(ws), wbytes, stream_handle()))
            return dx, dhx, dcx, dw
        L.check(L.lib.flb200_rnn_backward(
            C.byref(d), ptr(input), ptr(hiddenState), ptr(cellState), ptr(weights), ptr(output),
            ptr(gradData.dy), ptr(gradData.dhy), ptr(gradData.dcy), ptr(dx), ptr(dhx), ptr(dcx),
            ptr(dw), ptr(reserve), reserve.numel(), ptr(ws), wbytes, stream_handle()))
        return dx, dhx, dcx, dw
