"""What the performance of this framework is measured on: whole passes through its public entry
points (workloads.py, nn.py, autograd.py), as a training loop or an inference server makes them.

  mnist   the README convnet                      training step, or scores in evaluation mode
  resnet  ResNet of bottleneck blocks             scores in evaluation mode
  block   one residual bottleneck block           training pass, or its output in evaluation mode
  asr     time-convolution acoustic model         training step, or frame scores
  rnn     fl::rnn, LSTM or GRU                    outputs, and with train their gradients
  lm      decoder-only Transformer language model training step, or next-token scores

A training pass is zeroGrad, forward, loss (or a given gradient of the output) and backward; its
outputs are the loss (or the output), every parameter's gradient and the batch-norm running
statistics it updates.  math: "strict" is the library's default (fp32 arithmetic), "tf32" its
tensor-core mode; bf16 and f16 operands run in "tf32".

Deep networks of relus are measured forward only, and trained block by block: in TF32 two correct
implementations round differently, about one relu in a thousand turns the other way in every layer,
and after tens of layers the gradients of a random network have little in common.
"""
import math

import torch

from flashlight_b200 import _lib as L
from flashlight_b200 import autograd as A
from flashlight_b200 import nn, workloads
from flashlight_b200.autograd import Variable
from flashlight_b200.extension import bernoulli_mask

MATH = {"strict": L.MATH_STRICT_F32, "tf32": L.MATH_TF32}
CELLS = {"lstm": (L.RNN_LSTM, 4), "gru": (L.RNN_GRU, 3)}
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def listed():
    return [
        # one digit scored by a server: a dozen launches, latency only; the default arithmetic
        dict(name="mnist_infer_b1", kind="mnist", train=False, batch=1, math="strict"),
        # the first benchmark configuration: the README convnet, batch 64, fp32
        dict(name="mnist_train_b64", kind="mnist", train=True, batch=64, math="strict"),
        # a small batch of photographs scored by a server
        dict(name="resnet50_infer_b8", kind="resnet", train=False, batch=8, size=224, blocks="3463",
             math="tf32"),
        # the same in the default fp32 arithmetic, an odd batch of smaller images
        dict(name="resnet50_infer_strict_b29", kind="resnet", train=False, batch=29, size=161,
             blocks="3463", math="strict"),
        # the headline's first stage (it holds most of ResNet-50's bytes) at batch 256 per GPU
        dict(name="block_train_tf32_b256", kind="block", train=True, batch=256, size=56,
             channels=256, planes=64, stride=1, dtype="f32"),
        # mixed-precision training: the first block of the second stage, which halves the image
        dict(name="block_train_f16_b64", kind="block", train=True, batch=64, size=56, channels=256,
             planes=128, stride=2, dtype="f16"),
        # three layers of the third benchmark configuration: 16 utterances of 1000 frames
        dict(name="asr_train_b16_t1000", kind="asr", train=True, batch=16, frames=1000,
             channels=1024, layers=3, math="tf32"),
        # the fourth: 3-layer bidirectional LSTM over 500 frames
        dict(name="bilstm_train_h1024_t500", kind="rnn", train=True, cell="lstm", inputs=80,
             hidden=1024, layers=3, both=True, batch=32, frames=500, math="tf32"),
        # a short utterance through a small recurrent encoder, sizes off the tiles
        dict(name="gru_infer_h320_t61", kind="rnn", train=False, cell="gru", inputs=80, hidden=320,
             layers=2, both=False, batch=5, frames=61, math="tf32"),
        # the fifth: 12-layer Transformer LM, bf16 with fp32 master weights
        dict(name="lm_train_12x768_t512", kind="lm", train=True, layers=12, width=768, vocab=32000,
             batch=8, frames=512, dtype="bf16"),
        # a smaller model fine-tuned on sequences that are no multiple of a tile
        dict(name="lm_train_4x512_t200", kind="lm", train=True, layers=4, width=512, vocab=10000,
             batch=3, frames=200, dtype="bf16"),
        # one prompt scored by a server
        dict(name="lm_infer_12x768_t128", kind="lm", train=False, layers=12, width=768, vocab=32000,
             batch=1, frames=128, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mnist", "resnet", "asr", "rnn", "lm", "block"])
    train = rng.random() < 0.7
    fp32 = rng.choice(["strict", "tf32"])
    while True:
        if kind == "mnist":
            case = dict(kind=kind, train=train, batch=_log(rng, 1, 1024), math=fp32)
        elif kind == "resnet":
            case = dict(kind=kind, train=False, batch=_log(rng, 1, 256), size=rng.randint(96, 256),
                        blocks=rng.choice(["1111", "2222", "3463"]), math=fp32)
        elif kind == "asr":
            case = dict(kind=kind, train=train, batch=_log(rng, 1, 16),
                        frames=_log(rng, 60, 1500), channels=64 * rng.randint(4, 16),
                        layers=rng.randint(2, 3 if train and fp32 == "tf32" else 12), math=fp32)
        elif kind == "rnn":
            case = dict(kind=kind, train=train, cell=rng.choice(["lstm", "gru"]),
                        inputs=rng.choice([40, 80, 256]), hidden=8 * _log(rng, 16, 128),
                        layers=rng.randint(1, 3), both=rng.random() < 0.5,
                        batch=_log(rng, 1, 48), frames=_log(rng, 20, 500), math="tf32")
        elif kind == "lm":
            case = dict(kind=kind, train=train, layers=rng.randint(2, 12),
                        width=64 * rng.randint(4, 16), vocab=32 * rng.randint(100, 1000),
                        batch=_log(rng, 1, 8), frames=8 * _log(rng, 4, 64),
                        dtype=rng.choice(["bf16", "bf16", "f32"]))
        else:
            planes = rng.choice([64, 128, 256])
            stride = rng.choice([1, 1, 2])
            size = rng.randint(7, 56)
            # a gradient is of a batch: of few pixels it would hang on single relus
            pixels = rng.uniform(2e4, 4e5) if train else _log(rng, 50, 1e5)
            case = dict(kind=kind, train=train, batch=max(1, round(pixels * stride ** 2 / size ** 2)),
                        size=size, channels=planes * 4 // stride, planes=planes, stride=stride,
                        dtype=rng.choice(["f16", "bf16", "f32"]))
        cost = work(case)["flops"] * (8 if case.get("math") == "strict" else 1)
        if cost < 3.5e12:
            return case


# ---------------------------------------------------------------------------------- preparation
class _Dropout(nn.Module):
    """Dropout whose device-drawn mask is the same for every pass of one seed."""

    def __init__(self, p, seed):
        super().__init__()
        self.p, self.seed = p, seed

    def forward(self, x):
        if not self.train_mode:
            return x
        mask = bernoulli_mask(tuple(x.tensor.shape), 1.0 - self.p, x.tensor.device, x.tensor.dtype,
                              seed=self.seed, offset=0)
        return A.dropout(x, self.p, mask)


class _Block(nn.Module):
    """Batch-norm + relu of what the layer below computed, then a bottleneck block (1x1, 3x3 which
    carries the stride, 1x1, each with batch-norm; relu after the first two and after the join), on
    activations of one type stored channels-last, with fp32 parameters."""

    def __init__(self, channels, planes, stride, dtype, gen):
        super().__init__()
        out = planes * 4
        self.below = nn.BatchNorm(2, channels, gen=gen)
        self.children = [self.below]
        mk = lambda i, o, k: (nn.Conv2D(i, o, k, k, bias=False, gen=gen), nn.BatchNorm(2, o, gen=gen))
        self.stages = [mk(channels, planes, 1), mk(planes, planes, 3), mk(planes, out, 1)]
        if channels != out or stride > 1:
            self.stages.append(mk(channels, out, 1))
        self.stride, self.dtype = stride, dtype
        for s in self.stages:
            self.children += list(s)

    def _conv(self, x, conv, stride, pad):
        return A.conv2d(x, A.cast(conv.params[0], self.dtype), None, stride, stride, pad, pad,
                        stats=True)

    def forward(self, x):
        (c1, b1), (c2, b2), (c3, b3) = self.stages[:3]
        x = self.below(x, relu=True)
        h = b1(self._conv(x, c1, 1, 0), relu=True)
        h = b2(self._conv(h, c2, self.stride, 1), relu=True)
        z = self._conv(h, c3, 1, 0)
        if len(self.stages) > 3:
            c, b = self.stages[3]
            x = b(self._conv(x, c, self.stride, 0))
        return b3(z, addend=x)


def _each_norm(model, f=lambda m: None):
    norms, todo = [], [model]
    while todo:
        m = todo.pop()
        todo += m.children
        if isinstance(m, nn.BatchNorm):
            norms.append(m)
            f(m)
    return norms


def _gather_running(model):
    """The running statistics of every batch-norm as slices of one buffer (one file to save)."""
    norms = _each_norm(model)
    flat = torch.cat([t for m in norms for t in (m.running_mean, m.running_var)])
    at = 0
    for m in norms:
        n = m.running_mean.numel()
        m.running_mean, m.running_var = flat[at:at + n], flat[at + n:at + 2 * n]
        at += 2 * n
    return flat


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ints = lambda hi, n: torch.randint(0, hi, (n,), generator=gen, device="cuda", dtype=torch.int32)
    B, kind = case["batch"], case["kind"]
    s = dict(case=case, math=MATH[case.get("math", "tf32")])
    if kind == "mnist":
        model = workloads.mnist_convnet(seed)
        model.trunk.children[9] = _Dropout(0.5, seed)
        s.update(x=rand(B, 1, 28, 28), target=ints(10, B))
    elif kind == "resnet":
        model = workloads.resnet50(seed, blocks=tuple(int(c) for c in case["blocks"]))
        # the head averages what the last stage leaves of the image
        side = _resnet_sides(case["size"])[-1]
        model.trunk.children[-3] = nn.Pool2D(side, side, 1, 1, 0, 0, L.POOL_AVG_EXCLUDE_PAD)
        s.update(x=rand(B, 3, case["size"], case["size"]), target=ints(1000, B),
                 running=_gather_running(model))
    elif kind == "asr":
        model = workloads.ConvAsr(channels=case["channels"], layers=case["layers"], seed=seed)
        s.update(x=rand(B, 80, 1, case["frames"]), target=ints(30, B * case["frames"]))
    elif kind == "rnn":
        H, T, dirs = case["hidden"], case["frames"], 2 if case["both"] else 1
        n, bound = _rnn_params(case), 1.0 / math.sqrt(H)
        w = (torch.rand(n, generator=gen, device="cuda") * 2 - 1) * bound
        s.update(x=Variable(rand(T, B, case["inputs"]), case["train"]), w=Variable(w, case["train"]),
                 dy=rand(T, B, H * dirs))
        return s
    elif kind == "lm":
        model = workloads.TransformerLM(vocab=case["vocab"], d=case["width"],
                                        heads=case["width"] // 64, ffn=4 * case["width"],
                                        layers=case["layers"], seed=seed,
                                        compute_dtype=DTYPES[case["dtype"]])
        model.embed.tensor.mul_(8.0)  # 0.16: the spread of a trained embedding, not of an initial one
        ids = ints(case["vocab"], B * case["frames"])
        s.update(x=ids.reshape(B, case["frames"]).long(), target=ints(case["vocab"], ids.numel()))
    else:
        dt = DTYPES[case["dtype"]]
        model = _Block(case["channels"], case["planes"], case["stride"], dt,
                       torch.Generator().manual_seed(seed))
        cl = lambda t: t.to(dt).contiguous(memory_format=torch.channels_last)
        side = (case["size"] - 1) // case["stride"] + 1
        # x: what a convolution left; dy: the gradient of a mean loss, scaled for 16-bit types
        s.update(x=Variable(cl(rand(B, case["channels"], case["size"], case["size"])), False),
                 dy=cl(rand(B, 4 * case["planes"], side, side) * 0.05),
                 running=_gather_running(model))
    model.train(case["train"])
    s["model"] = model
    if "running" in s and not case["train"]:  # a server's statistics are those of its training
        _each_norm(model, lambda m: setattr(m, "momentum", 1.0))
        A.set_math_mode(s["math"])
        model.train(True)
        _scores(s, kind)
        model.train(False)
    return s


# ----------------------------------------------------------------------------------------- pass
def _gradients(params):
    """The gradients; of a Transformer as one vector, as for clipping by their common norm."""
    grads = [p.grad for p in params]
    return grads if len(grads) <= 32 else [torch.cat([g.reshape(-1) for g in grads])]


def _scores(s, kind):
    model = s["model"]
    if kind in ("mnist", "resnet", "block"):
        x = s["x"] if kind == "block" else Variable(s["x"], False)
        return model.forward(x).tensor
    if kind == "asr":
        h = Variable(s["x"], False)
        for conv in model.convs:
            h = A.relu(model.ln(conv(h)))
        frames = h.tensor.permute(0, 3, 2, 1).reshape(-1, model.channels)
        return A.log_softmax(model.head(Variable(frames, False))).tensor
    # the blocks of TransformerLM.loss, and the scores instead of the loss
    B, T = s["x"].shape
    x = A.embedding(A.cast(model.embed, model.compute_dtype), s["x"])
    for blk in model.blocks:
        x = A.add(x, model._attention(model._ln(x, blk["ln1"]), blk, B, T, None))
        h = model._lin(blk["w1"], model._ln(x, blk["ln2"]), gelu=True)
        x = A.add(x, model._lin(blk["w2"], h))
    return model._lin(model.head, model._ln(x, model.ln_f)).tensor


def run(s):
    case = s["case"]
    A.set_math_mode(s["math"])
    if case["kind"] == "rnn":
        x, w = s["x"], s["w"]
        x.zeroGrad(), w.zeroGrad()
        y, hy, cy = A.rnn(x, None, None, w, case["hidden"], case["layers"], CELLS[case["cell"]][0],
                          case["both"])
        out = [y.tensor, hy.tensor] + ([cy.tensor] if cy is not None else [])
        if case["train"]:
            y.backward(s["dy"])
            out += [x.grad, w.grad]
        return out
    if not case["train"]:
        return _scores(s, case["kind"])
    model = s["model"]
    model.zeroGrad()
    if case["kind"] == "block":
        y = model(s["x"])
        first = y.tensor
        y.backward(s["dy"])
        rest = []
    else:
        loss = model.loss(s["x"], s["target"])
        first = loss.tensor
        loss.backward()
        rest = []
    if "running" in s:
        rest.append(s["running"])
    return [first] + rest + _gradients(model.parameters())


# ------------------------------------------------------------------------------ work, tolerance
def _resnet_sides(size):
    """Extent of the image after the stem's convolution and in each of the four stages."""
    half = lambda v: (v - 1) // 2 + 1 if v % 2 else v // 2
    sides = [half(size)]
    sides.append(half(sides[0]))
    for _ in range(3):
        sides.append(half(sides[-1]))
    return sides


def _rnn_params(case):
    G, H, dirs = CELLS[case["cell"]][1], case["hidden"], 2 if case["both"] else 1
    return sum(dirs * G * H * ((case["inputs"] if l == 0 else H * dirs) + H + 2)
               for l in range(case["layers"]))


def work(case):
    """Multiply-adds of the contractions; every input, parameter, gradient and result once."""
    B, kind, train = case["batch"], case["kind"], case["train"]
    macs, params, io, es = 0, 0, 0, 4
    if kind == "mnist":
        macs = B * (784 * 32 * 25 + 196 * 64 * 32 * 25 + 3136 * 1024 + 10240)
        params, io = 32 * 26 + 64 * 801 + 3137 * 1024 + 10250, B * 784
    elif kind == "resnet":
        sides = _resnet_sides(case["size"])
        macs, params, io = B * sides[0] ** 2 * 64 * 147, 64 * 149 + 2049 * 1000, B * 3 * case["size"] ** 2
        cin = 64
        for i, n in enumerate(int(c) for c in case["blocks"]):
            p, side = 64 << i, sides[i + 1]
            for j in range(n):
                before = sides[i] if i and j == 0 else side
                macs += B * (before ** 2 * cin * p + side ** 2 * 13 * p * p)
                params += cin * p + 13 * p * p + 12 * p
                if j == 0:
                    macs += B * side ** 2 * cin * 4 * p
                    params += cin * 4 * p + 8 * p
                cin = 4 * p
        macs += B * 2048 * 1000
    elif kind == "asr":
        C, n = case["channels"], case["layers"]
        params = 13 * C * (80 + (n - 1) * C) + n * C + 30 * (C + 1)
        macs, io = B * case["frames"] * params, B * case["frames"] * 80
    elif kind == "rnn":
        dirs = 2 if case["both"] else 1
        params = _rnn_params(case)
        macs = B * case["frames"] * params
        io = B * case["frames"] * (case["inputs"] * (2 if train else 1)
                                   + case["hidden"] * dirs * (2 if train else 1))
    elif kind == "lm":
        d, T, V, n = case["width"], case["frames"], case["vocab"], case["layers"]
        params = 2 * V * d + V + n * (12 * d * d + 13 * d) + 2 * d
        macs = B * T * (n * 12 * d * d + V * d) + n * B * T * T * d  # half the scores are masked
        io = B * T * (1 if train else V)
    else:
        C, p, side = case["channels"], case["planes"], (case["size"] - 1) // case["stride"] + 1
        params = C * p + 13 * p * p + 12 * p
        macs = B * (case["size"] ** 2 * C * p + side ** 2 * 13 * p * p)
        if C != 4 * p or case["stride"] > 1:
            params += 4 * C * p + 8 * p
            macs += B * side ** 2 * C * 4 * p
        io = B * (case["size"] ** 2 * C + side ** 2 * 4 * p) * (2 if train else 1) // 2  # 16 bits
    return {"bytes": es * (io + params * (2 if train else 1)), "flops": 2 * macs * (3 if train else 1)}


def tolerance(case):
    """What the arithmetic gives and no more: the largest differences seen after a change of the
    parameters' last bit, with some room.  bf16 and TF32 round every operand (2^-9, 2^-11), and a
    relu or pooling window within a rounding error of a tie turns the other way, which moves whole
    gradient elements; most rows of an embedding's gradient are zero, which makes its largest
    difference large beside the root mean square."""
    kind, train, dtype = case["kind"], case["train"], case.get("dtype")
    if case.get("math") == "strict":
        return {"rel": 1e-2 if train and kind == "asr" else 2e-3 if train else 1e-4}
    if kind == "lm":
        return {"rel": 2.5e-2 if dtype == "bf16" else 5e-3, "max": 0.99}
    if kind == "block":
        return {"rel": (2.5e-2 if dtype != "f32" else 2e-2) if train else 3e-3, "max": 0.9}
    if kind == "resnet":
        return {"rel": 2.5e-2}
    if train and kind in ("asr", "mnist"):
        return {"rel": 2e-2 if kind == "asr" else 1.5e-2, "max": 0.9}
    return {"rel": 2e-3}
