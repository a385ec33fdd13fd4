"""Kernels of a stream are launched before the kernel in front of them has ended and wait for it themselves.
Training steps made of most of the library's kernels give the same bits where every launch is waited for
on the host, in a stream of their own, and as replays of a captured graph."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

STEPS = r"""
import sys, torch
sys.path.insert(0, %r)
from flashlight_b200 import _lib as L, autograd as A, workloads
g = torch.Generator(device="cuda").manual_seed(3)
rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
ints = lambda hi, n: torch.randint(0, hi, (n,), generator=g, device="cuda", dtype=torch.int32)
tokens = ints(3200, 400)
cases = [
    (L.MATH_STRICT_F32, workloads.mnist_convnet(1), rand(5, 1, 28, 28), ints(10, 5)),
    (L.MATH_TF32, workloads.resnet50(2, blocks=(1, 1, 1, 1)), rand(2, 3, 224, 224), ints(1000, 2)),
    (L.MATH_TF32, workloads.ConvAsr(channels=64, layers=2, seed=3), rand(2, 80, 1, 90), ints(30, 180)),
    (L.MATH_TF32, workloads.TransformerLM(vocab=3200, d=256, heads=4, ffn=1024, layers=2, seed=4,
                                          compute_dtype=torch.bfloat16), tokens.reshape(2, 200).long(),
     ints(3200, 400)),
]
cases[0][1].trunk.children[9] = torch.nn.Identity()  # (dropout draws a mask per pass)
def step(mode, model, x, t):
    A.set_math_mode(mode)
    model.zeroGrad()
    loss = model.loss(x, t)
    loss.backward()
    return [loss.tensor] + [p.grad for p in model.parameters()]
""" % str(ROOT)


def run(tail, path, **env):
    res = subprocess.run([sys.executable, "-c", STEPS + tail, path], env=dict(os.environ, **env),
                         capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr[-2000:]
    return torch.load(path)


def test_chained_launches(tmp_path):
    plain = """
out = []
for _ in range(3):  # the last of three passes in one queue
    out = [[v.clone() for v in step(*c)] for c in cases]
torch.save([[v.cpu() for v in o] for o in out], sys.argv[1])
"""
    want = run(plain, str(tmp_path / "blocking.pt"), CUDA_LAUNCH_BLOCKING="1")
    got = run(plain, str(tmp_path / "queued.pt"))
    side = run("s = torch.cuda.Stream()\ns.wait_stream(torch.cuda.current_stream())\n"
               "torch.cuda.set_stream(s)\n" + plain, str(tmp_path / "stream.pt"))
    graph = run("""
out, s = [], torch.cuda.Stream()
s.wait_stream(torch.cuda.current_stream())
with torch.cuda.stream(s):
    for _ in range(2):
        for c in cases: step(*c)
torch.cuda.synchronize()
for c in cases[2:]:  # (without running statistics)
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr, stream=s):
        o = step(*c)
    for _ in range(3): gr.replay()
    torch.cuda.synchronize()
    out.append([v.cpu() for v in o])
    for v in o: v.zero_()
torch.save(out, sys.argv[1])
""", str(tmp_path / "graph.pt"))
    for k, (a, b, c) in enumerate(zip(want, got, side)):
        assert all(torch.equal(x, y) for x, y in zip(a, b)), f"case {k}"
        assert all(torch.equal(x, y) for x, y in zip(a, c)), f"case {k} in its own stream"
    for k, (a, b) in enumerate(zip(want[2:], graph)):
        assert all(torch.equal(x, y) for x, y in zip(a, b)), f"case {k + 2} from a graph"


def test_chained_around_other_launches(tmp_path):
    """Recurrences (cluster kernels that are launched as before, and hold all tensor memory) between chained
    kernels, a 16-bit residual block, gradients copied by a second stream behind an event while the first goes
    on, and replays of networks with batch-norm and pooling (of gradients: they do not depend on the running
    statistics)."""
    more = r"""
from flashlight_b200.autograd import Variable
class Block:
    def __init__(self):
        gen = torch.Generator().manual_seed(7)
        self.b = workloads.Bottleneck(64, 32, 1, gen, "cuda")
    def zeroGrad(self): self.b.zeroGrad()
    def parameters(self): return self.b.parameters()
    def loss(self, x, t):
        convs = [self.b.c1, self.b.c2, self.b.c3, self.b.down.children[0]]
        x = Variable(x, False)
        conv = lambda h, c, p: A.conv2d(h, A.cast(c.params[0], torch.float16), None, 1, 1, p, p, stats=True)
        h = self.b.b1(conv(x, convs[0], 0), relu=True)
        h = self.b.b2(conv(h, convs[1], 1), relu=True)
        down = self.b.down.children[1](conv(x, convs[3], 0))
        return Head(self.b.b3(conv(h, convs[2], 0), addend=down), t)
class Head:  # the gradient of the block's output is the target
    def __init__(self, y, t): self.y, self.t, self.tensor = y, t, y.tensor
    def backward(self): self.y.backward(self.t)
cl = lambda t: t.half().contiguous(memory_format=torch.channels_last)
cases[2:] = [
    (L.MATH_TF32, workloads.BiLstm(24, 72, 2), rand(9, 5, 24), rand(9, 5, 144)),
    (L.MATH_TF32, workloads.BiLstm(24, 520, 1), rand(7, 3, 24), rand(7, 3, 1040)),
    (L.MATH_TF32, Block(), cl(rand(2, 64, 14, 14)), cl(rand(2, 128, 14, 14) * 0.05)),
]
"""
    plain = more + """
other, out = torch.cuda.Stream(), []
for _ in range(3):
    out = []
    for c in cases:
        v = step(*c)
        e = torch.cuda.Event()
        e.record()
        with torch.cuda.stream(other):
            other.wait_event(e)
            out.append([t.clone() for t in v])
            e2 = torch.cuda.Event()
            e2.record()
        A.relu(Variable(rand(64, 64), False))  # the first stream goes on
        torch.cuda.current_stream().wait_event(e2)
torch.cuda.synchronize()
torch.save([[v.cpu() for v in o] for o in out], sys.argv[1])
"""
    want = run(plain, str(tmp_path / "blocking.pt"), CUDA_LAUNCH_BLOCKING="1")
    got = run(plain, str(tmp_path / "queued.pt"))
    graph = run(more + """
out, s = [], torch.cuda.Stream()
s.wait_stream(torch.cuda.current_stream())
with torch.cuda.stream(s):
    for _ in range(2):
        for c in cases: step(*c)
torch.cuda.synchronize()
for c in cases:
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr, stream=s):
        o = step(*c)
    for _ in range(3): gr.replay()
    torch.cuda.synchronize()
    out.append([v.cpu() for v in o])
    for v in o: v.zero_()
torch.save(out, sys.argv[1])
""", str(tmp_path / "graph.pt"))
    for k, (a, b, c) in enumerate(zip(want, got, graph)):
        assert all(torch.equal(x, y) for x, y in zip(a, b)), f"case {k}"
        assert all(torch.equal(x, y) for x, y in zip(a, c)), f"case {k} from a graph"
