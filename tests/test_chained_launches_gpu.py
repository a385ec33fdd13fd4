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
