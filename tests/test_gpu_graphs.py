"""GPU: calls captured into CUDA graphs own their scratch and counters, whatever ran on the capturing stream before, and
the status word outlives replays."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


def _step(seed, n=700, B=1, H=4, d=64):
    """A decode step that is split over CTAs, with its last CTA merging: inputs, and the call on copies of the caches."""
    from lookahead_keys_attention_b200 import castle_decode_step
    gen = torch.Generator("cuda").manual_seed(seed)
    new = [torch.randn(B, H, 1, d, device="cuda", generator=gen).bfloat16() for _ in range(6)]
    base = [torch.randn(B, H, n + 8, d, device="cuda", generator=gen).bfloat16() for _ in range(4)]
    bufs = [b.clone() for b in base]

    def call():
        for a, b in zip(bufs, base):
            a.copy_(b)
        return castle_decode_step(*new, *bufs, n, d ** -0.5)

    return call


def _capture(call, stream, pool=None):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, pool=pool):
        out = call()
    return graph, out


def test_a_graph_does_not_need_another_ones_replay():
    steps = [_step(i) for i in range(2)]
    want = [s() for s in steps]
    stream = torch.cuda.Stream()
    # memory of the pool that the graphs will use, left full of large numbers
    dirt, _ = _capture(lambda: [torch.full((1 << 16,), 1 << 20, dtype=torch.int32, device="cuda") for _ in range(64)] and None, stream)
    dirt.replay()
    torch.cuda.synchronize()
    graphs = [_capture(s, stream, dirt.pool()) for s in steps]
    for i in (1, 0, 1):
        graphs[i][1].zero_()
        graphs[i][0].replay()
        torch.cuda.synchronize()
        assert torch.equal(graphs[i][1], want[i])


def test_graphs_of_one_stream_replay_beside_each_other_and_eager_calls():
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(0)
    m = Castle(256, heads=4, prenorm=True).cuda().bfloat16()
    xs = [torch.randn(2, 900, 256, device="cuda").bfloat16() for _ in range(3)]
    with torch.no_grad():
        want = [m(x) for x in xs]
        stream, others = torch.cuda.Stream(), [torch.cuda.Stream() for _ in range(2)]
        graphs = [_capture(lambda x=x: m(x), stream) for x in xs[:2]]
        for _ in range(20):
            for (g, out), s in zip(graphs, others):
                out.zero_()
                s.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(s):
                    for _ in range(5):
                        g.replay()
            with torch.cuda.stream(stream):
                eager = [m(xs[2]) for _ in range(5)]
            torch.cuda.synchronize()
            assert all(torch.equal(out, w) for (_, out), w in zip(graphs, want)) and all(torch.equal(e, want[2]) for e in eager)


CHILD = """
import torch
from lookahead_keys_attention_b200 import Castle, check_status, ops
torch.manual_seed(0)
m = Castle(256, heads=4, prenorm=True).cuda().bfloat16()
x = torch.randn(2, 300, 256, device="cuda").bfloat16().requires_grad_()
grad = torch.randn(2, 300, 256, device="cuda").bfloat16()
w = torch.randn(8, 8, device="cuda", requires_grad=True)
(w @ w).sum().backward()                     # the library's handles, of the engine's thread too
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):                    # the framework's first call of the process, backward included
    out = m(x)
    grads = torch.autograd.grad(out, [x, *m.parameters()], grad)
word = ops.status_word("cuda")
assert int(word.item()) == 0
g.replay()
torch.cuda.synchronize()
want = torch.autograd.grad(m(x), [x, *m.parameters()], grad)
for a, b in zip(grads, want):
    assert (a.float() - b.float()).norm() <= 4e-3 * b.float().norm()
word.fill_(1)
g.replay()
try:
    check_status()
except RuntimeError as e:
    assert "status 1" in str(e)
    print("fine")
"""


def test_first_call_under_capture_and_the_status_word():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
