"""GPU: several host threads on one stream.  A call hands values from launch to launch through the stream's scratch, so the
launches of two calls must not mix."""
import sys
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _decoder(dim, heads, d, batch, dtype, n=96, tokens=150):
    from lookahead_keys_attention_b200 import Castle, cache_from_buffers
    torch.manual_seed(dim + batch)
    m = Castle(dim, heads=heads, dim_head=d, prenorm=True).cuda().to(dtype)
    x = torch.randn(batch, tokens, dim, device="cuda").to(dtype)
    start = [torch.randn(batch, heads, n + tokens, d, device="cuda").to(dtype) for _ in range(4)]

    def go():
        with torch.no_grad():
            cache, outs = cache_from_buffers(*[b.clone() for b in start], n), []
            for i in range(tokens):
                out, cache = m(x[:, i:i + 1], cache=cache)
                outs.append(out)
            return [torch.cat(outs, 1), *cache], 0.0

    return go


def _trainer(dim, heads, d, batch, dtype, n=200, steps=25):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(dim + n)
    m = Castle(dim, heads=heads, dim_head=d, prenorm=True).cuda().to(dtype)
    x = torch.randn(batch, n, dim, device="cuda").to(dtype).requires_grad_()
    g = torch.randn(batch, n, dim, device="cuda").to(dtype)

    def go():
        for _ in range(steps):
            out = m(x)
            grads = torch.autograd.grad(out, [x, *m.parameters()], g)
        return [out.detach(), *grads], 4e-3   # gradients summed in arrival order differ by a few ulps

    return go


@pytest.mark.parametrize("side_stream", [False, True])
def test_threads_on_one_stream(side_stream):
    from lookahead_keys_attention_b200 import check_status
    work = [_decoder(512, 8, 64, 1, torch.bfloat16), _decoder(256, 4, 64, 2, torch.float32), _decoder(384, 3, 128, 5, torch.float16),
            _trainer(256, 4, 64, 3, torch.float32), _trainer(256, 2, 128, 2, torch.bfloat16)]
    stream = torch.cuda.Stream() if side_stream else torch.cuda.default_stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        alone = [f()[0] for f in work]
    results, errors = [None] * len(work), []

    def run(i):
        try:
            with torch.cuda.stream(stream):
                results[i] = work[i]()
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=run, args=(i,)) for i in range(len(work))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    torch.cuda.synchronize()
    check_status()
    assert not errors, errors
    for (got, tol), want in zip(results, alone):
        for a, b in zip(got, want):
            if tol == 0.0:
                assert torch.equal(a, b)
            else:
                assert (a.float() - b.float()).norm().item() <= tol * b.float().norm().item()
