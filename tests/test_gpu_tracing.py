"""GPU: what records or intercepts torch operations still finds them in a plain layer."""
import warnings

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return (a.float() - b.float()).norm().item() / b.float().norm().item()


def _dirty_memory():   # what a graph that lost its kernels would read
    for k in range(10, 21):
        torch.full((1 << k,), 1e4, device="cuda")


@pytest.mark.parametrize("dtype,kw", [(torch.bfloat16, {}), (torch.float32, dict(prenorm=True, rotary_emb=True)),
                                      (torch.float16, dict(prenorm=True, dim_head=128))])
def test_jit_trace_of_the_layer(dtype, kw):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(0)
    m = Castle(96, heads=2, **kw).cuda().to(dtype)
    x, y, g = (torch.randn(2, 140, 96, device="cuda").to(dtype) for _ in range(3))
    y.requires_grad_()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        traced = torch.jit.trace(m, x, check_trace=False)
    _dirty_memory()
    out, want = traced(y), m(y)
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-3
    assert _rel(out, want) <= tol
    wanted = [y, *m.parameters()]
    for a, b in zip(torch.autograd.grad(out, wanted, g), torch.autograd.grad(want, wanted, g)):
        assert _rel(a, b) <= tol


@pytest.mark.parametrize("packed", [False, True])
def test_jit_trace_of_the_operators(packed):
    from lookahead_keys_attention_b200 import castle_attention, castle_attention_packed

    def f(t):
        if packed:
            return castle_attention_packed(t, 0.125, True)
        qu, ku, vu, qc, kc, vc = (t[:, :, i].permute(0, 2, 1, 3) for i in range(6))
        return castle_attention(qc, kc, vc, qu, ku, vu, 0.125, True)

    a, b = (torch.randn(2, 140, 6, 2, 64, device="cuda") * 3 ** -0.5 for _ in range(2))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        traced = torch.jit.trace(f, a, check_trace=False)
    _dirty_memory()
    b.requires_grad_()
    got, want = traced(b), f(b)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and not want[1].requires_grad
    g = torch.randn_like(got[0])
    assert _rel(torch.autograd.grad(got[0], b, g)[0], torch.autograd.grad(want[0], b, g)[0]) <= 4e-3
