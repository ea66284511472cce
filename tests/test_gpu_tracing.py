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


class _Scaled(torch.Tensor):
    """A weight that emulates another precision where it is used."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        plain = lambda t: t.as_subclass(torch.Tensor) * 2 if isinstance(t, cls) and func is torch.nn.functional.linear else t   # noqa: E731
        return super().__torch_function__(func, types, tuple(plain(a) for a in args), kwargs)


def test_torch_functions_are_called_where_they_may_be_replaced():
    from torch.overrides import TorchFunctionMode
    from lookahead_keys_attention_b200 import Castle

    class DoubleLinear(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            y = func(*args, **(kwargs or {}))
            return y * 2 if func is torch.nn.functional.linear else y

    torch.manual_seed(0)
    m = Castle(96, heads=2).cuda().bfloat16().requires_grad_(False)
    x = torch.randn(2, 140, 96, device="cuda").bfloat16()
    last = m.combine_heads.weight.clone()
    with torch.no_grad():
        plain, cache = m(x, return_next_cache=True)
        step, _ = m(x[:, :1], cache=cache)
        with torch.device("cuda"):                    # a default device replaces nothing
            assert torch.equal(m(x), plain)
        m.to_all_qkv.weight.mul_(2)
        m.combine_heads.weight.mul_(2)
        want, cache = m(x, return_next_cache=True)
        want_step, _ = m(x[:, :1], cache=cache)
        m.to_all_qkv.weight.mul_(0.5)
        m.combine_heads.weight.mul_(0.5)
        assert torch.equal(m.combine_heads.weight, last)
        with DoubleLinear():
            got, cache = m(x, return_next_cache=True)
            got_step, _ = m(x[:, :1], cache=cache)
        assert _rel(got, want) <= 1e-2 and _rel(got_step, want_step) <= 1e-2
        for sub in (m.to_all_qkv, m.combine_heads):
            sub._parameters["weight"] = sub.weight.detach().as_subclass(_Scaled)
        assert _rel(m(x), want) <= 1e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [140, 600])   # 280 positions: products of the framework's own; 1200: the library's
def test_batched_gradients_of_the_output_projection(dtype, n):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(n)
    m = Castle(96, heads=2).cuda().to(dtype)
    x = torch.randn(2, n, 96, device="cuda").to(dtype)
    g = torch.randn(3, 2, n, 96, device="cuda").to(dtype)
    for frozen in (True, False):
        m.to_all_qkv.requires_grad_(not frozen)
        out, w = m(x), m.combine_heads.weight
        got, = torch.autograd.grad(out, w, g, is_grads_batched=True, retain_graph=True)
        # sums in another order: a 16-bit result may be rounded the other way (2^-8 of a value), an fp32 one differs by sqrt(k) 2^-24
        for a, b in zip(got, g):
            assert _rel(a, torch.autograd.grad(out, w, b, retain_graph=True)[0]) <= (4e-3 if dtype == torch.bfloat16 else 1e-5)


def test_dispatch_modes_see_the_products_of_the_gradient():
    from torch.utils._python_dispatch import TorchDispatchMode
    from lookahead_keys_attention_b200 import Castle
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    torch.manual_seed(0)
    m = Castle(96, heads=2).cuda()
    x, g = (torch.randn(2, 140, 96, device="cuda") for _ in range(2))
    wanted = [x.requires_grad_(), *m.parameters()]
    out = m(x)
    plain = torch.autograd.grad(out, wanted, g, retain_graph=True)
    with Watch():
        got = torch.autograd.grad(out, wanted, g)
    assert seen.count(torch.ops.aten.mm.default) == 4   # both weights, the merged heads, the input
    for a, b in zip(got, plain):   # the core's gradient is rounded to its 16-bit operands' type: by at most 2^-10 of a value another way
        assert _rel(a, b) <= 2e-3
