"""GPU: values that are not finite.  A NaN score reaches every row that sees it whatever the key's position in its tile, so
that a diverging run is seen; the exponential that is computed without the special-function unit agrees with exp2 over its
whole range."""
import pytest
import torch

from oracle import castle_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("which", ["kc", "qu"])
@pytest.mark.parametrize("key", [0, 1, 2, 16, 33, 129, 255])
def test_nan_key_reaches_every_row_that_sees_it(d, which, key):
    from lookahead_keys_attention_b200 import castle_attention
    torch.manual_seed(key)
    names = ("qc", "kc", "vc", "qu", "ku", "vu")
    v = [(torch.randn(1, 2, 260, d, device="cuda") * 3 ** -0.5).bfloat16() for _ in names]
    v[names.index(which)][0, 1, key, 5] = float("nan")
    for t in v:
        t.requires_grad_()
    out = castle_attention(*v, d ** -0.5)
    with torch.no_grad():
        ref = O.castle_parallel(*(t.float() for t in v), d ** -0.5)
    # (a NaN in qu makes the key's gates NaN from the next position on; the dense form's 0 * NaN reaches further back)
    assert torch.equal(out.isnan(), ref.isnan()) if which == "kc" else bool((out.isnan() <= ref.isnan()).all())
    assert out[0, 1, key + 1:].isnan().all() and not out[0, 0].isnan().any()
    # a row whose soft-max is NaN has NaN weights for all of its keys, so no key's value gradient is finite
    dvc = torch.autograd.grad(out, v[2], torch.ones_like(out))[0]
    assert dvc[0, 1].isnan().all() and not dvc[0, 0].isnan().any()


def test_exp2_of_the_score_passes():
    """Over the range of normal results the error is the polynomial's (1.0e-7 of the value) and one rounding of the last
    fused step (2^-24 = 0.6e-7): at most 1.7e-7, which is also what ex2.approx is good to."""
    from lookahead_keys_attention_b200 import _lib as L
    inf, nan = float("inf"), float("nan")
    edges = torch.tensor([nan, -nan, inf, -inf, 128.0, 129.0, 1e30, -1e30, -126.5, -127.0, -200.0, 0.0], device="cuda")
    whole = torch.arange(-126, 128, device="cuda", dtype=torch.float32)
    dense = torch.linspace(-126, 127.99, 1 << 23, device="cuda")
    near = torch.linspace(-1, 1, 1 << 20, device="cuda") ** 5       # many small arguments
    x = torch.cat([edges, whole, dense, near])
    y = torch.empty_like(x)
    L.check(L.load().castle_selftest_exp2(x.data_ptr(), y.data_ptr(), x.numel(), None), "exp2")
    torch.cuda.synchronize()
    want = torch.tensor([nan, nan, inf, 0, inf, inf, inf, 0, 0, 0, 0, 1], device="cuda")
    assert torch.equal(y[:12].isnan(), want.isnan()) and torch.equal(y[2:12], want[2:])
    assert torch.equal(y[12:12 + whole.numel()], torch.exp2(whole.double()).float())
    ref = torch.exp2(x[12:].double())
    assert ((y[12:].double() - ref).abs() / ref).max().item() <= 1.7e-7


@pytest.mark.parametrize("N,dtype,d", [(300, torch.float32, 64), (300, torch.float32, 128), (6200, torch.bfloat16, 64)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_a_bad_upstream_gradient_is_seen_and_stays_where_it_is(N, dtype, d, bad):
    """Callers whose gradient is rescaled for fp16 operands: the (batch, head) pair of a bad element gets gradients that are
    not finite (what loss scalers look for), and the other pairs the same as without it."""
    from lookahead_keys_attention_b200 import castle_attention_packed
    torch.manual_seed(N)
    x = (torch.randn(2, N, 6, 2, d, device="cuda") * 3 ** -0.5).to(dtype).requires_grad_()
    g = (torch.randn(2, 2, N, d, device="cuda") * 1e-3).to(dtype)
    out = castle_attention_packed(x, d ** -0.5)
    good = torch.autograd.grad(out, x, g, retain_graph=True)[0]
    g[1, 1, N // 2, 3] = bad
    grad = torch.autograd.grad(out, x, g)[0]
    assert not grad[1, :, :, 1].isfinite().all()
    for b, h in [(0, 0), (0, 1), (1, 0)]:
        a, w = grad[b, :, :, h].float(), good[b, :, :, h].float()
        assert (a - w).norm().item() <= 4e-3 * w.norm().item()   # sums in arrival order differ by a few ulps


@pytest.mark.parametrize("top", [1e-20, 1e9, 3e13, 1e30])
def test_the_gradients_magnitude_does_not_matter(top):
    """A power of two of the upstream gradient is one of the gradients."""
    from lookahead_keys_attention_b200 import castle_attention_packed
    torch.manual_seed(0)
    x = (torch.randn(1, 200, 6, 2, 64, device="cuda") * 3 ** -0.5).requires_grad_()
    g = torch.randn(1, 2, 200, 64, device="cuda")
    f = 2.0 ** torch.tensor(top).log2().round().item()
    out = castle_attention_packed(x, 0.125)
    a, b = (torch.autograd.grad(out, x, t, retain_graph=True)[0] for t in (g * f, g))
    # below 2^-24 of the usual magnitude the factor stays 2^24 and fp16 loses what lies under its range
    assert (a.double() / f - b.double()).norm().item() <= 4e-3 * b.double().norm().item() or top < 1e-9
    assert a.isfinite().all()


def test_conversion_keeps_nan():
    from lookahead_keys_attention_b200 import _lib as L
    x = torch.tensor([1.0, float("nan"), float("inf"), -float("inf"), 7e4, 0.0, -3.0, 5.0], device="cuda").bfloat16()
    y = torch.empty_like(x, dtype=torch.float16)
    L.check(L.load().castle_convert_16bit(L.BF16, x.data_ptr(), y.data_ptr(), x.numel(), None, None), "convert")
    want = x.float().clamp(-65504, 65504).half()
    assert y[1].isnan() and torch.equal(y[2:], want[2:]) and y[0] == 1
