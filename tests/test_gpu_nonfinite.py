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
