"""GPU: the rotary frequencies wherever and however the module's buffer holds them, and rotary embeddings of the
caller's own in the place of the module's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(m, x, g):
    x = x.detach().requires_grad_()
    out, cache = m(x, return_next_cache=True)
    grads = torch.autograd.grad(out, [x, *m.parameters()], g)
    with torch.no_grad():
        step, cache = m(x[:, :1], cache=cache)
    return [out.detach(), step, cache.qu_cache], grads


@pytest.mark.parametrize("form", ["cpu", "strided", "double", "row", "one"])
@pytest.mark.parametrize("hooked", [False, True])
def test_frequencies_of_another_device_stride_or_type(form, hooked):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(0)
    m = Castle(96, heads=2, dim_head=64, rotary_emb=True).cuda().bfloat16()
    m.rotary_emb.freqs = m.rotary_emb.freqs.float()
    x, g = (torch.randn(2, 140, 96, device="cuda").bfloat16() for _ in range(2))
    if hooked:   # the submodules called as modules
        m.to_all_qkv.register_forward_hook(lambda *a: None)
    if form == "one":
        m.rotary_emb.freqs = m.rotary_emb.freqs[3].repeat(32)
    want, want_grads = _run(m, x, g)
    f = m.rotary_emb.freqs
    m.rotary_emb.freqs = {"cpu": f.cpu(), "strided": torch.stack([f, f + 1], 1)[:, 0], "double": f.double(), "row": f[None],
                          "one": f[0]}[form]
    got, grads = _run(m, x, g)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert all((a.float() - b.float()).norm() <= 4e-3 * b.float().norm() for a, b in zip(grads, want_grads))


@pytest.mark.parametrize("freqs", [torch.ones(16), torch.ones(64), torch.ones(32, 1), torch.ones(0)])
def test_frequencies_of_another_shape_are_refused(freqs):
    from lookahead_keys_attention_b200 import Castle
    m = Castle(96, heads=2, dim_head=64, rotary_emb=True).cuda().bfloat16()
    m.rotary_emb.freqs = freqs.cuda()
    for n in (1, 140):
        with torch.no_grad(), pytest.raises(RuntimeError, match="rotary frequencies"):
            m(torch.zeros(2, n, 96, device="cuda", dtype=torch.bfloat16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_rotary_embedding_of_the_callers_own(dtype):
    from lookahead_keys_attention_b200 import Castle
    from lookahead_keys_attention_b200.castle import _Rotary
    torch.manual_seed(0)
    m = Castle(96, heads=2, dim_head=64, rotary_emb=True, prenorm=True).cuda().to(dtype)
    x, g = (torch.randn(2, 140, 96, device="cuda").to(dtype) for _ in range(2))
    want, want_grads = _run(m, x, g)

    class Same(_Rotary):
        def rotate(self, t, offset=0):
            self.calls += 1
            return super().rotate(t, offset)

    own = Same(64).cuda().to(dtype)
    own.calls = 0
    m.rotary_emb = own
    got, grads = _run(m, x, g)
    assert own.calls == 10   # five tensors, prompt and step
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-3
    for a, b in zip([*got, *grads], [*want, *want_grads]):
        assert (a.float() - b.float()).norm() <= tol * b.float().norm()
    m.rotary_emb.rotate = lambda t, offset=0: t      # and what it does is what counts
    plain, _ = _run(m, x, g)
    m.rotary_emb = None
    for a, b in zip(plain, _run(m, x, g)[0]):
        assert (a.float() - b.float()).norm() <= tol * b.float().norm()
