"""GPU: what a training forward keeps for its backward goes through autograd's saved tensors - hooks see all of it, so
activation checkpointing recomputes it and save_on_cpu moves it off the GPU."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu
B, N, DIM, H = 2, 300, 96, 2


def _layer(dtype, prenorm, rotary, d):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(d)
    m = Castle(DIM, heads=H, dim_head=d, prenorm=prenorm, rotary_emb=rotary).cuda().to(dtype)
    x = torch.randn(B, N, DIM, device="cuda").to(dtype).requires_grad_()
    assert m._plain_layer() is not None
    return m, [x, *m.parameters()], torch.randn(B, N, DIM, device="cuda").to(dtype)


def _grads(f, wanted, g):
    out = f(wanted[0])
    return [out.detach(), *torch.autograd.grad(out, wanted, g)]


def _same(a, b):   # the sums that are added in arrival order differ by a few ulps from run to run
    for x, y in zip(a, b):
        assert (x.float() - y.float()).norm().item() <= 4e-3 * y.float().norm().item()


LAYERS = [(torch.bfloat16, False, False, 64), (torch.bfloat16, True, True, 64), (torch.float32, True, False, 64),
          (torch.float16, False, True, 128), (torch.float32, False, True, 32)]


@pytest.mark.parametrize("dtype,prenorm,rotary,d", LAYERS)
def test_hooks_see_everything_the_layer_keeps(dtype, prenorm, rotary, d):
    m, wanted, g = _layer(dtype, prenorm, rotary, d)
    plain = _grads(m, wanted, g)
    seen = []

    def pack(t):
        seen.append((tuple(t.shape), t.dtype))
        return t.cpu().contiguous()   # other strides than the forward's, as save_on_cpu gives them

    before = torch.cuda.memory_allocated()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        out = m(wanted[0])
    # nothing of the forward but its output is held on the device
    assert torch.cuda.memory_allocated() - before <= out.numel() * out.element_size() + 4096
    _same([out.detach(), *torch.autograd.grad(out, wanted, g)], plain)
    dp = 64 if d <= 64 else 128
    assert ((B, H, N, dp), torch.float32) in seen   # the lookahead state


@pytest.mark.parametrize("dtype,prenorm,rotary,d", LAYERS)
def test_layer_under_checkpoint(dtype, prenorm, rotary, d):
    m, wanted, g = _layer(dtype, prenorm, rotary, d)
    plain = _grads(m, wanted, g)
    for early_stop in (True, False):
        with torch.utils.checkpoint.set_checkpoint_early_stop(early_stop):
            before = torch.cuda.memory_allocated()
            out = checkpoint(m, wanted[0], use_reentrant=False)
            assert torch.cuda.memory_allocated() - before <= out.numel() * out.element_size() + 4096
            _same([out.detach(), *torch.autograd.grad(out, wanted, g)], plain)


@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 64), (torch.float32, 64), (torch.float16, 128), (torch.bfloat16, 32)])
@pytest.mark.parametrize("packed", [False, True])
def test_operator_under_checkpoint_and_on_cpu(dtype, d, packed):
    from lookahead_keys_attention_b200 import castle_attention, castle_attention_packed
    torch.manual_seed(d)
    x = (torch.randn(B, N, 6, H, d, device="cuda") * 3 ** -0.5).to(dtype).requires_grad_()
    g = torch.randn(B, H, N, d, device="cuda").to(dtype)

    def f(x):
        if packed:
            return castle_attention_packed(x, d ** -0.5)
        qu, ku, vu, qc, kc, vc = (x[:, :, i].permute(0, 2, 1, 3) for i in range(6))
        return castle_attention(qc, kc, vc, qu, ku, vu, d ** -0.5)

    plain = _grads(f, [x], g)
    _same(_grads(lambda t: checkpoint(f, t, use_reentrant=False), [x], g), plain)
    with torch.autograd.graph.save_on_cpu():
        out = f(x)
    _same([out.detach(), *torch.autograd.grad(out, [x], g)], plain)


def test_checkpoint_around_more_than_the_layer():
    """The second forward runs inside the unpacking of the layer's tensors and has to record its own graph there."""
    m, wanted, g = _layer(torch.bfloat16, True, False, 64)
    first, last = (torch.nn.Linear(DIM, DIM, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    wanted = [*wanted, *first.parameters(), *last.parameters()]

    def f(x):
        return last(torch.nn.functional.gelu(m(first(x))))

    plain = _grads(f, wanted, g)
    _same(_grads(lambda t: checkpoint(f, t, use_reentrant=False), wanted, g), plain)


def test_hooks_that_change_a_tensor_are_refused():
    m, wanted, g = _layer(torch.bfloat16, False, False, 64)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.half() if t.dtype == torch.bfloat16 else t):
        out = m(wanted[0])
    with pytest.raises(RuntimeError, match="saved tensor came back"):
        torch.autograd.grad(out, wanted, g)


@pytest.mark.parametrize("change", ["device", "rows", "type"])
@pytest.mark.parametrize("prenorm,sizes", [(True, (DIM, 64 * H)), (True, (6 * 64 * H, DIM)), (True, (B, N, DIM)), (True, (B * N, DIM)),
                                           (True, (B * N, 64 * H)), (False, (B, N, DIM))])
def test_hooks_that_change_one_tensor_of_the_layer_are_refused(prenorm, sizes, change):
    """The weights, the input, the projection's input and the merged heads, one at a time, in a call whose products are the
    framework's own launches: they get addresses and would read host memory or past the end."""
    m, wanted, g = _layer(torch.float32, prenorm, False, 64)
    changed = []

    def unpack(t):
        if tuple(t.shape) != sizes:
            return t
        changed.append(t)
        return {"device": t.cpu, "rows": lambda: t[..., :-1, :], "type": t.half}[change]()

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        out = m(wanted[0])
    with pytest.raises(RuntimeError, match="saved tensor came back"):
        torch.autograd.grad(out, wanted, g)
    assert len(changed) == 1


def test_only_what_a_gradient_needs_is_guarded_against_changes():
    """As with the single operations: a frozen projection's input may change after the forward."""
    m, wanted, g = _layer(torch.bfloat16, False, False, 64)
    x = wanted[0].detach().clone()
    m.to_all_qkv.weight.requires_grad_(False)
    h = x.clone().requires_grad_()
    y = h * 1
    out = m(y)
    plain = torch.autograd.grad(m(h), [h, m.combine_heads.weight], g)
    with torch.no_grad():
        y.zero_()
    _same(torch.autograd.grad(out, [h, m.combine_heads.weight], g), plain)
