"""GPU: exceptions keep their types on the way through the native host path (csrc/host.cpp)."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu


class Refused(Exception):
    pass


def _refuse(t):
    raise Refused("no")


@pytest.mark.parametrize("layer", [False, True])
def test_an_exception_of_a_hook_keeps_its_type(layer):
    from lookahead_keys_attention_b200 import Castle, castle_attention_packed
    if layer:
        f = Castle(96, heads=2, prenorm=True).cuda().bfloat16()
        x = torch.randn(1, 130, 96, device="cuda").bfloat16().requires_grad_()
    else:
        f = lambda t: castle_attention_packed(t, 0.125)   # noqa: E731
        x = torch.randn(1, 130, 6, 2, 64, device="cuda").bfloat16().requires_grad_()
    with pytest.raises(Refused), torch.autograd.graph.saved_tensors_hooks(_refuse, lambda t: t):
        f(x)


def test_checkpoint_may_stop_the_second_forward_early():
    """Non-reentrant checkpointing ends its recomputation with an exception out of the last hook it needs."""
    from lookahead_keys_attention_b200 import castle_attention_packed
    x = torch.randn(1, 130, 6, 2, 64, device="cuda").bfloat16().requires_grad_()
    g = torch.randn(1, 2, 130, 64, device="cuda").bfloat16()
    plain = torch.autograd.grad(castle_attention_packed(x, 0.125), x, g)[0]
    again = torch.autograd.grad(checkpoint(castle_attention_packed, x, 0.125, use_reentrant=False), x, g)[0]
    assert (again.float() - plain.float()).norm().item() <= 4e-3 * plain.float().norm().item()   # dqc is summed in arrival order


def test_out_of_memory_keeps_its_type():
    from lookahead_keys_attention_b200 import castle_attention_packed, check_status, release_workspaces
    x = torch.randn(1, 8192, 6, 16, 64, device="cuda").half()   # 600 MB of scratch
    with torch.no_grad():
        release_workspaces()
        torch.cuda.empty_cache()
        assert torch.cuda.memory_reserved() - torch.cuda.memory_allocated() < 256 << 20
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / total)
        try:
            with pytest.raises(torch.OutOfMemoryError):
                castle_attention_packed(x, 0.125)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        castle_attention_packed(x, 0.125)   # nothing is left half made
    check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,N", [(0, 40), (2, 0), (0, 1)])
def test_empty_tensors_are_refused(dtype, B, N):
    from lookahead_keys_attention_b200 import Castle, castle_attention, castle_attention_packed
    x = torch.zeros(B, 2, N, 64, device="cuda", dtype=dtype)
    with pytest.raises(RuntimeError):
        castle_attention(x, x, x, x, x, x, 0.125)
    with pytest.raises(RuntimeError):
        castle_attention_packed(torch.zeros(B, N, 6, 2, 64, device="cuda", dtype=dtype), 0.125)
    with pytest.raises(RuntimeError):
        Castle(32, heads=2).cuda().to(dtype)(torch.zeros(B, N, 32, device="cuda", dtype=dtype))


@pytest.mark.parametrize("dual", ["x", "to_all_qkv", "norm"])
def test_forward_mode_differentiation_is_refused(dual):
    """Instead of dropping the tangent."""
    import torch.autograd.forward_ad as fwAD
    from lookahead_keys_attention_b200 import Castle, castle_attention_packed
    m = Castle(32, heads=2, prenorm=True).cuda().requires_grad_(False)
    x = torch.randn(2, 40, 32, device="cuda")
    with fwAD.dual_level():
        weights = {}
        if dual == "x":
            x = fwAD.make_dual(x, torch.ones_like(x))
        else:
            w = getattr(m, dual).weight.detach().clone()
            weights = {dual + ".weight": fwAD.make_dual(w, torch.ones_like(w))}
        with pytest.raises(NotImplementedError, match="forward-mode"):
            torch.func.functional_call(m, weights, (x,))
        p = torch.randn(1, 40, 6, 2, 64, device="cuda")
        with pytest.raises(NotImplementedError, match="forward-mode"):
            castle_attention_packed(fwAD.make_dual(p, p), 0.125)


def test_tensors_of_another_device_are_refused():
    from lookahead_keys_attention_b200 import Castle, cache_from_buffers, castle_attention, castle_attention_packed, castle_decode_step
    z = lambda n, dev="cuda": torch.zeros(2, 2, n, 64, device=dev, dtype=torch.bfloat16)   # noqa: E731
    new, caches = [z(1) for _ in range(6)], [z(40) for _ in range(4)]
    for i in range(4):
        with pytest.raises(RuntimeError, match="device"):
            castle_decode_step(*new, *[z(40, "cpu") if j == i else c for j, c in enumerate(caches)], 30, 0.125)
    for i in range(1, 6):
        with pytest.raises(RuntimeError, match="device"):
            castle_decode_step(*[z(1, "cpu") if j == i else t for j, t in enumerate(new)], *caches, 30, 0.125)
    with pytest.raises(RuntimeError, match="device"):   # pinned host memory, too: the step's bulk copies do not read it
        castle_decode_step(*new, *[z(40, "cpu").pin_memory() for _ in range(4)], 30, 0.125)
    six = [z(40) for _ in range(6)]
    out = [z(40)] * 3 + [z(40, "cpu")]
    with pytest.raises(RuntimeError, match="device"):
        castle_attention(*six, 0.125, True, out)
    with pytest.raises(RuntimeError, match="device"):
        castle_attention_packed(torch.zeros(2, 40, 6, 2, 64, device="cuda", dtype=torch.bfloat16), 0.125, True, out)
    with torch.no_grad():
        m, x = Castle(32, heads=2).cuda().bfloat16(), torch.zeros(2, 1, 32, device="cuda", dtype=torch.bfloat16)
        with pytest.raises(RuntimeError, match="device"):
            m(x, cache=cache_from_buffers(*[z(40, "cpu") for _ in range(4)], 30))
