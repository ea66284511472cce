"""GPU: the layer's native path (csrc/host.cpp, csrc/norm.cu) - RMSNorm against torch in fp64, and the whole module's
gradients against the same module forced through its submodules, where autograd differentiates each operation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 264), (33, 512), (1000, 96), (257, 4096)])
def test_rmsnorm(dtype, rows, dim):
    from lookahead_keys_attention_b200 import _lib as L
    lib, code, eps = L.load(), {torch.bfloat16: L.BF16, torch.float16: L.F16, torch.float32: L.F32}[dtype], 1e-3
    torch.manual_seed(dim)
    x, dy = (torch.randn(rows, dim, device="cuda").to(dtype) for _ in range(2))
    w = (torch.rand(dim, device="cuda") + 0.5).to(dtype)
    y, dx, dw, rstd = torch.empty_like(x), torch.empty_like(x), torch.empty_like(w), torch.empty(rows, device="cuda")
    ws = torch.empty(lib.castle_rmsnorm_bwd_workspace_bytes(rows, dim), dtype=torch.uint8, device="cuda")
    L.check(lib.castle_rmsnorm_fwd(code, rows, dim, x.data_ptr(), w.data_ptr(), eps, y.data_ptr(), rstd.data_ptr(), None), "fwd")
    L.check(lib.castle_rmsnorm_bwd(code, rows, dim, dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
                                   dw.data_ptr(), ws.data_ptr(), ws.numel(), None), "bwd")
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    yd = torch.nn.functional.rms_norm(xd, (dim,), wd, eps)
    gx, gw = torch.autograd.grad(yd, [xd, wd], dy.double())
    tol = {torch.bfloat16: 1e-2, torch.float16: 2e-3, torch.float32: 1e-5}[dtype]
    for a, b in ((y, yd), (dx, gx), (dw, gw)):
        assert (a.double() - b).abs().max().item() <= tol * max(1.0, b.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("prenorm,rotary,d", [(False, False, 64), (True, False, 128), (True, True, 64), (False, True, 32)])
@pytest.mark.parametrize("frozen", [(), ("x",), ("to_all_qkv",), ("combine_heads",), ("x", "to_all_qkv", "norm")])
def test_layer_gradients_match_the_submodules(dtype, prenorm, rotary, d, frozen):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(d)
    m = Castle(96, heads=2, dim_head=d, prenorm=prenorm, rotary_emb=rotary).cuda().to(dtype)
    for n, p in m.named_parameters():
        p.requires_grad_(n.split(".")[0] not in frozen)
    x = torch.randn(3, 150, 96, device="cuda").to(dtype).transpose(0, 1).contiguous().transpose(0, 1).requires_grad_("x" not in frozen)
    g = torch.randn(3, 150, 96, device="cuda").to(dtype)
    wanted = [t for t in (x, *m.parameters()) if t.requires_grad]

    def go():
        out = m(x)
        return [out.detach(), *torch.autograd.grad(out, wanted, g)]

    native = go()
    handle = m.to_all_qkv.register_forward_hook(lambda *a: None)   # a hook makes the module call its submodules
    assert m._plain_layer() is None
    single = go()
    handle.remove()
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-3
    for a, b in zip(native, single):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert (a.float() - b.float()).norm().item() <= tol * b.float().norm().item()


def test_layer_backward_twice_and_inplace_change_raise():
    from lookahead_keys_attention_b200 import Castle
    m = Castle(64, heads=1).cuda()
    x = torch.randn(1, 40, 64, device="cuda", requires_grad=True)
    out = m(x)
    out.sum().backward(retain_graph=True)
    first = x.grad.clone()
    out.sum().backward()
    assert torch.allclose(x.grad, 2 * first, atol=1e-3)
    with pytest.raises(RuntimeError, match="second time"):
        out.sum().backward()
    out = m(x)
    with torch.no_grad():
        m.combine_heads.weight.mul_(2)
    with pytest.raises(RuntimeError, match="inplace"):
        out.sum().backward()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("prenorm", [False, True])
@pytest.mark.parametrize("batch", [1, 3, 12])
def test_input_at_an_odd_offset(dtype, prenorm, batch):
    """A contiguous view that starts between 16-byte boundaries: prompt with gradients, and single tokens on each route."""
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(batch)
    m = Castle(96, heads=2, prenorm=prenorm).cuda().to(dtype)
    g = torch.randn(batch, 40, 96, device="cuda").to(dtype)
    flat = torch.randn(batch * 40 * 96 + 1, device="cuda").to(dtype)
    token = torch.randn(batch * 96 + 1, device="cuda").to(dtype)

    def go(x, t):
        x = x.detach().requires_grad_()
        out, cache = m(x, return_next_cache=True)
        grads = torch.autograd.grad(out, [x, *m.parameters()], g)
        with torch.no_grad():
            step, _ = m(t, cache=cache)
        return [out.detach(), step, *grads]

    odd, even = (flat[1:].view(batch, 40, 96), token[1:].view(batch, 1, 96)), (flat[1:].clone().view(batch, 40, 96), token[1:].clone().view(batch, 1, 96))
    assert odd[0].data_ptr() % 16 and odd[1].data_ptr() % 16 and odd[0].is_contiguous()
    for a, b in zip(go(*odd), go(*even)):
        assert (a.float() - b.float()).norm().item() <= 4e-3 * b.float().norm().item()


@pytest.mark.parametrize("n", [140, 600])   # products of the framework's own, and the library's, which autocast would change
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("prenorm", [False, True])
def test_backward_under_autocast(dtype, prenorm, n):
    from lookahead_keys_attention_b200 import Castle
    torch.manual_seed(n)
    m = Castle(96, heads=2, prenorm=prenorm).cuda().to(dtype)
    x, g = (torch.randn(2, n, 96, device="cuda").to(dtype) for _ in range(2))
    wanted = [x.requires_grad_(), *m.parameters()]
    out = m(x)
    plain = torch.autograd.grad(out, wanted, g, retain_graph=True)
    for other in (torch.float16, torch.bfloat16):
        with torch.autocast("cuda", dtype=other):
            got = torch.autograd.grad(out, wanted, g, retain_graph=True)
        for a, b in zip(got, plain):   # the same launches; dqc, dku and dvu are added in arrival order
            assert a.dtype == b.dtype and (a.float() - b.float()).norm().item() <= 4e-3 * b.float().norm().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_lazily_negated_tensors(dtype):
    """Their memory holds the values without the sign (as the imaginary part of a conjugate does)."""
    from lookahead_keys_attention_b200 import Castle, castle_attention, castle_decode_step
    torch.manual_seed(0)
    lazy = torch._neg_view
    m = Castle(96, heads=2, prenorm=True).cuda().to(dtype)
    six = [(torch.randn(2, 2, 140, 64, device="cuda") * 3 ** -0.5).to(dtype) for _ in range(6)]
    x, g = (torch.randn(2, 140, 96, device="cuda").to(dtype) for _ in range(2))
    gs, rows = torch.randn(2, 2, 140, 64, device="cuda").to(dtype), [torch.randn(2, 2, 1, 64, device="cuda").to(dtype) for _ in range(6)]

    def go(neg):
        a = neg(x.clone()).requires_grad_()
        out, cache = m(a, return_next_cache=True)
        grads = torch.autograd.grad(out, [a, *m.parameters()], neg(g))
        with torch.no_grad():
            step, _ = m(neg(x[:, :1].clone()), cache=cache)
        ts = [neg(t.clone()).requires_grad_() for t in six]
        y = castle_attention(*ts, 0.125)
        return [out.detach(), step, *grads, y.detach(), *torch.autograd.grad(y, ts, neg(gs)),
                castle_decode_step(*[neg(r) for r in rows], *[torch.ones(2, 2, 9, 64, device="cuda", dtype=dtype) for _ in range(4)], 8, 0.125)]

    for a, b in zip(go(lazy), go(torch.neg)):   # single operations around the lazily negated input: 16-bit roundings that fall the other way
        assert (a.float() - b.float()).norm().item() <= 2e-2 * b.float().norm().item()
