"""GPU: the element-wise passes around the parallel kernels (csrc/transform.cu) and the rotated, self-merging decode
step, against the same arithmetic in torch operations and the oracle."""
import ctypes

import pytest
import torch

from oracle import castle_oracle as O

pytestmark = pytest.mark.gpu

CODES = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


@pytest.mark.parametrize("src,dst,B,H,N,d,dd,rotary", [
    (torch.float32, torch.float16, 2, 3, 130, 64, 64, False), (torch.bfloat16, torch.float16, 1, 5, 77, 128, 128, True),
    (torch.bfloat16, torch.bfloat16, 1, 1, 1, 24, 64, True), (torch.float16, torch.float32, 3, 2, 33, 64, 40, False),
    (torch.float32, torch.float16, 1, 40, 9, 96, 128, True), (torch.float16, torch.bfloat16, 2, 7, 2049, 128, 128, False)])
def test_transform(src, dst, B, H, N, d, dd, rotary):
    """Rotation, copies, factor, conversion, cut and zero-padded rows; strided sources and destinations."""
    from lookahead_keys_attention_b200 import _lib as L
    from lookahead_keys_attention_b200.castle import _Rotary
    from lookahead_keys_attention_b200.ops import _desc
    lib = L.load()
    torch.manual_seed(N)
    x = (torch.randn(B, N, 6, H, d, device="cuda") * 2).to(src)
    x.view(-1)[0] = 7e4 if src != torch.float16 else 6e4
    out = torch.full((B, N, 6, H, dd), 9.0, device="cuda", dtype=dst)
    copies = torch.full((2, B, H, N + 3, d), 9.0, device="cuda", dtype=src)
    mul = torch.tensor([0.25], device="cuda")
    rot = _Rotary(d).cuda().to(src)
    view = lambda t, i: t[:, :, i].permute(0, 2, 1, 3)
    arr = lambda ts: (L.CastleTensor * 6)(*ts)
    none = L.CastleTensor(None, 0, 0, 0)
    r = L.CastleRotary(rot.freqs.data_ptr(), CODES[src], 0, 5)
    prob = L.CastleProblem(B, H, N, d, CODES[src], 1.0)
    cs = arr([_desc(copies[0][:, :, :N]), none, none, none, _desc(copies[1][:, :, :N]), none])
    rc = lib.castle_transform(ctypes.byref(prob), 6, arr([_desc(view(x, i)) for i in range(6)]),
                              arr([_desc(view(out, i)) for i in range(6)]), CODES[dst], dd, cs,
                              ctypes.byref(r) if rotary else None, 0x1f, mul.data_ptr(), None)
    L.check(rc, "castle_transform")
    for i in range(6):
        y = rot.rotate(view(x, i), 5) if rotary and i != 5 else view(x, i)
        if i in (0, 4):
            c = copies[0 if i == 0 else 1]
            assert torch.equal(c[:, :, :N], y) and bool((c[:, :, N:] == 9).all())
        e = y.float() * 0.25
        e = torch.nn.functional.pad(e, (0, dd - d)) if dd > d else e[..., :dd]
        if dst == torch.float16 and src != dst:
            e = e.clamp(-65504, 65504)
        assert torch.equal(view(out, i), e.to(dst)), i


def test_transform_inverse_rotation():
    from lookahead_keys_attention_b200 import _lib as L
    from lookahead_keys_attention_b200.castle import _Rotary
    from lookahead_keys_attention_b200.ops import _desc
    x = torch.randn(2, 3, 50, 64, device="cuda")
    rot = _Rotary(64).cuda()
    y, z = rot.rotate(x, 0), torch.empty_like(x)
    prob, r = L.CastleProblem(2, 3, 50, 64, 2, 1.0), L.CastleRotary(rot.freqs.data_ptr(), 2, 1, 0)
    L.check(L.load().castle_transform(ctypes.byref(prob), 1, ctypes.byref(_desc(y)), ctypes.byref(_desc(z)), 2, 64, None,
                                      ctypes.byref(r), 1, None, None), "castle_transform")
    assert torch.allclose(x, z, atol=1e-5)


@pytest.mark.parametrize("dtype", list(CODES))
@pytest.mark.parametrize("n,top", [(8, 1.0), (1 << 20, 63.9), (4096, 64.0), (4096, 1e-12), (800, 0.0)])
def test_amax_scale(dtype, n, top):
    from lookahead_keys_attention_b200 import _lib as L
    x = (torch.rand(n, device="cuda") * 0.9 * top).to(dtype)
    x[n // 2] = -top
    amax = x.abs().max().float().clamp_min(1e-30)
    s = torch.ldexp(torch.ones_like(amax), (torch.frexp(64.0 / amax)[1] - 1).clamp(-24, 24))
    state, out = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.empty(2, device="cuda")
    for _ in range(2):   # the second call finds the words as the first one left them
        L.check(L.load().castle_amax_scale(CODES[dtype], x.data_ptr(), n, state.data_ptr(), out.data_ptr(), None), "amax")
        assert out.tolist() == [s.item(), 1 / s.item()] and state.tolist() == [0, 0]


@pytest.mark.parametrize("d,dtype", [(16, torch.bfloat16), (32, torch.float16), (64, torch.bfloat16), (64, torch.float32),
                                     (128, torch.bfloat16)])
@pytest.mark.parametrize("t", [1, 31, 33, 64, 500])
@torch.no_grad()
def test_rotary_decode_step_with_fine_splits(d, dtype, t):
    """The module's cached step with rotary (rotated in the kernel, rows cut finely, merged by the last CTA of a pair)
    against the oracle on rows rotated by torch operations; two steps, so that the counters are used twice."""
    from lookahead_keys_attention_b200 import Castle, cache_from_buffers, check_status
    torch.manual_seed(t)
    B, H, dim = 2, 3, 64
    m = Castle(dim, heads=H, dim_head=d, rotary_emb=True).cuda().to(dtype)
    bufs = [torch.randn(B, H, t + 2, d, device="cuda").to(dtype) * 0.5 for _ in range(4)]
    ref = O.Cache(*(b[:, :, :t].float().cpu() for b in bufs))
    cache = cache_from_buffers(*bufs, t)
    x = torch.randn(B, 2, dim, device="cuda").to(dtype)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    for i in range(2):
        out, cache = m(x[:, i:i + 1], cache=cache)
        qu, ku, vu, qc, kc, vc = m._split(m.to_all_qkv(x[:, i:i + 1]))
        qc, kc, qu, ku, vu = (m.rotary_emb.rotate(v, t + i) for v in (qc, kc, qu, ku, vu))
        ro, ref = O.castle_decode_step(*[v.float().cpu() for v in (qc, kc, vc, qu, ku, vu)], ref, m.scale)
        ro = m.combine_heads(ro.permute(0, 2, 1, 3).reshape(B, 1, H * d).cuda().to(dtype))
        assert (out.float() - ro.float()).abs().max().item() <= 2 * tol
        assert torch.allclose(cache.U.float().cpu(), ref.U, atol=2 * tol, rtol=1e-2)
        atol = 1e-4 if dtype == torch.float32 else 2e-2   # the projection of one token may be summed in another order
        assert torch.allclose(cache.qu_cache[:, :, t + i].float(), qu[:, :, 0].float(), atol=atol)
        ref = O.Cache(*(c.float().cpu() for c in cache))
    check_status()
