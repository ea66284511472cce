"""GPU: a layer's cached token as one launch (csrc/token_layer.cu) against the submodules and the step's own kernel, at the
edges of what it takes: CTAs of a cluster without rows, two rows per lane group, the last size that fits and the next one; and
against the oracle in fp64."""
import ctypes

import pytest
import torch

from oracle import castle_oracle as O

pytestmark = pytest.mark.gpu

BF16, F16, F32 = torch.bfloat16, torch.float16, torch.float32
# Both round the six new rows, the rewritten lookahead keys, the head outputs and the result to the type; sums run in fp32 in
# another order, so some of these roundings fall the other way: by one unit in the last place, less than that in the norm.
TOL = {BF16: 2.0 ** -8, F16: 2.0 ** -10, F32: 1e-5}


def _fits(dtype, B, H, d, t, dim, out):
    from lookahead_keys_attention_b200 import _lib as L
    code = {BF16: L.BF16, F16: L.F16, F32: L.F32}[dtype]
    return L.load().castle_token_layer_fits(ctypes.byref(L.CastleProblem(B, H, 1, d, code, d ** -0.5)), t, dim, out)


@pytest.mark.parametrize("dtype,B,H,d,t,dim,out,norm,rotary,fits", [
    (BF16, 1, 1, 32, 0, 8, 8, False, False, 1), (F32, 1, 1, 32, 1, 8, 13, True, True, 1), (F16, 1, 3, 64, 7, 24, 24, True, False, 1),
    (BF16, 1, 8, 64, 771, 512, 512, True, True, 1), (F32, 2, 8, 64, 129, 512, 512, False, False, 1), (F32, 5, 5, 64, 90, 320, 77, True, True, 1),
    (F32, 3, 15, 32, 33, 480, 480, False, True, 1), (BF16, 3, 7, 128, 250, 896, 100, True, False, 1), (F16, 1, 15, 128, 1000, 1920, 1920, False, True, 1),
    (BF16, 1, 2, 64, 2048, 128, 128, False, False, 1), (BF16, 1, 2, 64, 2049, 128, 128, False, False, 0), (F32, 2, 8, 64, 512, 512, 512, True, False, 1),
    (F32, 2, 8, 64, 513, 512, 512, True, False, 0), (BF16, 1, 4, 128, 1024, 4096, 8, False, False, 1), (BF16, 1, 16, 64, 10, 128, 128, False, False, 0),
    (BF16, 4, 8, 64, 10, 128, 128, False, False, 0), (F32, 1, 2, 128, 17, 2056, 8, False, False, 0), (BF16, 1, 2, 16, 17, 64, 64, False, False, 0)])
def test_one_launch_against_the_operators(dtype, B, H, d, t, dim, out, norm, rotary, fits):
    from lookahead_keys_attention_b200 import Castle, cache_from_buffers, check_status
    assert _fits(dtype, B, H, d, t, dim, out) == fits
    torch.manual_seed(t)
    m = Castle(dim, heads=H, dim_head=d, prenorm=norm, rotary_emb=rotary)
    m.combine_heads = torch.nn.Linear(H * d, out, bias=False)
    if norm:
        torch.nn.init.uniform_(m.norm.weight, 0.5, 1.5)
    m.to("cuda", dtype)
    x = torch.randn(B, 3, dim, device="cuda").to(dtype)
    bufs = [torch.randn(B, H, t + 4, d, device="cuda").to(dtype) for _ in range(4)]
    for b in bufs:
        b[:, :, t + 3] = 9   # the row behind the last one stays
    with torch.no_grad():
        new, old = cache_from_buffers(*[b.clone() for b in bufs], t), cache_from_buffers(*[b.clone() for b in bufs], t)
        for i in range(3):
            y, new = m(x[:, i:i + 1], cache=new)
            z, old = m._forward_operators(x[:, i:i + 1], old, True)
            assert y.shape == z.shape and (y.double() - z.double()).norm() <= TOL[dtype] * z.double().norm()
        for a, b in zip(new, old):
            assert (a.double() - b.double()).norm() <= TOL[dtype] * b.double().norm()
        assert all(bool((b[:, :, t + 3] == 9).all()) for b in new._state.bufs)
    check_status()


def test_nan_and_infinity_reach_the_output():
    from lookahead_keys_attention_b200 import Castle, cache_from_buffers
    torch.manual_seed(0)
    m = Castle(128, heads=2, dim_head=64).to("cuda", BF16)
    x = torch.randn(1, 1, 128, device="cuda").to(BF16)
    for value in (float("nan"), float("inf")):
        bufs = [torch.randn(1, 2, 70, 64, device="cuda").to(BF16) for _ in range(4)]
        bufs[2][0, 1, 33, 5] = value
        with torch.no_grad():
            y, _ = m(x, cache=cache_from_buffers(*bufs, 65))
        assert not bool(y.isfinite().all())


def _exact(m, x, caches, t):
    """The token in fp64 on the CPU, from the layer's weights and the caches as they are stored."""
    w = {k: v.double().cpu() for k, v in m.state_dict().items()}
    h = x.double().cpu()
    if "norm.weight" in w:
        h = torch.nn.functional.rms_norm(h, h.shape[-1:], w["norm.weight"], torch.finfo(torch.float32).eps)
    qu, ku, vu, qc, kc, vc = O.split_heads(h @ w["to_all_qkv.weight"].t(), m.heads)
    if m.rotary_emb is not None:
        ang = t * m.rotary_emb.freqs.double().cpu()

        def rotate(v):
            a, b = v[..., 0::2], v[..., 1::2]
            return torch.stack((a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()), -1).flatten(-2)
        qu, ku, vu, qc, kc = map(rotate, (qu, ku, vu, qc, kc))
    out, cache = O.castle_decode_step(qc, kc, vc, qu, ku, vu, O.Cache(*(c.double().cpu() for c in caches)), m.scale)
    return out.permute(0, 2, 1, 3).flatten(2) @ w["combine_heads.weight"].t(), cache


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("B,H,d,t,dim,norm,rotary", [(1, 1, 32, 0, 8, False, False), (1, 8, 64, 300, 512, True, True), (2, 8, 64, 128, 512, False, False),
                                                      (3, 5, 32, 33, 480, True, True), (1, 3, 128, 250, 896, True, False)])
def test_one_launch_against_fp64(dtype, B, H, d, t, dim, norm, rotary):
    from lookahead_keys_attention_b200 import Castle, cache_from_buffers, check_status
    assert _fits(dtype, B, H, d, t, dim, dim) == 1
    torch.manual_seed(dim + t)
    m = Castle(dim, heads=H, dim_head=d, prenorm=norm, rotary_emb=rotary)
    if norm:
        torch.nn.init.uniform_(m.norm.weight, 0.5, 1.5)
    m.to("cuda", dtype)
    x = torch.randn(B, 1, dim, device="cuda").to(dtype)
    bufs = [torch.randn(B, H, t + 4, d, device="cuda").to(dtype) for _ in range(4)]
    want, caches = _exact(m, x, [b[:, :, :t] for b in bufs], t)
    with torch.no_grad():
        y, new = m(x, cache=cache_from_buffers(*bufs, t))
    # Roundings to the type between x and the result, at most half a unit (u) each: the norm, the new rows, U, the head outputs and
    # the result, and u of a score moves a probability by no more than the row does; the rotation has four of its own (its cosines and
    # sines, two products, their sum), its angle another 2^-24 t.  fp32: the sums' order and exp, some ten units.
    u = {BF16: 2.0 ** -9, F16: 2.0 ** -12, F32: 4 * 2.0 ** -24}[dtype]
    tol = (6 + 4 * rotary) * u + rotary * t * 2.0 ** -24
    for a, b in zip((y, *new), (want, *caches)):
        assert a.shape == b.shape and (a.double().cpu() - b).norm() <= tol * b.norm()
    check_status()
