"""GPU: a layer's cached token as one launch (csrc/token_layer.cu) against the submodules and the step's own kernel, at the
edges of what it takes: CTAs of a cluster without rows, two rows per lane group, the last size that fits and the next one."""
import ctypes

import pytest
import torch

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
