"""GPU: the transform pass over its ways of dividing lines between threads: one head and tensor, widths whose threads do not fill
a block, more lines than a block takes at once, more heads than the multiplication replaces a division for."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N,d,dd,count", [(1, 1, 1, 8, 8, 1), (1, 1, 700, 64, 64, 1), (2, 1, 33, 24, 64, 6), (1, 3, 5, 40, 64, 6), (1, 7, 129, 128, 72, 2),
                                              (1, 16, 1201, 128, 128, 6), (1, 40000, 1, 8, 16, 1), (2, 5, 2, 120, 128, 5)])
@pytest.mark.parametrize("src,dst", [("bf16", "fp16"), ("fp32", "bf16"), ("fp16", "fp32")])
def test_lines(src, dst, B, H, N, d, dd, count):
    from lookahead_keys_attention_b200 import _lib as L
    types = {"bf16": (torch.bfloat16, L.BF16), "fp16": (torch.float16, L.F16), "fp32": (torch.float32, L.F32)}
    (st, sc), (dt, dc) = types[src], types[dst]
    torch.manual_seed(N)
    x = (torch.randn(B, N, count, H, d, device="cuda") * 100).to(st)
    y = torch.full((B, N, count, H, dd + 8), 7.0, device="cuda").to(dt)

    def descriptors(t):
        return (L.CastleTensor * 6)(*[L.CastleTensor(t[:, :, i].data_ptr(), t.stride(0), t.stride(3), t.stride(1)) for i in range(count)])
    a, b, mul = descriptors(x), descriptors(y), torch.tensor([0.5], device="cuda")
    p = L.CastleProblem(B, H, N, d, sc, 1.0)
    L.check(L.load().castle_transform(ctypes.byref(p), count, ctypes.cast(a, ctypes.POINTER(L.CastleTensor)), ctypes.cast(b, ctypes.POINTER(L.CastleTensor)), dc, dd,
                                      None, None, 0, mul.data_ptr(), None), "transform")
    want = torch.zeros(B, N, count, H, dd, device="cuda")
    w = min(d, dd)
    want[..., :w] = x[..., :w].float() * 0.5
    assert bool((y[..., :dd] == want.to(dt)).all()) and bool((y[..., dd:] == 7).all())
