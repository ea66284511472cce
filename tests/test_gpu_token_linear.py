"""GPU: one token's norm and projection as one launch (csrc/token_linear.cu) against torch in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,k,n", [(1, 8, 1), (1, 512, 3072), (2, 520, 17), (3, 96, 2400), (5, 1000, 64), (8, 3072, 129), (4, 40, 15), (6, 264, 7000)])
@pytest.mark.parametrize("norm", [False, True])
def test_token_linear(dtype, rows, k, n, norm):
    from lookahead_keys_attention_b200 import _lib as L
    code = {torch.bfloat16: L.BF16, torch.float16: L.F16, torch.float32: L.F32}[dtype]
    torch.manual_seed(n)
    wide = torch.randn(rows, k + 8, device="cuda").to(dtype)
    x, w = wide[:, :k], (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype)
    g, eps = torch.rand(k, device="cuda").to(dtype) + 0.5, 1e-3
    y = torch.full((rows + 1, n), 7.0, device="cuda", dtype=dtype)
    L.check(L.load().castle_token_linear(code, rows, k, n, x.data_ptr(), k + 8, g.data_ptr() if norm else None, eps,
                                         w.data_ptr(), y.data_ptr(), 0, None), "token_linear")
    h = torch.nn.functional.rms_norm(x, (k,), g, eps) if norm else x
    ref = h.double() @ w.double().T
    tol = {torch.bfloat16: 2e-2, torch.float16: 3e-3, torch.float32: 2e-5}[dtype]
    assert (y[:rows].double() - ref).abs().max().item() <= tol * max(1.0, ref.abs().max().item())
    assert bool((y[rows] == 7).all())


def test_token_linear_refuses_what_does_not_fit():
    from lookahead_keys_attention_b200 import _lib as L
    lib = L.load()
    assert lib.castle_token_linear_fits(L.F32, 8, 3072) and not lib.castle_token_linear_fits(L.F32, 9, 64)
    assert not lib.castle_token_linear_fits(L.F32, 8, 3080) and not lib.castle_token_linear_fits(L.F32, 1, 12)
    assert lib.castle_token_linear_fits(L.BF16, 8, 8192) and not lib.castle_token_linear_fits(L.BF16, 9, 64)
    assert not lib.castle_token_linear_fits(L.BF16, 8, 16384)
