"""GPU: RMSNorm's two gradients where one pass makes them and where two do, at the edges of its columns and row ranges, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# a 16-bit result is rounded once (half a unit in the last place at most); in fp32 the sums' roundings remain, some sqrt(terms) of them
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11), (torch.float32, 1e-6)])
@pytest.mark.parametrize("rows,dim", [(1, 8), (7, 248), (31, 256), (33, 264), (65, 504), (2369, 512), (100, 520), (20000, 512), (40001, 64)])
def test_norm_gradients(dtype, tol, rows, dim):
    from lookahead_keys_attention_b200 import _lib as L
    lib, code = L.load(), {torch.bfloat16: L.BF16, torch.float16: L.F16, torch.float32: L.F32}[dtype]
    torch.manual_seed(rows)
    x, dy = (torch.randn(rows, dim, device="cuda").to(dtype) for _ in range(2))
    w, rstd = (torch.rand(dim, device="cuda") + 0.5).to(dtype), torch.rand(rows, device="cuda") + 0.5
    ws = torch.empty(lib.castle_rmsnorm_bwd_workspace_bytes(rows, dim), dtype=torch.uint8, device="cuda")

    def run(want_dx, want_dw):
        dx, dw = torch.full_like(x, 7.0), torch.full_like(w, 7.0)
        L.check(lib.castle_rmsnorm_bwd(code, rows, dim, dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(),
                                       dx.data_ptr() if want_dx else None, dw.data_ptr() if want_dw else None, ws.data_ptr(), ws.numel(), None), "bwd")
        return dx.double(), dw.double()

    dx, dw = run(True, True)
    r, d, xd = rstd.double()[:, None], dy.double(), x.double()
    gx = r * (d * w.double() - xd * r * r * (d * w.double() * xd).mean(-1, keepdim=True))
    gw = (d * xd * r).sum(0)
    for got, want in ((dx, gx), (dw, gw), (run(True, False)[0], gx), (run(False, True)[1], gw)):
        assert (got - want).norm() <= tol * want.norm()
    again = run(True, True)
    assert torch.equal(again[0], dx) and torch.equal(again[1], dw)
