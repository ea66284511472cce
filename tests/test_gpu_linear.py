"""GPU: the small products of csrc/linear.cu against fp64, in every layout, at the edges of tiles and of the chunks of k."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# Sums in fp32 of exact products; a 16-bit result is rounded once (half a unit in the last place: 2^-9 and 2^-12 of a value, a
# third of that in the norm), an fp32 one differs by the rounding of the sums, which grows slower than sqrt(k) units of 2^-24.
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -9), (torch.float16, 2.0 ** -12), (torch.float32, 1e-6)])
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("m,n,k", [(1, 64, 64), (197, 3072, 512), (512, 768, 128), (128, 128, 512), (129, 72, 200), (512, 128, 776), (40, 200, 1000),
                                   (256, 1000, 136), (127, 65 * 8, 384), (8, 8, 8), (1024, 192, 40)])
def test_product(dtype, tol, layout, m, n, k):
    from lookahead_keys_attention_b200 import _lib as L, check_status, ops
    code = {torch.bfloat16: L.BF16, torch.float16: L.F16, torch.float32: L.F32}[dtype]
    if layout == 2:
        m = (m + 7) // 8 * 8
    torch.manual_seed(m + n + k)

    def matrix(rows, cols):   # rows further apart than they are long
        return torch.randn(rows, cols + 8, device="cuda").to(dtype)[:, :cols]
    a, b = matrix(k, m) if layout == 2 else matrix(m, k), matrix(n, k) if layout == 0 else matrix(k, n)
    c = torch.full((m + 1, n + 8), 7.0, device="cuda", dtype=dtype)
    L.check(L.load().castle_linear(code, layout, m, n, k, a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), c.data_ptr(), c.stride(0),
                                   ops.status_word("cuda").data_ptr(), None), "linear")
    ref = (a.double().T if layout == 2 else a.double()) @ (b.double().T if layout == 0 else b.double())
    assert (c[:m, :n].double() - ref).norm() <= tol * ref.norm()
    assert bool((c[m] == 7).all()) and bool((c[:, n:] == 7).all())
    check_status()


def test_refusals():
    from lookahead_keys_attention_b200 import _lib as L, ops
    lib, t, s = L.load(), torch.zeros(64, 64, device="cuda"), ops.status_word("cuda").data_ptr()

    def call(dtype=L.F32, layout=0, m=64, n=64, k=64, ld=64, ptr=t.data_ptr()):
        return lib.castle_linear(dtype, layout, m, n, k, ptr, ld, t.data_ptr(), ld, t.data_ptr(), ld, s, None)
    assert call(layout=3) != 0 and call(dtype=5) != 0 and call(m=0) != 0 and call(n=62) != 0 and call(k=62) != 0 and call(layout=2, m=62) != 0
    assert call(ld=60) != 0 and call(ld=66) != 0 and call(ptr=t.data_ptr() + 4) != 0 and call(ptr=None) != 0
