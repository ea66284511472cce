"""GPU: the cached step where its rule for splitting rows over CTAs changes: one wave or several, shares at the bound, parts of
unequal length, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# U and out are rounded once to the type, the gate comes from __expf (2 units of 2^-23 of its argument's size) in fp32 sums: half
# a unit in the last place, in fp32 some 1e-6 of the norm
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float32, 5e-6)])
@pytest.mark.parametrize("B,H,t,d", [(1, 128, 1025, 64), (2, 74, 1100, 128), (4, 50, 2049, 64), (1, 400, 520, 32), (37, 16, 257, 64), (1, 300, 4000, 16),
                                     (6, 100, 130, 128), (1, 160, 1999, 64), (2, 64, 2100, 128)])
def test_step_over_splits(dtype, tol, B, H, t, d):
    from lookahead_keys_attention_b200 import castle_decode_step, check_status
    torch.manual_seed(t)
    scale = d ** -0.5
    qc, kc, vc, qu, ku, vu = [(torch.randn(B, H, 1, d, device="cuda") * 3 ** -0.5).to(dtype) for _ in range(6)]
    bufs = [(torch.randn(B, H, t + 2, d, device="cuda") * 3 ** -0.5).to(dtype) for _ in range(4)]
    U, quc, kcc, vcc = [b[:, :, :t].double() for b in bufs]
    out = castle_decode_step(qc, kc, vc, qu, ku, vu, *bufs, t, scale)
    gate = torch.sigmoid(scale * (quc * ku.double()).sum(-1, keepdim=True))
    U = (U + gate * vu.double()).to(dtype).double()
    su = scale * (U * qc.double()).sum(-1)
    s = torch.cat([scale * (kcc * qc.double()).sum(-1) - su * torch.sigmoid(su), scale * (kc.double() * qc.double()).sum(-1)], -1)
    ref = torch.softmax(s, -1).unsqueeze(2) @ torch.cat([vcc, vc.double()], 2)
    assert (out.double() - ref).norm() <= tol * ref.norm()
    assert (bufs[0][:, :, :t].double() - U).norm() <= tol * U.norm()
    for b, row in zip(bufs, (torch.zeros_like(qu), qu, kc, vc)):
        assert bool((b[:, :, t:t + 1] == row).all())
    check_status()
