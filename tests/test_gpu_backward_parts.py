"""GPU: dim_head-128 backward with its long walks cut in two parts (few pairs) against the same pairs in a call of many, whose
walks are whole."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)])
@pytest.mark.parametrize("B,H,N", [(1, 1, 769), (1, 2, 896), (2, 1, 1001), (1, 3, 1333), (1, 2, 2177)])
def test_cut_walks_match_whole_ones(dtype, tol, B, H, N):
    from lookahead_keys_attention_b200 import castle_attention, check_status
    torch.manual_seed(N)
    few = [(torch.randn(B, H, N, 128, device="cuda") * 3 ** -0.5).to(dtype) for _ in range(6)]
    g = torch.randn(B, H, N, 128, device="cuda").to(dtype)
    copies = -(-160 // (B * H))   # more than 148 pairs: nothing is cut
    outs = []
    for ts, grad in ((few, g), ([t.repeat(copies, 1, 1, 1) for t in few], g.repeat(copies, 1, 1, 1))):
        ts = [t.requires_grad_() for t in ts]
        outs.append(torch.autograd.grad(castle_attention(*ts, 128 ** -0.5), ts, grad))
    # The parts form the same tiles and sum them in fp32; two sums instead of one round a 16-bit result the other way now and then.
    for name, a, b in zip(("dqc", "dkc", "dvc", "dqu", "dku", "dvu"), *outs):
        b = b[:B]
        assert (a.double() - b.double()).norm() <= tol * b.double().norm(), name
    check_status()
