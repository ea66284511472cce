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


# pairs x blocks of eight, chunk: all chunks cut as the whole call is; none in the whole call, all in chunks; the last chunk alone
@pytest.mark.parametrize("H,chunk,same", [(5, 2, 5), (18, 10, 0), (18, 17, 17)])
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)])
def test_cut_walks_in_chunks_of_the_pairs(monkeypatch, dtype, tol, H, chunk, same):
    """A smaller workspace runs the pairs in chunks; each decides by its own pairs whether its walks are cut, and the parts' sums
    are found by the pair's number in the whole call."""
    from lookahead_keys_attention_b200 import castle_attention, check_status, ops
    N, d = 1001, 128
    torch.manual_seed(H)
    ts = [(torch.randn(1, H, N, d, device="cuda") * 3 ** -0.5).to(dtype).requires_grad_() for _ in range(6)]
    g = torch.randn(1, H, N, d, device="cuda").to(dtype)
    out = castle_attention(*ts, d ** -0.5)
    whole = torch.autograd.grad(out, ts, g)
    sums, pair = (H * N * (3 * d + 1) * 4 + 1023) // 1024 * 1024, 8 * 9 // 2 * 3 * 32768
    monkeypatch.setattr(ops, "MAX_WORKSPACE_BYTES", sums + chunk * pair + 512)
    ops.release_workspaces()
    out = castle_attention(*ts, d ** -0.5)
    chunked = torch.autograd.grad(out, ts, g)
    ops.release_workspaces()
    check_status()
    for name, a, b in zip(("dqc", "dkc", "dvc", "dqu", "dku", "dvu"), chunked, whole):
        if name != "dqc":   # added in arrival order; the others by their owner, the same way where the walks are the same
            assert torch.equal(a[:, :same], b[:, :same]), name
        # two fp32 sums instead of one round a 16-bit result the other way now and then
        assert (a.double() - b.double()).norm() <= tol * b.double().norm(), name
