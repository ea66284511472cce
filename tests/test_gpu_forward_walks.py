"""GPU: dim_head-64 forward whose CTAs take one walk after the other against single pairs in calls of their own, where a CTA has one
walk: output, lookahead keys and the rows stored for a decode cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)])
# pairs x blocks: 148 and 149 walks, two and three turns of the CTAs, one block each, masked last blocks, T tiles inside and up front, the
# longest walks of the rule; first, for each number of blocks below eight, the last problem with a CTA per walk and the first without
@pytest.mark.parametrize("B,H,N", [(1, 148, 77), (3, 25, 250), (6, 9, 384), (5, 11, 380), (2, 23, 511), (1, 47, 512), (4, 10, 640), (1, 41, 639), (5, 7, 768), (4, 9, 760), (1, 31, 896), (4, 8, 890),
                                   (2, 37, 256), (1, 149, 77), (1, 297, 128), (3, 99, 300), (5, 30, 1000), (7, 19, 1153), (3, 45, 1665), (2, 40, 3072)])
def test_walk_after_walk_matches_single_walks(dtype, tol, B, H, N):
    from lookahead_keys_attention_b200 import castle_attention, check_status
    torch.manual_seed(N)
    ts = [(torch.randn(B, H, N, 64, device="cuda") * 3 ** -0.5).to(dtype) for _ in range(6)]
    bufs = [torch.full((B, H, N + 3, 64), 7.0, device="cuda", dtype=dtype) for _ in range(4)]
    with torch.no_grad():
        out, _ = castle_attention(*ts, 64 ** -0.5, True, cache_out=[b[:, :, :N] for b in bufs])
        for b, h in [(0, 0), (B // 2, H // 3), (B - 1, H - 2), (B - 1, H - 1)]:
            ref, U = castle_attention(*[t[b:b + 1, h:h + 1] for t in ts], 64 ** -0.5, True)
            # the same tiles in the same order; a T tile that is computed elsewhere or a state in parts may round a 16-bit value the other way
            for got, want in ((out, ref), (bufs[0], U)):
                assert (got[b, h, :N].double() - want[0, 0].double()).norm() <= tol * want.double().norm()
    for buf, t in zip(bufs[1:], (ts[3], ts[1], ts[2])):
        assert torch.equal(buf[:, :, :N], t)
    assert all(bool((buf[:, :, N:] == 7.0).all()) for buf in bufs)
    check_status()
