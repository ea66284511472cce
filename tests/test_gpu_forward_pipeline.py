"""GPU: the forward's dispatch - masked T tiles computed up front or inside the walk, walks whole or cut in two or three
parts, many short walks - against the oracle, output and lookahead keys."""
import pytest
import torch

from oracle import castle_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N,d", [
    (2, 3, 384, 64), (2, 3, 385, 64), (2, 3, 384, 128), (2, 3, 512, 128),      # three and four query blocks, T inside
    (1, 1, 1024, 64), (1, 1, 1023, 128), (1, 2, 1500, 64), (1, 2, 2049, 128),  # three parts
    (1, 12, 1100, 64), (1, 9, 1281, 128),                                      # two parts
    (3, 7, 1030, 64), (3, 7, 1030, 128),                                       # whole walks, more than one wave
    (38, 4, 257, 64), (30, 3, 641, 64), (100, 3, 1, 64),                       # many short walks
    (12, 4, 1500, 64), (28, 1, 2000, 64), (16, 1, 2750, 128)])                 # T up front: walk after walk, a CTA per walk
def test_forward_dispatch(B, H, N, d):
    from lookahead_keys_attention_b200 import castle_attention_packed, check_status
    torch.manual_seed(N + d)
    packed = (torch.randn(B, N, 6, H, d, device="cuda") * 3 ** -0.5).half()
    with torch.no_grad():
        out, U = castle_attention_packed(packed, d ** -0.5, True)
        again, _ = castle_attention_packed(packed, d ** -0.5, True)
    check_status()
    assert torch.equal(out, again)
    qu, ku, vu, qc, kc, vc = (packed[:, :, i].permute(0, 2, 1, 3).float() for i in range(6))
    for b in range(0, B, max(1, B // 3)):
        v = [t[b:b + 1] for t in (qc, kc, vc, qu, ku, vu)]
        ref, ref_u = O.castle_parallel(*v, d ** -0.5, return_U=True)
        assert ((out[b:b + 1].float() - ref).abs() - 5e-3 * ref.abs()).max().item() <= 5e-3
        assert ((U[b:b + 1].float() - ref_u).abs() - 5e-3 * ref_u.abs()).max().item() <= 5e-3 + 2 * 2.0 ** -10 * ref_u.abs().max().item()
