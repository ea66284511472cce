"""GPU: the dim_head-64 backward's walks, whose products, tiles and passes are issued by different warps - one block, two, odd and
even numbers of steps, ragged last blocks, more CTAs than one wave - against the oracle's gradients of every pair;
the three gradients that a CTA owns repeat bit for bit, the three that are summed repeat up to the order of the sums."""
import pytest
import torch

from oracle import castle_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N", [(1, 1, 17), (1, 2, 128), (2, 1, 129), (1, 3, 384), (1, 1, 901), (4, 12, 640)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_backward_d64(B, H, N, dtype):
    from lookahead_keys_attention_b200 import castle_attention_packed, check_status
    torch.manual_seed(N)
    d = 64
    packed = (torch.randn(B, N, 6, H, d, device="cuda") * 3 ** -0.5).to(dtype).requires_grad_()
    go = torch.randn(B, H, N, d, device="cuda").to(dtype)
    grads = [torch.autograd.grad(castle_attention_packed(packed, d ** -0.5), [packed], go)[0] for _ in range(2)]
    check_status()
    for i in (0, 4, 5):   # dqu, dkc, dvc
        assert torch.equal(grads[0][:, :, i], grads[1][:, :, i]), i
    for i in (1, 2, 3):   # dku, dvu, dqc: fp32 sums over up to 8 key blocks in arrival order
        # a sum is off by 8 units of 2^-24 of its terms' magnitudes, some 16 times its own, so a share f = 8 * 16 * 2^-24 / u of the results rounds
        # the other way, by u = 2^-8 (2^-11) of itself: u * sqrt(f) = 1.7e-4 (6e-5) of the norm
        a, b = grads[0][:, :, i].float(), grads[1][:, :, i].float()
        assert (a - b).norm().item() <= (1.7e-4 if dtype == torch.bfloat16 else 6e-5) * b.norm().item(), i
    v = [packed[:, :, i].detach().permute(0, 2, 1, 3).float().requires_grad_() for i in (3, 4, 5, 0, 1, 2)]
    ref = torch.autograd.grad(O.castle_parallel(*v, d ** -0.5), v, go.float())
    for r, i in zip(ref, (3, 4, 5, 0, 1, 2)):
        g = grads[0][:, :, i].permute(0, 2, 1, 3).float()
        # operands of 8 or 11 bits through some six roundings, each half a unit of the last place at most; of every pair
        off = (g - r).flatten(2).norm(dim=2) / r.flatten(2).norm(dim=2)
        assert off.max().item() <= (1.2e-2 if dtype == torch.bfloat16 else 4e-3), i
