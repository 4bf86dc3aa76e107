"""One key that is not finite, at every column of a block in turn (a head each): its score reaches the output and the gradients of the
rows behind it whichever way the exponential of its column is computed, and no row in front of it."""
import pytest
import torch

import landmark_attention_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("block,D,dtype", [(64, 64, torch.bfloat16), (64, 128, torch.float16), (51, 128, torch.bfloat16)])
def test_key_that_is_not_finite(block, D, dtype, bad):
    H, L = block - 1, 256
    g = torch.Generator(device="cuda").manual_seed(block + D)
    q, k, v = [torch.randn(1, H, L, D, generator=g, device="cuda").to(dtype) for _ in range(3)]
    do = torch.randn(1, H, L, D, generator=g, device="cuda").to(dtype)
    q[..., 0] = 1                                          # +inf times 1: a score of +inf
    im = torch.arange(L, device="cuda").view(1, L) % block == block - 1

    def call(k):
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        out = P.fused_landmark_attention(*t, None, block_size=64) if block == 64 else P.landmark_attention_masked(*t, im, max_groups=16)
        return (out.detach(), *torch.autograd.grad(out, t, do))

    clean = call(k)
    heads = torch.arange(H, device="cuda")
    k[0, heads, block + heads, 0] = bad                    # head h: column h of the second block
    out, dq, dk, dv = call(k)
    last = 2 * block
    assert all(torch.isfinite(t).all() for t in clean)
    for h in range(H):
        assert torch.equal(out[0, h, :block + h], clean[0][0, h, :block + h]), h
        assert out[0, h, block + h:last - 1].isnan().all() and out[0, h, last:].isnan().all(), h
        assert dq[0, h, last:].isnan().all(), h
        # every key of the block shares its rows' sum (its landmark, the last one, has no value of its own)
        assert dk[0, h, block:last].isnan().all() and dv[0, h, block:last - 1].isnan().all(), h
