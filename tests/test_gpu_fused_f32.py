"""The tiled fp32 kernels (blocks of 64) against the oracle: edges of the 32-row tiles, histories, odd head dims, one and several key
blocks per cluster, strided operands and gradients; and gradients that arrive as [B, L, H, D] views in 16 bits."""
import pytest
import torch

import landmark_attention_b200 as P
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,H,Lq,hist,D", [(2, 2, 64, 0, 64), (1, 3, 256, 128, 128), (1, 2, 320, 64, 40), (1, 1, 128, 0, 104),
                                           (2, 1, 192, 320, 64), (1, 2, 64, 0, 8)])
def test_f32_forward_and_backward(B, H, Lq, hist, D):
    g = torch.Generator().manual_seed(Lq + D)
    Lk = Lq + hist
    q, k, v, do = [torch.randn(B, n, H, D, generator=g).transpose(1, 2) for n in (Lq, Lk, Lk, Lq)]
    qc, kc, vc = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
    out = P.fused_landmark_attention(qc, kc, vc, None)
    grads = torch.autograd.grad(out, [qc, kc, vc], do.to(DEV))
    exp = O.landmark_attention_grads(q, k, v, do, 64)
    for name, got, e in zip(("o", "dq", "dk", "dv"), (out, *grads), exp):
        assert (got.detach().cpu() - e).abs().max().item() < 1e-4, name
    again = torch.autograd.grad(P.fused_landmark_attention(qc, kc, vc, None), [qc, kc, vc], do.to(DEV))
    assert all(torch.equal(a, b) for a, b in zip(again, grads))


@pytest.mark.parametrize("Lq,hist", [(1, 0), (33, 64), (95, 0), (130, 128)])
def test_f32_ragged_forward(Lq, hist):
    g = torch.Generator().manual_seed(Lq)
    q, k, v = [torch.randn(1, 2, n, 64, generator=g) for n in (Lq, Lq + hist, Lq + hist)]
    out = P.fused_landmark_attention(q.to(DEV), k.to(DEV), v.to(DEV), None)
    pad = [torch.nn.functional.pad(t, (0, 0, 0, -Lq % 64)) for t in (q, k, v)]
    exp = O.landmark_attention(*pad, 64, sm_scale=0.125)[:, :, :Lq]
    assert (out.cpu() - exp).abs().max().item() < 1e-4


@pytest.mark.parametrize("masked", [False, True])
def test_strided_gradient_equals_the_dense_one(masked):
    g = torch.Generator(device=DEV).manual_seed(3)
    q, k, v = [torch.randn(2, 3, 256, 128, generator=g, device=DEV).bfloat16().requires_grad_(True) for _ in range(3)]
    do = torch.randn(2, 256, 3, 128, generator=g, device=DEV).bfloat16().transpose(1, 2)
    im = (torch.arange(256, device=DEV).view(1, 256) + torch.tensor([[3], [200]], device=DEV)) % 51 == 50
    im[1] = False                                              # one row of each kernel family
    call = (lambda: P.landmark_attention_masked(q, k, v, im, max_groups=8)) if masked else (lambda: P.fused_landmark_attention(q, k, v))
    a = torch.autograd.grad(call(), [q, k, v], do)
    b = torch.autograd.grad(call(), [q, k, v], do.contiguous())
    assert all(torch.equal(x, y) for x, y in zip(a, b))
