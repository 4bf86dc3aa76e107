"""The tensor-core kernels on lengths that are not whole tiles and on head dims below 128 (no padded copies: TMA fills in
zeros), forward and backward against the oracle: edges of the 64-key blocks and 128-row tiles, one and two tiles per CTA, histories,
strided [B, L, H, D] operands."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Lq,hist,D", [
    (1, 2, 1, 0, 128), (1, 2, 63, 0, 128), (1, 2, 64, 64, 128), (2, 2, 65, 0, 128), (1, 2, 127, 192, 128), (1, 2, 129, 0, 128),
    (1, 2, 257, 128, 128), (2, 80, 140, 0, 128), (1, 3, 200, 64, 64), (1, 2, 256, 0, 64), (1, 160, 300, 0, 64), (1, 2, 77, 0, 40),
    (1, 2, 190, 64, 96), (1, 1, 385, 320, 8)])
def test_ragged_lengths_and_small_heads(B, H, Lq, hist, D, dtype):
    g = torch.Generator().manual_seed(Lq + D)
    Lk = Lq + hist
    q, k, v = [(torch.randn(B, n, H, D, generator=g) * 0.5).to(dtype) for n in (Lq, Lk, Lk)]
    do = torch.randn(B, H, Lq, D, generator=g).to(dtype)
    qc, kc, vc = [t.to(DEV).transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    out = P.fused_landmark_attention(qc, kc, vc, None)
    grads = torch.autograd.grad(out, [qc, kc, vc], do.to(DEV))
    n = min(H, 3)                                          # the oracle on a few heads
    f = [t.transpose(1, 2)[:, -n:].float() for t in (q, k, v)]
    pad = -Lq % 64                                         # the oracle wants whole blocks: zero rows behind the real ones
    fp = [torch.nn.functional.pad(t, (0, 0, 0, pad)) for t in (*f, do[:, -n:].float())]
    exp = [t[:, :, :r] for t, r in zip(O.landmark_attention_grads(*fp, 64, sm_scale=D ** -0.5), (Lq, Lq, Lk, Lk))]
    for name, got, e in zip(("o", "dq", "dk", "dv"), (out, *grads), exp):
        got = got.detach()[:, -n:].float().cpu()
        assert torch.isfinite(got).all(), name
        assert (got - e).abs().max().item() < 2e-2 * max(1.0, e.abs().max().item()), name
        assert ((got - e).norm() / e.norm().clamp_min(1e-6)).item() < 1e-2 or e.norm() < 1e-3, name
    assert L.device_status() == 0


@pytest.mark.parametrize("form", ["heads", "batch", "rows", "offset", "features"])
@pytest.mark.parametrize("Lq,hist,D,blk", [(77, 64, 128, 64), (100, 0, 64, 32), (256, 0, 128, 64), (45, 0, 40, 2)])
def test_operands_that_tma_cannot_address(Lq, hist, D, blk, form):
    # they are copied: the same result as dense operands give, also where the sequence ends inside a block, and gradients of the views
    g = torch.Generator(device="cuda").manual_seed(Lq)
    B, H, Lk = 2, 3, Lq + hist
    def make(L):
        base = torch.randn(B, H, L, D, device="cuda", generator=g).to(torch.bfloat16)
        return {"heads": lambda: base[:, :1].expand(B, H, L, D), "batch": lambda: base[:1].expand(B, H, L, D),
                "rows": lambda: base[:, :, :1].expand(B, H, L, D),
                "offset": lambda: torch.cat((base.new_zeros(3), base.reshape(-1)))[3:].view(B, H, L, D),
                "features": lambda: torch.stack((base, base), -1).flatten(-2)[..., ::2]}[form]()
    q, k, v = make(Lq), make(Lk), make(Lk)
    do = torch.randn(B, H, Lq, D, device="cuda", generator=g).to(torch.bfloat16)
    runs = []
    for dense in (False, True):
        a = [t.contiguous().requires_grad_(True) if dense else t.requires_grad_(True) for t in (q.detach(), k.detach(), v.detach())]
        o = P.fused_landmark_attention(*a, None, block_size=blk)
        runs.append((o, *torch.autograd.grad(o, a, do)))
    for got, exp in zip(*runs):
        assert got.shape == exp.shape and torch.equal(got, exp)
