"""Forward on both sides of the lines between one and two query tiles a CTA: by sequence length for blocks of 64, for heads of 64
features and for groups as key tiles, and by the size of the grid."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Lq,D,block", [
    (40, 768, 128, 64), (40, 896, 128, 64), (1, 896, 128, 64), (40, 833, 128, 64),      # six and seven tiles, few and many heads
    (8, 4096, 64, 64), (8, 4224, 64, 64),                                               # 32 and 33 tiles
    (20, 1536, 128, 32), (20, 1664, 128, 32),                                           # twelve and thirteen tiles
    (9, 4096, 64, 64), (9, 4224, 64, 64),                                               # 32 and 33 tiles, two an SM and more
    (20, 1920, 128, 32), (20, 2000, 128, 32), (18, 2048, 128, 32),                      # 15 and 16 tiles, few and many heads
    (20, 2048, 64, 32), (20, 2080, 64, 32), (17, 2080, 64, 32)])                        # 16 and 17 tiles
def test_both_sides_of_the_tile_lines(H, Lq, D, block):
    g = torch.Generator().manual_seed(Lq + H)
    q, k, v = [(torch.randn(1, H, Lq, D, generator=g) * 0.5).to(torch.bfloat16) for _ in range(3)]
    out = P.fused_landmark_attention(q.cuda(), k.cuda(), v.cuda(), None, block_size=block)
    pad = -Lq % block                                      # the oracle wants whole blocks: zero rows behind the real ones
    f = [torch.nn.functional.pad(t.float(), (0, 0, 0, pad)) for t in (q, k, v)]
    for h in {0, H // 2, H - 1}:                           # (a head at a time: the oracle holds its scores)
        one = [t[:, h:h + 1] for t in f]
        exp = O.landmark_attention_grads(*one, torch.zeros_like(one[0]), block, sm_scale=D ** -0.5)[0][:, :, :Lq]
        got = out[:, h:h + 1].float().cpu()
        # weights rounded to 16 bits in front of the product, the result behind it: the bound of the other kernel tests
        assert (got - exp).abs().max().item() < 2e-2, h
        assert ((got - exp).norm() / exp.norm()).item() < 1e-2, h
    assert L.device_status() == 0
