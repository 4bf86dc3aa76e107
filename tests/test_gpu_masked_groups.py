"""Landmark groups as key tiles: groups of up to 64 keys at odd offsets, adjacent landmarks, landmarks on the first and last
key, an empty open group, key histories, batches that mix rows of both kernel families, and regular blocks below 64 with
ragged lengths and small heads."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L
from oracle import landmark_oracle as O
from test_gpu_masked import compare, make, oracle, run

pytestmark = pytest.mark.gpu
DEV = "cuda"


def flags_at(B, T, *rows):
    im = torch.zeros(B, T, dtype=torch.bool)
    for b, at in enumerate(rows):
        im[b, list(at)] = True
    return im


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_groups_of_every_kind(dtype):
    B, H, T = 4, 2, 256
    g, q, k, v, do = make(B, H, T, dtype, 23)
    im = flags_at(B, T, range(63, T, 64),                                  # 64-key groups, the last key a landmark
                  [0, 1, 40, 41, 42, 105, 168, 231],                       # first keys, adjacent ones, 63-key gaps
                  [17, 60, 124, 188, 252],                                 # 64-key groups at an offset, a short open group
                  [])                                                      # no landmark: the other kernel family
    compare(run(q, k, v, do, im, 16), oracle(q, k, v, do, im), "groups")
    assert L.device_status() == 0


@pytest.mark.parametrize("T,blk", [(128, 26), (384, 51), (640, 33), (1024, 26), (1024, 64)])
def test_windows_of_many_lengths(T, blk):
    B, H = 3, 2
    g, q, k, v, do = make(B, H, T, torch.bfloat16, T + blk)
    off = torch.randint(0, blk, (B, 1), generator=g)
    im = (torch.arange(T).view(1, T) + off) % blk == blk - 1
    compare(run(q, k, v, do, im, min(64, T // blk + 2)), oracle(q, k, v, do, im), f"{T} {blk}")
    assert L.device_status() == 0


def test_many_units_per_cta():
    B, H, T = 5, 7, 384
    g, q, k, v, do = make(B, H, T, torch.bfloat16, 3)
    off = torch.randint(0, 51, (B, 1), generator=g)
    im = (torch.arange(T).view(1, T) + off) % 51 == 50
    im[2] = False                                                          # skipped units in the middle of the walk
    ref = run(q, k, v, do, im, 10)
    L.lib().lmk_debug_set_max_ctas(3)
    try:
        got = run(q, k, v, do, im, 10)
    finally:
        L.lib().lmk_debug_set_max_ctas(0)
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
    compare(ref, oracle(q, k, v, do, im), "units")


@pytest.mark.parametrize("Lq,hist,D,blk", [(200, 32, 128, 32), (77, 0, 64, 32), (300, 48, 128, 16), (1000, 320, 128, 32),
                                           (130, 90, 96, 45), (64, 0, 64, 2)])
def test_regular_blocks_below_64(Lq, hist, D, blk):
    g = torch.Generator().manual_seed(Lq)
    B, H, Lk = 2, 3, Lq + hist
    q, k, v = [(torch.randn(B, n, H, D, generator=g) * 0.5).to(torch.bfloat16) for n in (Lq, Lk, Lk)]
    do = torch.randn(B, H, Lq, D, generator=g).to(torch.bfloat16)
    qc, kc, vc = [t.to(DEV).transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    out = P.fused_landmark_attention(qc, kc, vc, None, block_size=blk)
    grads = torch.autograd.grad(out, [qc, kc, vc], do.to(DEV))
    pad = -Lq % blk
    f = [torch.nn.functional.pad(t, (0, 0, 0, pad)) for t in (*[t.transpose(1, 2).float() for t in (q, k, v)], do.float())]
    exp = [t[:, :, :r] for t, r in zip(O.landmark_attention_grads(*f, blk, sm_scale=D ** -0.5), (Lq, Lq, Lk, Lk))]
    for name, got, e in zip(("o", "dq", "dk", "dv"), (out, *grads), exp):
        got = got.detach().float().cpu()
        assert (got - e).abs().max().item() < 2e-2 * max(1.0, e.abs().max().item()), name
        assert ((got - e).norm() / e.norm()).item() < 1.2e-2, name
    assert L.device_status() == 0
