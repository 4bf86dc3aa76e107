"""The chunk's rows behind a retrieved prefix (lmk_cached_rows) against the oracle's grouped softmax over the concatenated scores: rows
that are not a multiple of the 16-row tiles, 16-key steps or 64-key tiles, prefixes of every remainder of four, landmarks in the prefix,
several landmarks within one lane's keys (evenly spaced, at random, next to each other), rows whose own key is a landmark, more landmarks
than groups."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,T,n_pre,every,strided", [
    (2, 3, 255, 204, 51, True), (1, 2, 1, 7, 4, False), (1, 2, 33, 64, 16, True), (2, 1, 130, 33, 5, False), (1, 2, 64, 130, 3, True),
    (1, 1, 500, 606, 64, False), (1, 2, 250, 102, 51, True)])
def test_rows_behind_a_prefix(B, H, T, n_pre, every, strided, dtype):
    g = torch.Generator().manual_seed(T * 7 + n_pre)
    rnd = lambda *s: torch.randn(*s, generator=g)
    if strided:
        q, k, v = [rnd(B, T, H, 128).to(dtype).transpose(1, 2) for _ in range(3)]
    else:
        q, k, v = [rnd(B, H, T, 128).to(dtype) for _ in range(3)]
    pre, vals = rnd(B, H, T, n_pre).to(dtype), rnd(B, H, T, n_pre, 128).to(dtype)
    flags = (torch.arange(T).view(1, T) + torch.arange(B).view(B, 1)) % every == every - 1
    pre_mem = torch.zeros(B, n_pre, dtype=torch.bool)
    pre_mem[:, every - 1::every] = True
    groups = int(flags.sum(-1).max() + pre_mem.sum(-1).max()) + 2
    scale = 128 ** -0.5
    att = ((q.float() @ k.float().transpose(-1, -2)).to(dtype).float() * scale).to(dtype)
    att = torch.cat((pre, att), dim=-1).float()
    row = torch.cat((pre_mem, flags), dim=-1)
    hidden = torch.ones(T, n_pre + T, dtype=torch.bool).triu(n_pre + 1)
    mask, is_mem, last = P.prepare_landmark_masks(row, hidden)
    p = O.grouped_softmax(att.masked_fill(mask, float("-inf")), is_mem, last, attn_mask=mask, guards=True).to(dtype).float()
    exp = p[..., n_pre:] @ v.float() + (p[..., :n_pre].unsqueeze(3) @ vals.float()).squeeze(3)
    dev = [x.to(DEV) for x in (q, k, v, pre, vals, row)]
    assert L.lib().lmk_cached_rows_supported(128, T, n_pre, L.dtype_code(dev[0])) == 1
    got = L.host().cached_attend(*dev, groups, scale)
    assert got is not None
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert (got.float().cpu() - exp).abs().max().item() < tol * max(1.0, exp.abs().max().item())
    assert ((got.float().cpu() - exp).norm() / exp.norm()).item() < (6e-3 if dtype == torch.bfloat16 else 8e-4)
    y = P.lm_landmark_attention(dev[0], dev[1], dev[2], flags.to(DEV), max_groups=groups, att_prefix=dev[3],
                                cache_values={"v": dev[4], "is_mem": pre_mem.to(DEV)})
    assert torch.equal(y, got)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,n_pre,density", [(130, 33, 0.5), (255, 204, 0.1), (64, 900, 0.03), (300, 1100, 0.06), (200, 1700, 0.4), (40, 61, 1.0)])
def test_landmarks_anywhere(T, n_pre, density, dtype):
    g = torch.Generator().manual_seed(T + n_pre)
    B, H = 2, 2
    q, k, v = [torch.randn(B, H, T, 128, generator=g).to(dtype) for _ in range(3)]
    # groups of very different levels: each needs a maximum of its own
    level = torch.repeat_interleave(torch.randn(B, 1, 1, n_pre // 7 + 1, generator=g) * 40, 7, -1)[..., :n_pre]
    pre = (torch.randn(B, H, T, n_pre, generator=g) + level).to(dtype)
    vals = torch.randn(B, H, T, n_pre, 128, generator=g).to(dtype)
    row = torch.rand(B, n_pre + T, generator=g) < density
    groups = int(row.sum(-1).max()) + 2
    att = ((q.float() @ k.float().transpose(-1, -2)).to(dtype).float() * 128 ** -0.5).to(dtype)
    att = torch.cat((pre, att), dim=-1).float()
    mask, is_mem, last = P.prepare_landmark_masks(row, torch.ones(T, n_pre + T, dtype=torch.bool).triu(n_pre + 1))
    p = O.grouped_softmax(att.masked_fill(mask, float("-inf")), is_mem, last, attn_mask=mask, guards=True).to(dtype).float()
    exp = p[..., n_pre:] @ v.float() + (p[..., :n_pre].unsqueeze(3) @ vals.float()).squeeze(3)
    got = L.host().cached_attend(*[x.to(DEV) for x in (q, k, v, pre, vals, row)], groups, 128 ** -0.5)
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert got is not None and (got.float().cpu() - exp).abs().max().item() < tol * max(1.0, exp.abs().max().item())
    # (with landmarks alone nothing has a weight: the output is zero)
    assert (got.float().cpu() - exp).norm().item() <= (6e-3 if dtype == torch.bfloat16 else 8e-4) * exp.norm().item()
    assert L.device_status() == 0


@pytest.mark.parametrize("every", [40, 3])               # one landmark a lane, several
def test_more_landmarks_than_groups_are_reported(every):
    q, k, v = [torch.randn(1, 2, 64, 128, device=DEV).to(torch.bfloat16) for _ in range(3)]
    pre, vals = torch.randn(1, 2, 64, 200, device=DEV).to(torch.bfloat16), torch.randn(1, 2, 64, 200, 128, device=DEV).to(torch.bfloat16)
    row = (torch.arange(264, device=DEV) % every == every - 1).view(1, 264)
    out = L.host().cached_attend(q, k, v, pre, vals, row, 3, 128 ** -0.5)
    assert L.device_status() == 501 and torch.isfinite(out).all() and L.device_status() == 0
