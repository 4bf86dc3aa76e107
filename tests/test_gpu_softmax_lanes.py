"""Grouped softmax rows with at most two landmarks in one lane's keys: shared memory holds the row, one segmented scan a pass
reduces all groups.  Edges: row lengths around the pieces of 4, 128 and 512 keys, landmarks on the first and last key of a
lane, rows with no landmark, two landmarks in a lane, rows that fall back because three share one, unaligned rows."""
import pytest
import torch

from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _grad_tol(dtype):
    return 2e-5 if dtype == torch.float32 else 2e-2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Lk", [1, 5, 128, 129, 300, 512, 513, 1000, 1025, 2047, 2048])
@pytest.mark.parametrize("guards", [True, False])
def test_sparse_landmarks(Lk, dtype, guards):
    import landmark_attention_b200 as P
    g = torch.Generator().manual_seed(Lk)
    B, H, Lq, k = 2, 3, 6, 4 * -(-Lk // 128)
    is_mem = torch.zeros(B, 1, Lq, Lk, dtype=torch.bool)
    for r in range(1, Lq):                                         # row 0 has no landmark
        is_mem[:, :, r, (k - 1 if r % 2 else 2 * k)::3 * k] = True
    is_mem[..., 0] = False
    if Lk > 8:
        is_mem[:, :, Lq - 1, 4:7:2] = k > 7                        # two landmarks in one lane: a group between them
        is_mem[:, :, Lq - 2, 1:6:2] = k > 7                        # three: the other form
    last = torch.zeros_like(is_mem)
    last[..., Lk - max(1, Lk // 5):] = True
    last &= ~is_mem
    hidden = (torch.rand(1, 1, Lq, Lk, generator=g) < 0.2) & ~last & ~is_mem if guards else None
    x = (torch.randn(B, H, Lq, Lk, generator=g) * 3).to(dtype)
    if guards:
        x = x.masked_fill(hidden, float("-inf"))
    gp = torch.randn(B, H, Lq, Lk, generator=g)
    n = int(is_mem.sum(-1).max()) + 2
    xo = x.float().requires_grad_(True)
    exp = O.grouped_softmax(xo, is_mem, last, attn_mask=hidden, guards=guards)
    (gx_exp,) = torch.autograd.grad(exp, [xo], gp)
    xd = x.to(DEV).requires_grad_(True)
    if guards:
        got, group = P.landmark_grouped_softmax_lm(xd, -1, is_mem.to(DEV), hidden.to(DEV), last.to(DEV), True, n)
        inner = torch.cumsum(is_mem.to(torch.int64), -1)
        for c in range(n - 1):
            member = (inner == c) & ~(is_mem | last | hidden)
            want = (exp * member).sum(-1)
            seen = member.expand_as(exp).any(-1)                   # a landmark without keys has a weight but no members
            assert (group[..., c].cpu() - want)[seen].abs().max().item() < 1e-5 if seen.any() else True
    else:
        got = P.landmark_grouped_softmax(xd, -1, is_mem.to(DEV), last.to(DEV), max_groups=n)
    assert (got.detach().cpu() - exp.detach()).abs().max().item() < 2e-6
    (gx,) = torch.autograd.grad(got, [xd], gp.to(DEV))
    assert gx.dtype == dtype and (gx.float().cpu() - gx_exp).abs().max().item() < _grad_tol(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Lk,block", [(1064, 32), (2048, 32), (1500, 51), (2047, 64), (700, 12)])
@pytest.mark.parametrize("guards", [True, False])
def test_regular_groups(Lk, block, dtype, guards):
    import landmark_attention_b200 as P
    g = torch.Generator().manual_seed(Lk + block)
    B, H, Lq = 1, 4, 3
    row = (torch.arange(Lk) % block == block - 1).view(1, Lk).expand(B, Lk)
    mask, is_mem, last = P.prepare_landmark_masks(row, torch.ones(Lq, Lk, dtype=torch.bool).triu(Lk - Lq - 200))
    x = (torch.randn(B, H, Lq, Lk, generator=g) * 3).to(dtype)
    x = x.masked_fill(mask, float("-inf") if guards else torch.finfo(dtype).min)
    gp = torch.randn(B, H, Lq, Lk, generator=g)
    xo = x.float().requires_grad_(True)
    exp = O.grouped_softmax(xo, is_mem, last, attn_mask=mask if guards else None, guards=guards)
    (gx_exp,) = torch.autograd.grad(exp, [xo], gp)
    xd, n = x.to(DEV).requires_grad_(True), Lk // block + 3
    if guards:
        got, group = P.landmark_grouped_softmax_lm(xd, -1, is_mem.to(DEV), mask.to(DEV), last.to(DEV), True, n)
        _, group_exp = O.grouped_softmax(xo, is_mem, last, attn_mask=mask, guards=True, return_group_prob=True, max_mem_cnt=n)
        assert (group.cpu() - group_exp.detach()).abs().max().item() < 2e-6
    else:
        got = P.landmark_grouped_softmax(xd, -1, is_mem.to(DEV), last.to(DEV))
    assert (got.detach().cpu() - exp.detach()).abs().max().item() < 2e-6
    (gx,) = torch.autograd.grad(got, [xd], gp.to(DEV))
    assert (gx.float().cpu() - gx_exp).abs().max().item() < _grad_tol(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Lq,Lk", [(1, 1), (40, 40), (129, 129), (200, 515), (1, 2048), (300, 1100)])
def test_causal_rows(Lq, Lk, dtype):
    import landmark_attention_b200 as P
    g = torch.Generator().manual_seed(Lk)
    B, H, block = 2, 2, max(2, Lk // 14)
    flags = (torch.arange(Lk).view(1, Lk) + torch.tensor([[0], [3]])) % block == block - 1
    x = (torch.randn(B, H, Lq, Lk, generator=g) * 3).to(dtype)
    gp = torch.randn(B, H, Lq, Lk, generator=g)
    mask, is_mem, last = P.prepare_landmark_masks(flags, torch.ones(Lq, Lk, dtype=torch.bool).triu(Lk - Lq + 1))
    xo = x.float().requires_grad_(True)
    exp = O.grouped_softmax(xo.masked_fill(mask, float("-inf")), is_mem, last, attn_mask=mask, guards=True)
    (gx_exp,) = torch.autograd.grad(exp, [xo], gp)
    xd = x.to(DEV).requires_grad_(True)
    got = P.landmark_grouped_softmax_causal(xd, flags.to(DEV), int(flags.sum(-1).max()) + 2)
    assert (got.detach().cpu() - exp.detach()).abs().max().item() < 2e-6
    (gx,) = torch.autograd.grad(got, [xd], gp.to(DEV))
    assert (gx.float().cpu() - gx_exp).abs().max().item() < _grad_tol(dtype)
