"""A backward kernel may start while the kernel in front of it is still running: dQ reads the row statistics and the output that the
forward writes, or the table of landmark groups that a kernel of its own works out, dK/dV reads delta = rowsum(O * dO) that dQ
writes.  All of that is scratch memory or fresh memory of the allocator,
which may hold anything, or the right values of a call before.  So: calls whose memory holds NaNs, many times, against the oracle and
bit by bit against one another."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as lib
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
CALLS = 50


def poison(*sizes):
    """Frees blocks of exactly these sizes (bytes) full of NaNs: the allocator hands them to the requests of these sizes that follow."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for n in (*sizes, 64 << 20)]
    del held


def first_difference(name, a, b):
    at = [int(i) for i in (a != b).nonzero()[0]]
    return f"{name} differs first at batch {at[0]}, head {at[1]}, tile {at[2] // 128}, row {at[2]}, feature {at[3]}"


def check_calls(call, sizes, names=("o", "dq", "dk", "dv")):
    """The tensors of the first call; the others have to give the same bits."""
    first = None
    for i in range(CALLS):
        poison(*sizes)
        got = [t.detach().clone() for t in call()]
        for name, t in zip(names, got):
            assert torch.isfinite(t).all(), f"call {i}: {name} not finite"
        if first is None:
            first = got
        for name, a, b in zip(names, first, got):
            assert torch.equal(a, b), f"call {i}: " + first_difference(name, a, b)
    assert lib.device_status() == 0
    return dict(zip(names, first))


def close(got, exp, what):
    # P and dS are rounded to 16 bits in front of the products and the results behind them: the bound of the other kernel tests
    got = got.float().cpu()
    assert (got - exp).abs().max().item() < 2e-2 * max(1.0, exp.abs().max().item()), what
    assert ((got - exp).norm() / exp.norm()).item() < 1e-2, what


@pytest.mark.parametrize("B,H,L,D", [(1, 32, 2048, 128), (4, 16, 1024, 64)])
def test_first_backward_into_poisoned_scratch(B, H, L, D):
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = [(torch.randn(B, H, L, D, generator=g, device="cuda") * 0.5).bfloat16().requires_grad_(True) for _ in range(3)]
    do = torch.randn(B, H, L, D, generator=g, device="cuda").bfloat16()

    def call():
        out = P.fused_landmark_attention(q, k, v, None, block_size=64)
        return (out, *torch.autograd.grad(out, [q, k, v], do))

    rows, data = 4 * B * H * L, 2 * B * H * L * D
    got = check_calls(call, [2 * rows, rows, data, data, data, data])        # L and M, delta, o, dq, dk, dv
    for b, h in ((0, 0), (B - 1, H - 1)):
        one = [t[b:b + 1, h:h + 1].detach().float().cpu() for t in (q, k, v, do)]
        for (name, t), e in zip(got.items(), O.landmark_attention_grads(*one, 64, sm_scale=D ** -0.5)):
            close(t[b:b + 1, h:h + 1], e, f"{name}, batch {b}, head {h}")


@pytest.mark.parametrize("B,H,L,D", [(64, 16, 256, 64), (16, 32, 256, 128), (8, 64, 384, 64), (32, 16, 449, 96), (64, 32, 64, 64)])
def test_units_with_few_key_blocks(B, H, L, D):
    # dQ units whose key blocks all fit the stages: the next unit's tiles are loaded as soon as the rows in shared memory are read
    g = torch.Generator(device="cuda").manual_seed(L + D)
    q, k, v = [(torch.randn(B, H, L, D, generator=g, device="cuda") * 0.5).bfloat16().requires_grad_(True) for _ in range(3)]
    do = torch.randn(B, H, L, D, generator=g, device="cuda").bfloat16()
    first = None
    for i in range(300):
        out = P.fused_landmark_attention(q, k, v, None, block_size=64)
        got = (out.detach(), *torch.autograd.grad(out, [q, k, v], do))
        first = first or got
        for name, a, b in zip(("o", "dq", "dk", "dv"), first, got):
            assert torch.equal(a, b), f"call {i}: " + first_difference(name, a, b)
    pad = -L % 64                                          # the oracle wants whole blocks: zero rows behind the real ones
    for b, h in ((0, 0), (B - 1, H - 1)):
        one = [torch.nn.functional.pad(t[b:b + 1, h:h + 1].detach().float().cpu(), (0, 0, 0, pad)) for t in (q, k, v, do)]
        for name, t, e in zip(("o", "dq", "dk", "dv"), first, O.landmark_attention_grads(*one, 64, sm_scale=D ** -0.5)):
            close(t[b:b + 1, h:h + 1], e[:, :, :L], f"{name}, batch {b}, head {h}")
    assert lib.device_status() == 0


def test_groups_into_poisoned_scratch():
    B, H, T, D, G = 16, 8, 512, 128, 16
    g = torch.Generator().manual_seed(5)
    q, k, v = [(torch.randn(B, H, T, D, generator=g) * 0.5).bfloat16() for _ in range(3)]
    do = torch.randn(B, H, T, D, generator=g).bfloat16()
    im = (torch.arange(T).view(1, T) + torch.randint(0, 51, (B, 1), generator=g)) % 51 == 50
    im[5] = False                                          # no landmark: a row for the two-pass kernels
    qc, kc, vc = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    doc, imc = do.cuda(), im.cuda()

    def call():
        out = P.landmark_attention_masked(qc, kc, vc, imc, max_groups=G)
        return (out, *torch.autograd.grad(out, [qc, kc, vc], doc))

    rows, data = 4 * B * H * T, 2 * B * H * T * D
    ws = int(lib.lib().lmk_attn_mask_bwd_workspace(B, H, T, G))               # delta, sums of the groups, tile table
    got = check_calls(call, [rows, G * rows, ws, data, data, data, data])    # R, A, o, dq, dk, dv
    for b, h in ((0, 0), (5, 3), (B - 1, H - 1)):
        f = [t[b:b + 1, h:h + 1].float().requires_grad_(True) for t in (q, k, v)]
        out = O.lm_attention(*f, im[b:b + 1])
        exp = (out.detach(), *torch.autograd.grad(out, f, do[b:b + 1, h:h + 1].float()))
        for (name, t), e in zip(got.items(), exp):
            close(t[b:b + 1, h:h + 1], e, f"{name}, batch {b}, head {h}")
