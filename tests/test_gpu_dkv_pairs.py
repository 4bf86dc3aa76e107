"""dK / dV units of two key blocks, for head dims of one and two 64-feature sub-tiles: sequences whose last pair has one block,
units of a single query tile, key histories, and CTAs that walk through one or many units (the same bits whatever their number)."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,H,Lq,hist,D,dtype", [
    (1, 3, 320, 0, 64, torch.bfloat16), (2, 2, 192, 64, 64, torch.float16), (1, 5, 128, 192, 64, torch.bfloat16),
    (1, 3, 320, 0, 128, torch.float16), (2, 3, 64, 64, 128, torch.bfloat16), (1, 4, 384, 320, 128, torch.bfloat16),
    (1, 4, 449, 64, 48, torch.bfloat16), (1, 2, 449, 0, 112, torch.float16)])
def test_units_of_key_block_pairs(B, H, Lq, hist, D, dtype):
    g = torch.Generator().manual_seed(Lq + hist + D)
    Lk = Lq + hist
    q, k, v = [(torch.randn(B, H, n, D, generator=g) * 0.5).to(dtype) for n in (Lq, Lk, Lk)]
    do = torch.randn(B, H, Lq, D, generator=g).to(dtype)

    def run(cap):
        L.lib().lmk_debug_set_max_ctas(cap)
        try:
            qc, kc, vc = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
            out = P.fused_landmark_attention(qc, kc, vc, None, block_size=64)
            return torch.autograd.grad(out, [qc, kc, vc], do.to(DEV))
        finally:
            L.lib().lmk_debug_set_max_ctas(0)

    ref = run(0)
    for cap in (1, 2, 5):
        assert all(torch.equal(a, b) for a, b in zip(run(cap), ref)), cap
    pad = -Lq % 64                                         # the oracle wants whole blocks: zero rows behind the real ones
    fp = [torch.nn.functional.pad(t.float(), (0, 0, 0, pad)) for t in (q, k, v, do)]
    exp = O.landmark_attention_grads(*fp, 64, sm_scale=D ** -0.5)[1:]
    for name, got, e, n in zip(("dq", "dk", "dv"), ref, exp, (Lq, Lk, Lk)):
        got, e = got.float().cpu(), e[:, :, :n]
        # P and dS are rounded to 16 bits in front of the products and the results behind them: the bound of the other kernel tests
        assert (got - e).abs().max().item() < 2e-2 * max(1.0, e.abs().max().item()), name
        assert ((got - e).norm() / e.norm()).item() < 1e-2, name
    assert L.device_status() == 0


@pytest.mark.parametrize("L_,D", [(320, 64), (449, 96), (256, 128)])
def test_outputs_off_a_16_byte_boundary(L_, D):
    # the C interface takes dK and dV at any word (2, 4 and 6 elements behind a boundary), and writes nothing beside them
    g = torch.Generator().manual_seed(D)
    B, H, dtype, lib = 2, 3, torch.bfloat16, L.lib()
    q, k, v, do = [(torch.randn(B, H, L_, D, generator=g) * 0.5).to(dtype).to(DEV) for _ in range(4)]
    n, code, scale, s3, st = q.numel(), L.dtype_code(q), D ** -0.5, L.strides3(q), L.stream_ptr(q.device)
    o, dq = torch.empty_like(q), torch.empty_like(q)
    l, m = [torch.empty(B * H, L_, device=DEV) for _ in range(2)]
    ws = torch.empty(int(lib.lmk_attn_bwd_workspace(B, H, L_, L_, D, 64, code, P.PATH_AUTO)), dtype=torch.uint8, device=DEV)
    L.check(lib.lmk_attn_fwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(l), L.ptr(m), B, H, L_, L_, D, s3, s3, s3, 64, scale,
                             code, P.PATH_AUTO, st), "lmk_attn_fwd")

    def backward(off):
        bufs = [torch.full((n + 16,), 7.0, dtype=dtype, device=DEV) for _ in range(2)]
        dk, dv = [b[off:off + n] for b in bufs]
        L.check(lib.lmk_attn_bwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(do), L.ptr(l), L.ptr(m), L.ptr(dq), L.ptr(dk),
                                 L.ptr(dv), L.ptr(ws), ws.numel(), B, H, L_, L_, D, s3, s3, s3, 64, scale, code, P.PATH_AUTO, st),
                "lmk_attn_bwd")
        for b in bufs:
            assert (b[:off] == 7).all() and (b[off + n:] == 7).all()
        return dk, dv

    ref = backward(0)
    for off in (2, 4, 6):
        assert all(torch.equal(a, b) for a, b in zip(backward(off), ref)), off
    assert L.device_status() == 0


@pytest.mark.parametrize("B,H,T,block,D", [(2, 3, 512, 51, 128), (1, 2, 256, 26, 128), (2, 2, 449, 32, 64), (1, 3, 320, 16, 96)])
def test_units_of_groups(B, H, T, block, D):
    # groups as key tiles: landmarks at each row's own positions (handed over as flags), or a regular pattern of smaller blocks
    g = torch.Generator().manual_seed(T + block)
    q, k, v, do = [(torch.randn(B, H, T, D, generator=g) * 0.5).to(torch.bfloat16) for _ in range(4)]
    flags = T % 128 == 0
    first = torch.randint(0, block, (B, 1), generator=g) if flags else block - 1
    im = ((torch.arange(T).view(1, T) - first) % block == 0).expand(B, T)

    def run(cap):
        L.lib().lmk_debug_set_max_ctas(cap)
        try:
            t = [x.to(DEV).requires_grad_(True) for x in (q, k, v)]
            out = (P.landmark_attention_masked(*t, im.to(DEV), max_groups=16) if flags
                   else P.fused_landmark_attention(*t, None, block_size=block))
            return (out.detach(), *torch.autograd.grad(out, t, do.to(DEV)))
        finally:
            L.lib().lmk_debug_set_max_ctas(0)

    ref = run(0)
    for cap in (1, 2, 5):
        assert all(torch.equal(a, b) for a, b in zip(run(cap), ref)), cap
    f = [x.float().requires_grad_(True) for x in (q, k, v)]
    out = O.lm_attention(*f, im)
    for name, got, e in zip(("o", "dq", "dk", "dv"), ref, (out.detach(), *torch.autograd.grad(out, f, do.float()))):
        got = got.float().cpu()
        assert (got - e).abs().max().item() < 2e-2 * max(1.0, e.abs().max().item()), name
        assert ((got - e).norm() / e.norm()).item() < 1e-2, name
    assert L.device_status() == 0
