"""Gradients of the retrieval entry points: where the tensor formulation of a call is differentiable, a call that wants gradients takes
that formulation, and gets its gradients; without gradients the native call runs."""

import pytest
import torch

import landmark_attention_b200 as P
from oracle import landmark_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
DTYPES = pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])


def problem(B, H, T, C, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda n: (torch.randn(B, H, n, 128, generator=g, device=DEV) * 0.5).to(dtype)
    return [rnd(n) for n in (C, C, T, T, T)], torch.randn(B, H, T, 128, generator=g, device=DEV).to(dtype)


def leaves(*ts):
    return [t.clone().requires_grad_(True) for t in ts]


def close(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return (a - b).abs().max().item() < 2e-2 and ((a - b).norm() / b.norm()).item() < 1e-2


@DTYPES
@pytest.mark.parametrize("T,blk,N,top_k", [(64, 64, 9, 2), (96, 32, 20, 3)])
def test_per_head_selection_is_differentiable(T, blk, N, top_k, dtype):
    (pk, pv, q, k, v), do = problem(1, 2, T, N * blk, dtype, T + N)
    cos, sin = P.rotary_tables_half(N * blk + T + 1, 128, dtype, DEV)
    call = lambda a, **kw: P.llama_retrieval_attention(*a, mem_freq=blk - 1, cache_top_k=top_k, cos=cos, sin=sin,
                                                       aggregate="max_over_tokens", **kw)
    a = leaves(q, k, v)
    exp, _, dbg = call(a, past_k=pk, past_v=pv, return_debug=True)
    grads = torch.autograd.grad(exp, a, do)
    # the values' gradients against the oracle: the selected blocks and the chunk as one sequence
    pos = torch.arange(N * blk, N * blk + T)
    qr, kr = [O.rotary_half_split(t.float().cpu(), pos.view(1, 1, T)) for t in (q, k)]
    keys, vals = [torch.cat((dbg[n].float().cpu().view(1, 2, top_k * blk, 128), t), 2) for n, t in (("sel_k", kr), ("sel_v", v.float().cpu()))]
    assert close(grads[2], O.landmark_attention_grads(qr, keys, vals, do.float().cpu(), blk)[3][:, :, top_k * blk:])

    cache = P.LandmarkKVCache(1, 2, N * blk + T, 128, dtype, DEV)
    cache.append(pk, pv)
    off = P.OffloadedLandmarkCache(1, 2, N + T // blk, blk, 128, dtype, DEV)
    off.append(pk, pv)
    for run in (lambda a: call(a, past_k=pk, past_v=pv)[0], lambda a: call(a, cache=cache)[0],
                lambda a: off.attend(*a, top_k, cos, sin)):
        a = leaves(q, k, v)
        out = run(a)
        assert out.requires_grad and torch.equal(out, exp)
        for got, want in zip(torch.autograd.grad(out, a, do), grads):
            assert torch.equal(got, want)
    torch.cuda.synchronize()
    assert torch.equal(off.k_host[:, :, N * blk:].to(DEV), k) and torch.equal(cache.v[:, :, N * blk:], v)
    with torch.no_grad():
        out, _ = call(leaves(q, k, v), past_k=pk, past_v=pv)
        assert not out.requires_grad and close(out, exp)


@DTYPES
@pytest.mark.parametrize("T,blk,N,tail,top_k", [(1, 32, 9, 17, 4), (3, 64, 5, 50, 2)])
def test_tokens_inside_an_unfinished_block_are_differentiable(T, blk, N, tail, top_k, dtype):
    C = N * blk + tail
    (pk, pv, q, k, v), do = problem(1, 2, T, C, dtype, C)
    cos, sin = P.rotary_tables_half(C + T + 1, 128, dtype, DEV)
    call = lambda a, **kw: P.llama_retrieval_attention(*a, mem_freq=blk - 1, cache_top_k=top_k, cos=cos, sin=sin, **kw)
    a = leaves(q, k, v, pk, pv)
    exp, _ = call(a[:3], past_k=a[3], past_v=a[4], materialize=False)
    grads = torch.autograd.grad(exp, a, do)
    # the values' gradients (new ones, and the cached ones of the unfinished block) against the oracle, with this call's selection
    _, _, dbg = call((q, k, v), past_k=pk, past_v=pv, return_debug=True)
    o = [t.float().cpu().requires_grad_(True) for t in (q, k, v, pk, pv)]
    want = torch.autograd.grad(O.llama_retrieval_attention(*o, blk, top_k, sel=dbg["sel"].long().cpu()), o, do.float().cpu())
    assert close(grads[2], want[2]) and close(grads[4][:, :, N * blk:], want[4][:, :, N * blk:])

    for wanted in ((0, 1, 2, 3, 4), (1,), (4,)):                 # also a gradient of one input alone
        a = [t.clone().requires_grad_(i in wanted) for i, t in enumerate((q, k, v, pk, pv))]
        out, _ = call(a[:3], past_k=a[3], past_v=a[4])
        assert out.requires_grad and torch.equal(out, exp)
        for i, got in zip(wanted, torch.autograd.grad(out, [a[i] for i in wanted], do)):
            assert torch.equal(got, grads[i])
    cache = P.LandmarkKVCache(1, 2, C + T, 128, dtype, DEV)
    cache.append(pk, pv)
    a = leaves(q, k, v)
    out, _ = call(a, cache=cache)
    for got, want in zip(torch.autograd.grad(out, a, do), grads):
        assert torch.equal(got, want)
    with torch.no_grad():
        out, _ = call(leaves(q, k, v), past_k=pk, past_v=pv)
        assert not out.requires_grad and close(out, exp)
