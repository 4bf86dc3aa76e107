"""Gradients of the retrieval entry points: where the tensor formulation of a call is differentiable, a call that wants gradients takes
that formulation, and gets its gradients; without gradients the native call runs."""

import types

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


@DTYPES
@pytest.mark.parametrize("wanted", [("q",), ("k",), ("v",), ("q", "k", "v")])
def test_block_cache_retrieval_is_differentiable(wanted, dtype):
    # the queries, and what an earlier chunk left in the unfinished block
    B, H, blk, T, tail = 1, 2, 16, 5, 7
    n = 4 * blk + tail
    (k, v, q, _, _), _ = problem(B, H, T, n, dtype, len(wanted))
    cfg = types.SimpleNamespace(batch_size=B, mem_cache_size=8, mem_cache_freq=blk - 1, n_head=H, n_embd=H * 128,
                                cache_topk=2, cache_selection_method="per_token_and_head")
    im = (torch.arange(n, device=DEV) % blk == blk - 1).view(1, n).expand(B, n)
    x = {name: t.clone().requires_grad_(name in wanted) for name, t in (("q", q), ("k", k), ("v", v))}
    st = P.MemLMCacheStorage(cfg, None, dtype=dtype, device=DEV)
    st.store_in_cache(x["k"], {"v": x["v"], "is_mem": im})
    att, d = st.retrieve_for_query(x["q"], None, None, 3 * blk + tail)
    g = torch.Generator(device=DEV).manual_seed(5)
    da, dv = [torch.randn(t.shape, generator=g, device=DEV).to(dtype) for t in (att, d["v"])]
    outs = [(att, da)] * att.requires_grad + [(d["v"], dv)] * d["v"].requires_grad
    grads = dict(zip(wanted, torch.autograd.grad([o for o, _ in outs], [x[w] for w in wanted], [go for _, go in outs])))
    # the tail's logits are q . rotated key / sqrt(D), its values are handed on once per token
    pos = torch.arange(3 * blk, 3 * blk + tail)
    qf, kt = [t.detach().float().cpu().requires_grad_(True) for t in (x["q"], x["k"][:, :, n - tail:])]
    logits = qf @ O.rotary_interleaved(kt, pos.view(1, 1, tail).expand(B, H, tail).float()).transpose(2, 3) / 128 ** 0.5
    want_q, want_k = torch.autograd.grad(logits, [qf, kt], da[..., 2 * blk:].float().cpu(), retain_graph=True)
    if "k" in wanted:
        assert close(grads["k"][:, :, n - tail:], want_k) and not grads["k"][:, :, :n - tail].any()
    if "v" in wanted:
        assert close(grads["v"][:, :, n - tail:], dv[:, :, :, 2 * blk:].float().sum(2)) and not grads["v"][:, :, :n - tail].any()
    if wanted == ("q",):
        # the gathered blocks' part comes on top of the tail's
        zero = torch.cat((torch.zeros_like(da[..., :2 * blk]), da[..., 2 * blk:]), -1)
        att, _ = st.retrieve_for_query(x["q"], None, None, 3 * blk + tail)
        assert close(torch.autograd.grad(att, x["q"], zero)[0], want_q)
    with torch.no_grad():
        fast, fd = st.retrieve_for_query(x["q"], None, None, 3 * blk + tail)
        assert not fast.requires_grad and close(fast, att.detach()) and torch.equal(fd["v"], d["v"].detach())
