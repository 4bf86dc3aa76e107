"""Retrieval of lm_benchmark's block cache on the 16-bit kernels (selection, logits and values in place, prefix part of att @ v)
against the gathered route of the same call: odd block sizes, tails, wrapped rings, both layouts, the three selection
methods, fewer blocks than picks, more than 128 blocks, token counts around the 16- and 64-token tiles."""
import types

import pytest
import torch

import landmark_attention_b200 as P

pytestmark = pytest.mark.gpu
DEV = "cuda"
CASES = [(2, 3, 51, 40, 3, 4, 153, 0, "per_token_and_head"), (1, 2, 16, 9, 2, 3, 65, 5, "per_token_and_head"),
         (1, 2, 8, 200, 3, 2, 130, 0, "per_token_and_head"), (2, 2, 51, 5, 1, 8, 17, 50, "per_token_and_head"),
         (2, 4, 33, 20, 2, 2, 64, 1, "max_over_heads"), (1, 3, 51, 70, 2, 4, 255, 7, "max_over_tokens")]


def store_with(B, H, blk, cap, rounds, top_k, tail, method, dtype, layout, g):
    cfg = types.SimpleNamespace(batch_size=B, mem_cache_size=cap, mem_cache_freq=blk - 1, n_head=H, n_embd=H * 128,
                                cache_topk=top_k, cache_selection_method=method)
    st = P.MemLMCacheStorage(cfg, None, dtype=dtype, device=DEV, layout=layout)
    for i in range(rounds):
        n = (max(1, cap * 2 // (rounds + 1))) * blk + (tail if i == rounds - 1 else 0)
        k, v = [torch.randn(B, H, n, 128, generator=g, device=DEV).to(dtype) for _ in range(2)]
        im = (torch.arange(n, device=DEV) % blk == blk - 1).view(1, n).expand(B, n)
        st.store_in_cache(k, {"v": v, "is_mem": im})
    return st


@pytest.mark.parametrize("dtype,layout", [(torch.bfloat16, "reference"), (torch.float16, "head_major")])
@pytest.mark.parametrize("B,H,blk,cap,rounds,top_k,T,tail,method", CASES)
def test_retrieval_and_prefix_attention_match_the_gathered_route(B, H, blk, cap, rounds, top_k, T, tail, method, dtype, layout):
    g = torch.Generator(device=DEV).manual_seed(cap + T)
    st = store_with(B, H, blk, cap, rounds, top_k, tail, method, dtype, layout, g)
    q, k, v = [torch.randn(B, H, T, 128, generator=g, device=DEV).to(dtype) for _ in range(3)]
    start = (top_k + 1) * blk + tail
    att, d = st.retrieve_for_query(q, None, None, start)
    native, st._retrieve_native = st._retrieve_native, lambda *a: None
    exp, ed = st.retrieve_for_query(q, None, None, start)
    assert native(q, *st._tables, st.last_incomplete_len, start) is not None and st.last_incomplete_len == tail
    assert att.shape == exp.shape and torch.equal(d["is_mem"], ed["is_mem"])
    assert torch.equal(d["v"], ed["v"])                        # same picks in the same order, same tail
    assert (att.float() - exp.float()).abs().max().item() < 3e-2
    im = (torch.arange(T, device=DEV) + tail) % blk == blk - 1
    im = im.view(1, T).expand(B, T)
    y = P.lm_landmark_attention(q, k, v, im, att_prefix=exp, cache_values=ed)
    with torch.enable_grad():                                  # the differentiable route: library matmuls
        ye = P.lm_landmark_attention(q.clone().requires_grad_(True), k, v, im, att_prefix=exp, cache_values=ed)
    assert (y.float() - ye.float()).abs().max().item() < 3e-2
    assert ((y.float() - ye.float()).norm() / ye.float().norm()).item() < 5e-3


@pytest.mark.parametrize("dtype,layout", [(torch.bfloat16, "reference"), (torch.float16, "head_major")])
@pytest.mark.parametrize("chunks", [(3, 3, 1, 9, 20, 7), (1,) * 19, (8, 2, 3, 3, 5), (5,)])
def test_chunks_below_a_block_are_stored_as_the_whole_is(chunks, dtype, layout):
    B, H, blk, cap, n = 2, 3, 8, 4, sum(chunks)          # the longest wraps the ring
    g = torch.Generator(device=DEV).manual_seed(n)
    k, v = [torch.randn(B, H, n, 128, generator=g, device=DEV).to(dtype) for _ in range(2)]
    im = (torch.arange(n, device=DEV) % blk == blk - 1).view(1, n).expand(B, n)
    cfg = types.SimpleNamespace(batch_size=B, mem_cache_size=cap, mem_cache_freq=blk - 1, n_head=H, n_embd=H * 128,
                                cache_topk=2, cache_selection_method="per_token_and_head")
    one, many = [P.MemLMCacheStorage(cfg, None, dtype=dtype, device=DEV, layout=layout) for _ in range(2)]
    for st in (one, many):
        for buf in (st.cache_mem_k, st.cache_mem_v, st.cache_lm_k):
            buf.zero_()
    one.store_in_cache(k, {"v": v, "is_mem": im})
    lo = 0
    for c in chunks:
        many.store_in_cache(k[:, :, lo:lo + c], {"v": v[:, :, lo:lo + c], "is_mem": im[:, lo:lo + c]})
        lo += c
    assert (many.last_incomplete_len, many.cache_iter, many.cache_size) == (one.last_incomplete_len, one.cache_iter, one.cache_size)
    tail = n % blk
    for a, b in ((many.cache_mem_k, one.cache_mem_k), (many.cache_mem_v, one.cache_mem_v), (many.cache_lm_k, one.cache_lm_k),
                 (many.last_incomplete_k[:, :, :tail], k[:, :, n - tail:]), (many.last_incomplete_v[:, :, :tail], v[:, :, n - tail:]),
                 (many.last_incomplete_ismem[:, :tail], im[:, n - tail:])):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,value", [(torch.uint8, 1), (torch.uint8, 255), (torch.int64, 7), (torch.float32, 0.5)])
def test_any_value_but_zero_marks_a_landmark(dtype, value):
    blk, n = 8, 19
    cfg = types.SimpleNamespace(batch_size=2, mem_cache_size=4, mem_cache_freq=blk - 1, n_head=2, n_embd=256, cache_topk=2,
                                cache_selection_method="per_token_and_head")
    k = torch.randn(2, 2, n, 128, device=DEV)
    im = (torch.arange(n, device=DEV) % blk == blk - 1).view(1, n).expand(2, n).to(dtype) * value
    st = P.MemLMCacheStorage(cfg, None, dtype=torch.float32, device=DEV)
    st.store_in_cache(k, {"v": k, "is_mem": im})
    assert (st.cache_size, st.last_incomplete_len) == (2, 3) and torch.equal(st.cache_lm_k[:, :, 0], k[:, :, blk - 1])
    im[1, 3] = value
    with pytest.raises(AssertionError):
        P.MemLMCacheStorage(cfg, None, dtype=torch.float32, device=DEV).store_in_cache(k, {"v": k, "is_mem": im})
