"""Prompt chunks behind a block cache as native calls (16 bits, head dim 128) against the tensor formulations of the same call: whole and
ragged chunk lengths, one and several query tiles, block sizes, more and fewer than 128 blocks, device and host caches."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L

pytestmark = pytest.mark.gpu
DEV = "cuda"


def close(a, b):
    a, b = a.float(), b.float()
    return (a - b).abs().max().item() < 2e-2 and ((a - b).norm() / b.norm()).item() < 1e-2


def problem(B, H, T, blk, N, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda n: torch.randn(B, n, H, 128, generator=g, device=DEV).to(dtype).transpose(1, 2)
    C = N * blk
    pk, pv = [rnd(C).contiguous() for _ in range(2)]
    return pk, pv, rnd(T), rnd(T), rnd(T), P.rotary_tables_half(C + T + 1, 128, dtype, DEV)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,T,blk,N,top_k", [(1, 3, 258, 32, 140, 4), (2, 2, 40, 64, 9, 6), (1, 2, 17, 16, 30, 1), (1, 2, 300, 64, 33, 3),
                                               (1, 8, 129, 32, 5, 5)])
def test_chunk_matches_the_gathered_route(B, H, T, blk, N, top_k, dtype):
    pk, pv, q, k, v, (cos, sin) = problem(B, H, T, blk, N, dtype, T)
    exp, (ek, ev) = P.llama_retrieval_attention(q, k, v, pk, pv, blk - 1, top_k, cos=cos, sin=sin, materialize=True)
    cache = P.LandmarkKVCache(B, H, N * blk + T, 128, dtype, DEV)
    cache.append(pk, pv)
    for args in (dict(cache=cache), dict(past_k=pk, past_v=pv)):
        got, (gk, gv) = P.llama_retrieval_attention(q, k, v, mem_freq=blk - 1, cache_top_k=top_k, cos=cos, sin=sin, **args)
        assert torch.equal(gk, ek) and torch.equal(gv, ev) and close(got, exp)
    assert L.device_status() == 0


@pytest.mark.parametrize("which", ["q", "k", "v", "qkv"])
@pytest.mark.parametrize("form", ["heads", "batch", "rows", "offset", "features"])
def test_chunk_of_any_strides(form, which):
    B, H, T, blk, N, dtype = 2, 3, 40, 32, 6, torch.bfloat16
    pk, pv, q, k, v, (cos, sin) = problem(B, H, T, blk, N, dtype, T)
    odd = {"heads": lambda t: t[:, :1].expand(B, H, T, 128), "batch": lambda t: t[:1].expand(B, H, T, 128),
           "rows": lambda t: t[:, :, :1].expand(B, H, T, 128),
           "offset": lambda t: torch.cat((t.new_zeros(3), t.reshape(-1)))[3:].view(B, H, T, 128),
           "features": lambda t: torch.stack((t, t), -1).flatten(-2)[..., ::2]}[form]
    q, k, v = [odd(t) if name in which else t for name, t in (("q", q), ("k", k), ("v", v))]
    exp, _ = P.llama_retrieval_attention(*[t.contiguous() for t in (q, k, v)], pk, pv, blk - 1, 3, cos=cos, sin=sin)
    cache = P.LandmarkKVCache(B, H, N * blk + T, 128, dtype, DEV)
    cache.append(pk, pv)
    for args in (dict(cache=cache), dict(past_k=pk, past_v=pv)):
        got, (gk, gv) = P.llama_retrieval_attention(q, k, v, mem_freq=blk - 1, cache_top_k=3, cos=cos, sin=sin, **args)
        assert torch.equal(got, exp) and torch.equal(gk[:, :, N * blk:], k) and torch.equal(gv[:, :, N * blk:], v)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,T,blk,N,top_k", [(1, 3, 256, 64, 140, 4), (2, 2, 96, 32, 20, 1), (1, 4, 128, 32, 129, 6), (1, 2, 64, 64, 3, 3)])
def test_per_head_selection_on_device_and_host_caches(B, H, T, blk, N, top_k, dtype):
    pk, pv, q, k, v, (cos, sin) = problem(B, H, T, blk, N, dtype, T + N)
    off = P.OffloadedLandmarkCache(B, H, N + 2 * T // blk, blk, 128, dtype, DEV)
    off.append(pk, pv)
    past = (pk, pv)
    for step in range(2):                      # the second chunk reads what the first one stored
        exp, past, _ = P.llama_retrieval_attention(q, k, v, past[0], past[1], blk - 1, top_k, cos=cos, sin=sin,
                                                   aggregate="max_over_tokens", return_debug=True)
        cache = P.LandmarkKVCache(B, H, past[0].shape[2], 128, dtype, DEV)
        cache.append(past[0][:, :, :-T], past[1][:, :, :-T])
        got, views = P.llama_retrieval_attention(q, k, v, mem_freq=blk - 1, cache_top_k=top_k, cos=cos, sin=sin, cache=cache,
                                                 aggregate="max_over_tokens")
        host = off.attend(q, k, v, top_k, cos, sin)
        assert torch.equal(views[0], past[0]) and torch.equal(views[1], past[1])
        assert close(got, exp) and torch.equal(host, got)
        cos, sin = P.rotary_tables_half(past[0].shape[2] + T + 1, 128, dtype, DEV)
    torch.cuda.synchronize()
    assert off.length == past[0].shape[2]
    assert torch.equal(off.k_host[:, :, :off.length].to(DEV), past[0]) and torch.equal(off.v_host[:, :, :off.length].to(DEV), past[1])
    assert torch.equal(off.lm_keys[:, :, :off.n_blocks], past[0][:, :, blk - 1::blk])


@pytest.mark.parametrize("T,blk,N,top_k", [(128, 128, 9, 2), (256, 256, 5, 1), (512, 256, 6, 3)])
def test_per_head_selection_of_large_blocks(T, blk, N, top_k):
    pk, pv, q, k, v, (cos, sin) = problem(1, 2, T, blk, N, torch.bfloat16, T)
    exp, past, _ = P.llama_retrieval_attention(q, k, v, pk, pv, blk - 1, top_k, cos=cos, sin=sin, aggregate="max_over_tokens",
                                               return_debug=True)
    cache = P.LandmarkKVCache(1, 2, N * blk + T, 128, torch.bfloat16, DEV)
    cache.append(pk, pv)
    off = P.OffloadedLandmarkCache(1, 2, N + T // blk, blk, 128, torch.bfloat16, DEV)
    off.append(pk, pv)
    got, views = P.llama_retrieval_attention(q, k, v, mem_freq=blk - 1, cache_top_k=top_k, cos=cos, sin=sin, cache=cache,
                                             aggregate="max_over_tokens")
    assert close(got, exp) and torch.equal(views[0], past[0]) and torch.equal(views[1], past[1])
    assert close(off.attend(q, k, v, top_k, cos, sin), exp) and off.length == N * blk + T
    torch.cuda.synchronize()
    assert torch.equal(off.k_host.to(DEV), past[0]) and torch.equal(off.v_host.to(DEV), past[1])


def test_ragged_chunk_against_the_host_cache_waits_in_the_tail():
    pk, pv, q, k, v, (cos, sin) = problem(1, 2, 100, 64, 10, torch.bfloat16, 1)
    off = P.OffloadedLandmarkCache(1, 2, 12, 64, 128, torch.bfloat16, DEV)
    off.append(pk, pv)
    exp, _, _ = P.llama_retrieval_attention(q, k, v, pk, pv, 63, 2, cos=cos, sin=sin, aggregate="max_over_tokens", return_debug=True)
    assert close(off.attend(q, k, v, 2, cos, sin), exp)
    assert (off.n_blocks, off.tail_len) == (11, 36) and torch.equal(off.tail_k[:, :, :36], k[:, :, 64:])
    with pytest.raises(AssertionError):
        off.attend(q, k, v, 2, cos, sin)


def test_a_chunk_refused_after_its_stores_began_leaves_nothing_in_flight():
    # blocks of one key are refused by the attention, which comes behind the copies to the host cache: what the current stream does next
    # must come behind them too
    T, H = 2048, 32
    k, v = [torch.randn(1, H, T, 128, device=DEV).to(torch.bfloat16) for _ in range(2)]
    off = P.OffloadedLandmarkCache(1, H, T + 8, 1, 128, torch.bfloat16, DEV)
    off.append(k[:, :, :8], v[:, :, :8])
    cos, sin = P.rotary_tables_half(T + 9, 128, torch.bfloat16, DEV)
    want = [t.cpu() for t in (k, v)]
    for _ in range(2):                                # the first call loads the kernels
        torch.cuda.synchronize()
        off.v_host[:, :, 8:].zero_()
        torch.cuda._sleep(20_000_000)                 # about 10 ms: the copies begin behind it, long after the call has returned
        with pytest.raises(AssertionError):
            off.attend(k, k, v, 1, cos, sin)
    assert off.n_blocks == 8
    torch.cuda.current_stream().synchronize()
    last = off.v_host[0, H - 1, -1].clone()       # the last row to arrive, read before anything that takes time
    assert torch.equal(last, want[1][0, H - 1, -1])
    assert torch.equal(off.k_host[:, :, 8:], want[0]) and torch.equal(off.v_host[:, :, 8:], want[1])
