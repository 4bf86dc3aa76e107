"""Token generation in one launch (lmk_decode_attend) against the gathered route of the same call: edges of the 16-row items
and of the 16 landmarks that a warp scores at a time, a query that is a landmark, whole-block caches, one to sixteen tokens, both cluster sizes."""
import pytest
import torch

import landmark_attention_b200 as P
from landmark_attention_b200 import _lib as L

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,T,blk,N,tail,top_k", [
    (1, 2, 1, 32, 40, 17, 4), (2, 3, 3, 64, 9, 50, 6), (1, 8, 1, 16, 5, 0, 5), (1, 1, 5, 16, 300, 11, 3), (1, 1, 2, 20, 7, 3, 2),
    (1, 40, 1, 64, 33, 62, 1), (4, 5, 1, 32, 1025, 31, 4), (1, 2, 16, 32, 64, 0, 2), (1, 2, 1, 16, 70, 9, 32)])
def test_decode_matches_the_gathered_route(B, H, T, blk, N, tail, top_k, dtype):
    g = torch.Generator(device=DEV).manual_seed(N + tail)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)
    C = N * blk + tail
    pk, pv = rnd(B, H, C, 128), rnd(B, H, C, 128)
    q, k, v = [rnd(B, T, H, 128).transpose(1, 2) for _ in range(3)]              # strided projections
    cos, sin = P.rotary_tables_half(C + T + 1, 128, dtype, DEV)
    exp, (ek, ev) = P.llama_retrieval_attention(q, k, v, pk, pv, blk - 1, top_k, cos=cos, sin=sin, materialize=True)
    assert L.lib().lmk_decode_supported(128, blk, min(top_k, N), C, T, L.dtype_code(q)) == 1
    cache = P.LandmarkKVCache(B, H, C + T, 128, dtype, DEV)
    cache.append(pk, pv)
    cache.k[:, :, C:] = float("nan")
    for args in (dict(cache=cache), dict(past_k=pk, past_v=pv)):
        got, (gk, gv) = P.llama_retrieval_attention(q, k, v, mem_freq=blk - 1, cache_top_k=top_k, cos=cos, sin=sin, **args)
        assert torch.equal(gk, ek) and torch.equal(gv, ev)
        assert (got.float() - exp.float()).abs().max().item() < 2e-2
        assert ((got.float() - exp.float()).norm() / exp.float().norm()).item() < 1e-2
