"""Forward-mode derivatives: the operators refuse a tangent (they have no forward-mode formula), whether or not gradients are
enabled, and what is a plain tensor formulation propagates it; none drops it without a word."""
import types

import pytest
import torch
from torch.autograd import forward_ad

import landmark_attention_b200 as P

pytestmark = pytest.mark.gpu
DEV = "cuda"
DT = torch.bfloat16


def rnd(*s):
    return torch.randn(*s, device=DEV).to(DT)


def dual(t):
    return forward_ad.make_dual(t, torch.ones_like(t))


def fused():
    P.fused_landmark_attention(rnd(1, 2, 128, 128), rnd(1, 2, 128, 128), dual(rnd(1, 2, 128, 128)))


def masked():
    q = rnd(1, 2, 128, 128)
    P.lm_landmark_attention(dual(q), q, q, (torch.arange(128, device=DEV) % 51 == 50).view(1, 128))


def rotary():
    P.rotary_apply(dual(rnd(1, 2, 64, 128)), rnd(1, 2, 64, 128), *P.rotary_tables_interleaved(64, 128, DT, DEV))


def softmax(flavour):
    x, hidden = torch.randn(1, 2, 64, 64, device=DEV), torch.ones(64, 64, dtype=torch.bool, device=DEV).triu(1)
    row = (torch.arange(64, device=DEV) % 16 == 15).view(1, 64)
    mask, is_mem, last = P.prepare_landmark_masks(row, hidden)
    if flavour == "lm":
        P.landmark_grouped_softmax_lm(dual(x), -1, is_mem, mask, last, False, 8)
    elif flavour == "llama":
        P.landmark_grouped_softmax(dual(x), -1, is_mem, last)
    else:
        P.landmark_grouped_softmax_causal(dual(x), row, 8)


def retrieval(tail, aggregate):
    T, C = 2 if tail else 64, 5 * 32 + tail
    q, k, v = [rnd(1, 2, T, 128) for _ in range(3)]
    cos, sin = P.rotary_tables_half(C + T + 1, 128, DT, DEV)
    P.llama_retrieval_attention(q, dual(k), v, rnd(1, 2, C, 128), rnd(1, 2, C, 128), 31, 2, cos=cos, sin=sin, aggregate=aggregate)


CALLS = [fused, masked, rotary, lambda: softmax("lm"), lambda: softmax("llama"), lambda: softmax("causal"),
         lambda: retrieval(17, None), lambda: retrieval(0, "max_over_tokens")]


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("call", CALLS)
def test_operators_refuse_tangents(call, grad):
    with torch.set_grad_enabled(grad), forward_ad.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
            call()


def test_block_cache_retrieval_propagates_tangents():
    B, H, blk, T, tail = 1, 2, 16, 5, 7
    n = 4 * blk + tail
    cfg = types.SimpleNamespace(batch_size=B, mem_cache_size=8, mem_cache_freq=blk - 1, n_head=H, n_embd=H * 128,
                                cache_topk=2, cache_selection_method="per_token_and_head")
    st = P.MemLMCacheStorage(cfg, None, dtype=DT, device=DEV)
    im = (torch.arange(n, device=DEV) % blk == blk - 1).view(1, n)
    st.store_in_cache(rnd(B, H, n, 128), {"v": rnd(B, H, n, 128), "is_mem": im})
    q = rnd(B, H, T, 128)
    with torch.no_grad(), forward_ad.dual_level():
        att, _ = st.retrieve_for_query(forward_ad.make_dual(q, q), None, None, 3 * blk + tail)
        primal, tangent = forward_ad.unpack_dual(att)
        assert torch.equal(primal, tangent)              # the logits are linear in q: along q itself they are their own tangent


def test_the_prefix_values_tangent_is_propagated():
    T, n = 64, 32
    q, k, v = [rnd(1, 2, T, 128) for _ in range(3)]
    im = (torch.arange(T, device=DEV) % 16 == 15).view(1, T)
    att, vals = rnd(1, 2, T, n), rnd(1, 2, T, n, 128)
    run = lambda x: P.lm_landmark_attention(q, k, v * 0, im, att_prefix=att, cache_values={"v": x})
    with torch.no_grad(), forward_ad.dual_level():
        primal, tangent = forward_ad.unpack_dual(run(forward_ad.make_dual(vals, vals)))
        # without values of its own the chunk's output is linear in the prefix' values
        assert ((primal.float() - tangent.float()).norm() / primal.float().norm()).item() < 1e-2
