"""The check of a landmark mask belongs to its own call: a call that was refused for another reason, a call inside the first
one's hooks and calls of other threads leave its verdict alone."""
import threading

import pytest
import torch

import landmark_attention_b200 as P

pytestmark = pytest.mark.gpu
DEV = "cuda"


def problem(rows=128):
    q, k, v = [torch.randn(1, 2, rows, 128, device=DEV).to(torch.bfloat16) for _ in range(3)]
    good = torch.arange(rows, device=DEV) % 64 == 63
    return q, k, v, good, torch.ones_like(good)


def test_a_refused_call_leaves_the_next_one_alone():
    q, k, v, good, bad = problem()
    want = P.fused_landmark_attention(q, k, v, good)
    torch.cuda._sleep(200_000_000)                     # about 0.1 s: the first check is still queued when the second call begins
    with pytest.raises(AssertionError, match="history"):
        P.fused_landmark_attention(q, k[:, :, 1:], v[:, :, 1:], bad)
    assert torch.equal(P.fused_landmark_attention(q, k, v, good), want)
    with pytest.raises(AssertionError, match="is_mem"):
        P.fused_landmark_attention(q, k, v, bad)


@pytest.mark.parametrize("outer_bad", [True, False])
def test_a_call_inside_a_saved_tensor_hook(outer_bad):
    q, k, v, good, bad = problem()
    inner = []

    def pack(t):
        if not inner:
            inner.append(None)
            with torch.no_grad():
                if outer_bad:
                    P.fused_landmark_attention(q, k, v, good)
                else:
                    with pytest.raises(AssertionError, match="is_mem"):
                        P.fused_landmark_attention(q, k, v, bad)
            inner.append(True)
        return t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        leaf = q.clone().requires_grad_(True)
        if outer_bad:
            with pytest.raises(AssertionError, match="is_mem"):
                P.fused_landmark_attention(leaf, k, v, bad)
        else:
            P.fused_landmark_attention(leaf, k, v, good)
    assert inner == [None, True]


def test_threads_get_their_own_verdicts():
    wrong = []

    def work(irregular):
        q, k, v, good, bad = problem()
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                try:
                    P.fused_landmark_attention(q, k, v, bad if irregular else good)
                    refused = False
                except AssertionError:
                    refused = True
                if refused != irregular:
                    wrong.append(irregular)

    threads = [threading.Thread(target=work, args=(i % 2 == 1,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
