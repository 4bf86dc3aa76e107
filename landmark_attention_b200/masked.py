"""Fused landmark attention with landmarks at arbitrary positions (one flag per batch row and key).

This is the attention of lm_benchmark's `CausalSelfAttention.forward` without cache -- scores, causal fill, mask block,
grouped softmax, att @ v (lm_benchmark/models/landmark.py:196-236, :210-224, :37-119) -- as one differentiable operator
on the tensor cores.  No [B,H,T,T] tensor exists at any point; the group ids are derived inside the kernels from
`is_mem [B, T]`.

The operator is registered with `torch.library` (`lmk::masked_attention`, with a fake implementation and an autograd
formula), so a model that calls it can be wrapped in `torch.compile(fullgraph=True)` as the reference's trainer does
(lm_benchmark/optim/base.py:57-61) without a graph break.
"""
import math

import torch

from . import _lib as L

DEFAULT_MAX_GROUPS = 64


def _register_fakes():
    """Shape functions of the operators that the host layer registers (lmk::masked_attention_fwd / _bwd)."""
    @torch.library.register_fake("lmk::masked_attention_fwd")
    def _(q, k, v, is_mem, sm_scale, max_groups):
        B, H, Lq, D = q.shape
        return (q.new_empty((B, H, Lq, D)), q.new_empty((B * H, Lq), dtype=torch.float32),
                q.new_empty((B * H, max_groups, Lq), dtype=torch.float32))

    @torch.library.register_fake("lmk::masked_attention_bwd")
    def _(q, k, v, is_mem, o, do, R, A, sm_scale, max_groups):
        return (q.new_empty(q.shape), k.new_empty(k.shape), v.new_empty(v.shape))


L.on_host_load(_register_fakes)


def _fwd(q, k, v, is_mem, sm_scale, max_groups):
    """(o, R, A); through the operator registry while a compiler traces, straight into the host layer otherwise."""
    if torch.compiler.is_compiling():
        return torch.ops.lmk.masked_attention_fwd(q, k, v, is_mem, sm_scale, max_groups)
    return L.host().masked_attention(q, k, v, is_mem, sm_scale, max_groups)


# the kernels' shape contract (include/b200lmk.h, lmk_attn_mask_fwd); kept in Python so that the check is traceable
_HEAD_DIM, _Q_TILE, _K_TILE, _MAX_KEYS, _MAX_GROUPS = 128, 128, 64, 32768, 64


def masked_attention_supported(q, k, max_groups=DEFAULT_MAX_GROUPS) -> bool:
    """True when the tensor-core kernels take this problem (bf16/fp16, D = 128, whole 128-row query tiles, 64-key
    tiles, max_groups within the build's limit).  Pure shape logic: no library call, so torch.compile can trace it."""
    if not q.is_cuda or q.dtype not in (torch.bfloat16, torch.float16):
        return False
    Lq, D, Lk = q.shape[2], q.shape[3], k.shape[2]
    return (D == _HEAD_DIM and Lq >= _Q_TILE and Lq % _Q_TILE == 0 and Lk % _K_TILE == 0 and Lk >= Lq
            and (Lk - Lq) % _K_TILE == 0 and Lk <= _MAX_KEYS and 0 < max_groups <= _MAX_GROUPS)


def landmark_attention_masked(q, k, v, is_mem, sm_scale=None, max_groups=DEFAULT_MAX_GROUPS):
    """Landmark attention of q [B,H,Lq,D] over k, v [B,H,Lk,D] with landmark flags is_mem [B, Lk] (bool or uint8).

    `max_groups` bounds the number of landmarks before any query (lm_benchmark's max_groups_for_softmax - 1); it sizes
    the statistics kept for the backward pass.  Raises NotImplementedError for shapes outside the kernels' contract."""
    if sm_scale is None:
        sm_scale = 1.0 / math.sqrt(q.size(-1))
    return _fwd(q, k, v, is_mem, float(sm_scale), int(max_groups))[0]
