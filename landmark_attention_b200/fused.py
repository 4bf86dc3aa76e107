"""Fused landmark attention: same Python API as the reference's `fused_landmark_attention`
(llama/ltriton/flash_landmark_attention.py:391-403) and an SDPA-style alias.
"""
import math
from typing import Optional

import torch

from . import _lib as L


class FusedLandmarkAttention:
    """The differentiable call behind `fused_landmark_attention` (FusedLandmarkAttention, flash_landmark_attention.py:308-389):
    forward keeps q, k, v, o and the softmax statistics L, M; backward recomputes the probabilities.  The autograd node
    itself is native (csrc/host_torch.cpp)."""

    @staticmethod
    def apply(q, k, v, n_prefix_q, sm_scale, block_size, path=L.PATH_AUTO):
        assert k.shape[-2] - q.shape[-2] == n_prefix_q * block_size
        return L.host().fused_attention(q, k, v, None, sm_scale, block_size, path)


def fused_landmark_attention(q, k, v, is_mem=None, sm_scale=None, block_size=64, path=L.PATH_AUTO):
    """Landmark attention over q [B,H,Lq,D], k/v [B,H,Lk,D]; the landmark is the last token of every block.

    Same call as the reference's `fused_landmark_attention(q, k, v, is_mem, sm_scale=None, block_size=64)`.
    `is_mem` may be None (fast path: no mask is read and the host is not synchronised); when given it must be the
    regular pattern over the keys, as the reference asserts (flash_landmark_attention.py:393-394).
    """
    if block_size > 64 and path == L.PATH_AUTO and q.is_cuda and q.dtype in (torch.bfloat16, torch.float16):
        out = _large_blocks(q, k, v, is_mem, sm_scale, block_size)
        if out is not None:
            return out
    return L.host().fused_attention(q, k, v, is_mem, sm_scale, block_size, path)


def _large_blocks(q, k, v, is_mem, sm_scale, block_size):
    """The tensor-core kernels behind the host call take blocks of up to 64 keys; larger ones run on the arbitrary-landmark
    tensor-core kernels with the regular pattern as flags, where those take the shape (None: they do not)."""
    from .masked import landmark_attention_masked
    B, Lq, Lk, D = q.shape[0], q.shape[2], k.shape[2], q.shape[3]
    if D > 128 or D % 8 != 0 or (Lk - Lq) % block_size != 0 or (Lk - Lq) % 64 != 0 or Lk < Lq:
        return None
    if sm_scale is None:
        sm_scale = 1.0 / math.sqrt(D)
    # rows of zeros appended to q, k and v come after every real query, so causality hides the extra keys and the extra
    # query rows are dropped again; zero columns change neither q k^T nor the real columns of p v
    rows, cols = -Lq % 128, 128 - D
    groups = max((Lk + rows) // block_size, 1)          # landmarks in front of any query
    if groups > 64 or sm_scale <= 0 or Lk + rows > 32768:
        return None
    if is_mem is not None:
        L.host().check_regular(is_mem, block_size)
    if rows or cols:
        q, k, v = [torch.nn.functional.pad(t, (0, cols, 0, rows)) for t in (q, k, v)]
    out = landmark_attention_masked(q, k, v, _regular_flags(B, Lk + rows, block_size, q.device), sm_scale, groups)
    return out[:, :, :Lq, :D] if rows or cols else out


_FLAGS = {}


def _regular_flags(batch, n_keys, block_size, device):
    """uint8 [batch, n_keys] with a landmark at the end of every block (one row, broadcast over the batch)."""
    key = (device, n_keys, block_size)
    row = _FLAGS.get(key)
    if row is None:
        if len(_FLAGS) > 64:
            _FLAGS.clear()
        row = (torch.arange(n_keys, device=device) % block_size == block_size - 1).to(torch.uint8).view(1, n_keys)
        _FLAGS[key] = row
    return row.expand(batch, n_keys)


def landmark_sdpa(query, key, value, attn_mask=None, dropout_p=0.0, is_causal=True, scale=None, *,
                  is_mem: Optional[torch.Tensor] = None, block_size: int = 64):
    """`torch.nn.functional.scaled_dot_product_attention` signature on top of fused landmark attention.
    Landmark attention is causal by construction; masks and dropout are not part of the operator."""
    if attn_mask is not None:
        raise ValueError("landmark_sdpa does not take attn_mask (the landmark pattern defines the mask)")
    if dropout_p != 0.0:
        raise ValueError("landmark_sdpa does not support dropout")
    if not is_causal:
        raise ValueError("landmark attention is causal; pass is_causal=True")
    return fused_landmark_attention(query, key, value, is_mem, sm_scale=scale, block_size=block_size)


def attn_forward_with_stats(q, k, v, block_size=64, sm_scale=None, path=L.PATH_AUTO):
    """Forward only; also returns the stored statistics (L, M) [B*H, Lq] for inspection and tests."""
    L.require_cuda(q, k, v)
    B, H, Lq, D = q.shape
    Lk = k.shape[2]
    if sm_scale is None:
        sm_scale = 1.0 / math.sqrt(D)
    q, k, v = [t if t.stride(3) == 1 else t.contiguous() for t in (q, k, v)]
    o = torch.empty((B, H, Lq, D), device=q.device, dtype=q.dtype)
    l = torch.empty((B * H, Lq), device=q.device, dtype=torch.float32)
    m = torch.empty((B * H, Lq), device=q.device, dtype=torch.float32)
    rc = L.lib().lmk_attn_fwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(l), L.ptr(m), B, H, Lq, Lk, D,
                              L.strides3(q), L.strides3(k), L.strides3(v), block_size, float(sm_scale),
                              L.dtype_code(q), path, L.stream_ptr(q.device))
    L.check(rc, "lmk_attn_fwd")
    return o, l, m
