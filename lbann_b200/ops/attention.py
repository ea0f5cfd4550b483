"""Fused scaled-dot-product attention (``csrc/attention_tc.cu``) with its PyTorch twin.

``attention(q, k, v, num_heads, scale, causal)`` takes token-major tensors ``[B, S, E]``
(any batch / token strides, e.g. the three column blocks of a packed ``[B, S, 3E]``
projection) and returns ``[B, S, E]``: per head ``softmax(scale * Q K^T [+ causal mask]) V``.
``attention_packed(qkv, ...)`` is the self-attention form whose backward writes the three
gradients straight into one ``[B, S, 3E]`` tensor.

The reference builds this from eight layers and keeps the ``[heads, S, S]`` scores in memory
(python/lbann/modules/transformer/attention.py:215-299); ``exec/model.py`` recognises that
sub-graph and routes it here.  On a GPU with 16-bit inputs, head dimension 128 and sequence
lengths that are multiples of 128 the tcgen05 kernels run; anything else takes the PyTorch
formulation below (fp32 softmax), which is also the test oracle.
"""
from __future__ import annotations

import math

import torch

from . import native


def reference_attention(q, k, v, num_heads: int, scale: float, causal: bool) -> torch.Tensor:
    """The same function in plain PyTorch (scores and softmax in fp32)."""
    B, Sq, E = q.shape
    Sk = k.shape[1]
    D = E // num_heads
    qh = q.reshape(B, Sq, num_heads, D).permute(0, 2, 1, 3).float()
    kh = k.reshape(B, Sk, num_heads, D).permute(0, 2, 1, 3).float()
    vh = v.reshape(B, Sk, num_heads, D).permute(0, 2, 1, 3).float()
    s = (qh @ kh.transpose(-1, -2)) * scale
    if causal:
        mask = torch.ones(Sq, Sk, dtype=torch.bool, device=q.device).triu(1)
        s = s.masked_fill(mask, float("-inf"))
    o = torch.softmax(s, dim=-1) @ vh
    return o.permute(0, 2, 1, 3).reshape(B, Sq, E).to(q.dtype)


def native_ok(q, k, v, num_heads: int, causal: bool) -> bool:
    if not (q.is_cuda and q.dtype in (torch.float16, torch.bfloat16) and k.dtype == q.dtype
            and v.dtype == q.dtype):
        return False
    B, Sq, E = q.shape
    Sk = k.shape[1]
    if E != num_heads * 128 or Sq % 128 or Sk % 128 or (causal and Sq != Sk):
        return False
    for t in (q, k, v):
        if t.stride(2) != 1 or t.stride(1) % 8 or t.stride(0) % 8 or t.data_ptr() % 16:
            return False
    return True


def attention(q, k, v, num_heads: int, scale: float | None = None, causal: bool = False) -> torch.Tensor:
    if scale is None:
        scale = 1.0 / math.sqrt(q.shape[-1] // num_heads)
    if native_ok(q, k, v, num_heads, causal):
        return native.nodes().attention(q, k, v, num_heads, float(scale), bool(causal))
    return reference_attention(q, k, v, num_heads, float(scale), bool(causal))


def attention_packed(qkv, num_heads: int, scale: float | None = None, causal: bool = False) -> torch.Tensor:
    """Self-attention on a packed ``[B, S, 3E]`` projection (queries, keys, values side by
    side along the last dimension)."""
    E = qkv.shape[2] // 3
    if scale is None:
        scale = 1.0 / math.sqrt(E // num_heads)
    q, k, v = qkv[:, :, :E], qkv[:, :, E:2 * E], qkv[:, :, 2 * E:]
    if qkv.dim() == 3 and native_ok(q, k, v, num_heads, causal):
        return native.nodes().attention_packed(qkv, num_heads, float(scale), bool(causal))
    return reference_attention(q, k, v, num_heads, float(scale), bool(causal))
