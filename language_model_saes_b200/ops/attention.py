"""Causal attention whose value width differs from the query/key width, on the sm_100a tensor cores.

A low-rank sparse attention dictionary runs one attention per QK head with the head's whole OV group as the value
(models/lorsa.py:642-661,864-904 of the reference project, which calls ``scaled_dot_product_attention``): ``q, k`` are
``[batch, seq, heads, d_qk]`` and ``v`` is ``[batch, seq, heads, d_v]`` with ``d_v`` a multiple of ``d_qk`` or unrelated
to it. ``csrc/attention.cu`` implements the forward pass with tcgen05 MMAs, accumulators in TMEM and TMA-fed operands;
``ref_causal_attention`` is the plain-torch oracle.
"""

from __future__ import annotations

import math

import torch

from . import sae_kernels as K


def library_attention_backends():
    """Context in which ``scaled_dot_product_attention`` may pick its memory-efficient or its plain backend only.

    A value width that differs from the query/key width rules the flash backend out, and the library then prefers its
    cuDNN backend on this architecture. With torch 2.11 / cuDNN 9 on sm_100 that backend's BACKWARD pass returned input
    gradients that depended on what the allocator's recycled memory held: correct in a fresh process, unrelated to the
    true gradient (cosine near 0) or NaN once freed blocks had been filled with a NaN pattern, for several stride layouts
    of the output gradient and at both a tiny and a training-size shape; its forward pass and both passes of the
    memory-efficient backend were correct in every such run. The backward pass follows the forward's choice, so the
    context is only needed around the forward call."""
    from torch.nn.attention import SDPBackend, sdpa_kernel

    return sdpa_kernel([SDPBackend.EFFICIENT_ATTENTION, SDPBackend.MATH])


def ref_causal_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float) -> tuple[torch.Tensor, torch.Tensor]:
    """fp32 ``(out [b, s, h, dv], lse [b, h, s])``."""
    s = q.shape[1]
    scores = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) * scale
    mask = torch.ones(s, s, dtype=torch.bool, device=q.device).tril()
    scores = scores.masked_fill(~mask, float("-inf"))
    lse = torch.logsumexp(scores, dim=-1)
    out = torch.einsum("bhqk,bkhg->bqhg", torch.softmax(scores, dim=-1), v.float())
    return out, lse


def supported(q: torch.Tensor, v: torch.Tensor) -> bool:
    return (
        q.is_cuda and q.ndim == 4 and v.ndim == 4 and q.shape[-1] in (64, 128) and v.shape[-1] % 64 == 0
        and q.shape[1] % 8 == 0 and q.shape[0] <= 65535
    )  # fmt: skip


def _operand(t: torch.Tensor) -> torch.Tensor:
    """``t`` as the kernels read it: bf16, contiguous, on a 16-byte boundary (a view into another tensor may start off one)."""
    t = t.detach().to(torch.bfloat16).contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


@torch.no_grad()
def causal_attention_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float | None = None,
                         want_lse: bool = False) -> tuple[torch.Tensor, torch.Tensor | None]:  # fmt: skip
    """``q, k [b, s, h, d_qk]``, ``v [b, s, h, d_v]`` -> bf16 ``out [b, s, h, d_v]`` (and fp32 ``lse [b, h, s]``)."""
    scale = 1.0 / math.sqrt(q.shape[-1]) if scale is None else scale
    if not supported(q, v):
        out, lse = ref_causal_attention(q, k, v, scale)
        return out.to(torch.bfloat16), (lse if want_lse else None)
    b, s, h, _ = q.shape
    q16, k16, v16 = (_operand(t) for t in (q, k, v))
    out = torch.empty(b, s, h, v.shape[-1], dtype=torch.bfloat16, device=q.device)
    lse = torch.empty(b, h, s, dtype=torch.float32, device=q.device) if want_lse else None
    K._ext().attn_fwd(q16, k16, v16, out, lse, float(scale), K.status_buffer(q.device))
    return out, lse


def causal_attention_bwd(q16, k16, v16, do16, lse, delta, scale: float, dtype: torch.dtype):
    """``(dq, dk, dv)`` in ``dtype`` (fp32, or bf16: fp32 sums rounded once) from contiguous bf16 ``[b, s, h, *]`` tensors and the row
    statistics ``lse``, ``delta [b, h, s]`` (``delta`` the dot products of output and output gradient). Two kernels."""
    dq, dk, dv = (torch.empty(t.shape, dtype=dtype, device=t.device) for t in (q16, k16, v16))
    K._ext().attn_bwd(q16, k16, v16, do16, lse, delta, dq, dk, dv, float(scale), K.status_buffer(q16.device))
    return dq, dk, dv


class CausalAttention(torch.autograd.Function):
    """Differentiable ``causal_attention_fwd``: three tcgen05 kernels (forward, dQ, dK/dV). Inputs of any float dtype are
    rounded to bf16 for the tensor cores; gradients are accumulated in fp32 and returned in the inputs' dtypes."""

    @staticmethod
    def forward(ctx, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float) -> torch.Tensor:
        q16, k16, v16 = (_operand(t) for t in (q, k, v))
        b, s, h, _ = q16.shape
        out = torch.empty(v16.shape, dtype=torch.bfloat16, device=q.device)
        lse = torch.empty(b, h, s, dtype=torch.float32, device=q.device)
        K._ext().attn_fwd(q16, k16, v16, out, lse, float(scale), K.status_buffer(q.device))
        ctx.save_for_backward(q16, k16, v16, out, lse)
        ctx.scale, ctx.dtypes = float(scale), (q.dtype, k.dtype, v.dtype)
        return out.to(v.dtype)

    @staticmethod
    def backward(ctx, dout: torch.Tensor):
        q16, k16, v16, out, lse = ctx.saved_tensors
        do16 = _operand(dout)
        delta = torch.empty_like(lse)
        K._ext().attn_delta(do16, out, delta)
        low = all(t == torch.bfloat16 for t in ctx.dtypes)
        dq, dk, dv = causal_attention_bwd(q16, k16, v16, do16, lse, delta, ctx.scale, torch.bfloat16 if low else torch.float32)
        return dq.to(ctx.dtypes[0]), dk.to(ctx.dtypes[1]), dv.to(ctx.dtypes[2]), None


def causal_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor | None = None, scale: float | None = None,
                     vt: torch.Tensor | None = None) -> torch.Tensor:  # fmt: skip
    """Differentiable causal attention ``[b, s, h, d_qk] x [b, s, h, d_v] -> [b, s, h, d_v]``; the tensor-core kernels
    when the shape is supported on a GPU, the torch oracle otherwise. The values may be given transposed instead, as
    ``vt [b, h, d_v, s]``, which costs a copy into the kernels' layout."""
    scale = 1.0 / math.sqrt(q.shape[-1]) if scale is None else scale
    if v is None and vt is None:
        raise ValueError("causal_attention takes the values as v or as vt")
    if vt is not None:
        v = vt.permute(0, 3, 1, 2)
    if not supported(q, v):
        return ref_causal_attention(q, k, v, scale)[0].to(v.dtype)
    return CausalAttention.apply(q, k, v, scale)
