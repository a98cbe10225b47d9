"""fp32 inference of a sparse dictionary on the GPU: TopK activation and decoder as kernels in place of dense tensor operations
(the eager statements of models/sae.py:288-377 and utils/math.py:81-171 in the reference project).

Both give what the dense operations give, NaN and infinities included, and neither makes the host wait. They apply to plain
forward passes only: whatever listens to or rewrites tensor operations (autograd, forward-mode differentiation, function
transforms, autocast, tracing, dispatch modes, tensor subclasses) gets the tensor operations."""

from __future__ import annotations

import torch
from torch.autograd import forward_ad
from torch.utils._python_dispatch import _get_current_dispatch_mode

from . import sae_kernels as K

MAX_K = 1024  # the selection kernel's bound comes from 2048 column groups
# bytes for the parts of W at a time (6 per element, 4 where it only proposes): 74 tiles of 256 features at d_model 4096, so that a piece still fills the GPU
PRODUCT_WORKSPACE = 512 << 20
MAX_ESTIMATE_WIDTH = 16384  # kEstimateMaxK in csrc/kernels.h


def plain_inference(*tensors: torch.Tensor) -> bool:
    """Whether nothing but the values of an operation on these CUDA tensors is wanted."""
    if torch.is_grad_enabled() and any(t.requires_grad for t in tensors):
        return False
    if not all(type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and t.dtype == torch.float32 for t in tensors):
        return False
    return not (
        any(t.device != tensors[0].device for t in tensors)
        or torch.is_autocast_enabled("cuda")
        or torch.jit.is_tracing()
        or torch.compiler.is_compiling()
        or forward_ad._current_level >= 0
        or torch._C._functorch.peek_interpreter_stack() is not None
        or _get_current_dispatch_mode() is not None
        or len(torch.overrides._get_current_function_mode_stack()) != 0
    )


def product_supported(x: torch.Tensor, W: torch.Tensor) -> bool:
    """``x [..., K] @ W [K, N]`` with the columns of ``W`` contiguous, large enough for the split of the operands to pay (it costs
    about what 60 rows cost on the fp32 pipes) and with full fp32 precision asked for."""
    K_, N = W.shape
    if x.ndim < 2 or x.shape[-1] != K_ or K_ % 4 != 0 or not 0 < K_ <= MAX_ESTIMATE_WIDTH or N == 0:
        return False
    M = x.numel() // K_
    return (M >= 256 and 2 * M * N * K_ >= 4e9 and M < 2**31 - 512 and N < 2**31 - 512 and x.is_contiguous()
            and W.t().is_contiguous() and x.data_ptr() % 16 == 0 and W.data_ptr() % 16 == 0
            and torch.get_float32_matmul_precision() == "highest")  # fmt: skip


def product(x: torch.Tensor, W: torch.Tensor) -> torch.Tensor:
    """``x @ W`` in fp32."""
    rows = x.detach().reshape(-1, x.shape[-1])
    out = torch.empty(rows.shape[0], W.shape[1], dtype=torch.float32, device=x.device)
    status = torch.zeros(4, dtype=torch.int32, device=x.device)
    K._ext().fp32_gemm(rows, W.detach().t(), out, status, None, None, None, None, True, PRODUCT_WORKSPACE)
    return out.view(*x.shape[:-1], W.shape[1])


def topk_dense_supported(h: torch.Tensor, k: int) -> bool:
    return h.ndim >= 1 and h.is_contiguous() and 1 <= k <= MAX_K and 0 < h.numel() < 2**62 and 0 < h.shape[-1] < 2**31 - 64


def topk_dense(h: torch.Tensor, bias: torch.Tensor | None, norm: torch.Tensor | None, k: int) -> torch.Tensor:
    """``topk(relu((h + bias) * norm)) / norm`` over the last dimension (``bias`` and ``norm`` optional)."""
    rows = h.reshape(-1, h.shape[-1])
    out = torch.empty_like(rows)
    K._ext().topk_dense(rows, bias.contiguous() if bias is not None else None, norm.contiguous() if norm is not None else None, k, out)
    return out.view(h.shape)


def half_product_pays(F: int, k: int) -> bool:
    """Whether one fp16 product proposes instead of three bf16 products of two parts. Its bound is five times as wide, so that about a sixth
    of ``k`` entries more are summed up, which costs more than two products save once ``k`` is a larger share of the features
    (4096 x 768 inputs, 32768 features: k 512 2.06 -> 2.17 ms; 24576 features: k 50 638 -> 465 us), and it selects by the maxima of 32 columns."""
    return F >= 128 * k


def topk_encode(x: torch.Tensor, W: torch.Tensor, bias: torch.Tensor | None, norm: torch.Tensor | None, k: int) -> torch.Tensor:
    """``topk_dense(x @ W, ...)`` for operands of ``product``: a coarser product proposes, and what it leaves in question is summed in
    ascending order of the input dimension, so that neither the choice nor the values depend on how it was made."""
    rows = x.detach().reshape(-1, x.shape[-1])
    B, F = rows.shape[0], W.shape[1]
    out = torch.empty(B, F, dtype=torch.float32, device=x.device)
    bias, norm = (t.contiguous() if t is not None else None for t in (bias, norm))
    if half_product_pays(F, k):
        K._ext().topk_encode(rows, W.detach().t(), bias, norm, k, PRODUCT_WORKSPACE, out)
        return out.view(*x.shape[:-1], F)
    h = torch.empty(B, F, dtype=torch.float32, device=x.device)
    lo = h.view(-1).view(torch.bfloat16)[: B * F].view(B, F)  # (read before anything is written to h)
    xn = torch.empty(B, dtype=torch.float32, device=x.device)
    widths = 4 + (F + 1) // 2  # (the columns' widths as bf16 behind four words)
    words = torch.zeros(4 + widths + 1 + B, dtype=torch.int32, device=x.device)
    status, top, todo = words[:4], words[4 : 4 + widths], words[4 + widths :]
    K._ext().fp32_gemm(rows, W.detach().t(), lo, status, xn, top, bias, norm, True, PRODUCT_WORKSPACE)
    K._ext().topk_estimate(lo, h, rows, W.detach().t(), xn, top, bias, norm, k, status, todo, out)
    return out.view(*x.shape[:-1], F)


def sparse_decode_supported(acts: torch.Tensor, W: torch.Tensor) -> bool:
    """Aligned operands, and a product that takes longer than the kernels that replace it: they need 24 us of launches, which a library
    product of 1e9 operations exceeds where features are many (256 x 4096 x 512: 67 us), and with few features, of which a token's
    50 codes are a larger share, one of 4e9 (4096 x 1024 x 256, 2.1e9: 45 against 55 us; 4096 x 1024 x 768, 6.4e9: 137 against 73 us)."""
    F, d = W.shape
    if not (acts.ndim >= 2 and acts.shape[-1] == F and acts.is_contiguous() and W.is_contiguous() and F % 4 == 0 and d % 4 == 0 and F > 0 and d > 0):
        return False
    B = acts.numel() // F
    return (2 * B * F * d >= (1e9 if F >= 4096 else 4e9) and acts.data_ptr() % 16 == 0 and W.data_ptr() % 16 == 0
            and F < 2**31 - 64 and 0 < B < 2**31 - 64)  # fmt: skip


def decode_bias_supported(acts: torch.Tensor, W: torch.Tensor, bias: torch.Tensor) -> bool:
    """Whether ``sparse_decode`` can add this bias: one aligned value per column of ``W``, nothing else wanted of the sum."""
    return plain_inference(acts, bias) and bias.shape == W.shape[1:] and bias.is_contiguous() and bias.data_ptr() % 16 == 0


def most_gathered(F: int) -> int:
    """Non-zeros of a row up to which gathering beats the product of the rows that are left over: 4096 tokens x 2048 x 768, 443 us as a
    product, 222 us gathered at 12 % and 805 us at 50 % (4096 x 8192 x 768: 1684 us against 793 us at 12 %)."""
    return F // 6


def sparse_decode(acts: torch.Tensor, W: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """``acts @ W`` (``+ bias [d]``) for ``acts [..., F]`` with few non-zeros; rows with more than ``most_gathered`` go to a product on the fp32 pipes."""
    rows = acts.reshape(-1, acts.shape[-1])
    (B, F), d = rows.shape, W.shape[1]
    tiles = min(512, -(-B // 128) * -(-d // 128) * 16)
    out = torch.empty(B, d, dtype=torch.float32, device=acts.device)
    part = torch.empty(tiles * 128 * 128, dtype=torch.float32, device=acts.device)
    todo = torch.zeros(2 + B + tiles, dtype=torch.int32, device=acts.device)
    K._ext().dense_decode(rows, W.detach(), bias.detach() if bias is not None else None, most_gathered(F), todo, part, out)
    return out.view(*acts.shape[:-1], d)
