"""fp32 TopK codes by one fp16 product: what its kernels store against 64 bits, a dictionary in pieces, and what becomes of rows when the product gave up."""

import pytest
import torch
from test_fp32_product_gpu import _in_order

from language_model_saes_b200.ops import inference as I
from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _same(out, want):
    differ = (out.nan_to_num(nan=-1.0) != want.nan_to_num(nan=-1.0)).nonzero()
    assert differ.numel() == 0, (differ[:4], len(differ))


def _data(B, F, K_, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x, w = torch.randn(B, K_, device=DEV, generator=g), torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    return x, w, 0.1 * torch.randn(F, device=DEV, generator=g), torch.rand(F, device=DEV, generator=g) + 0.5


@pytest.mark.parametrize("B,F,K_,k,workspace", [(257, 1153, 64, 9, 1), (270, 4104, 132, 32, 1), (130, 9001, 68, 50, 4 * 128 * 512 * 4), (300, 2049, 1028, 16, 1)])
@pytest.mark.parametrize("data", ["normal", "loss in the last piece", "cancelling", "bad columns", "no gate"])
def test_pieces(B, F, K_, k, workspace, data, monkeypatch):
    """Pieces of one tile and of several, the last one ragged; rows decided by the first proposal, and more than an eighth of them by the second."""
    assert I.half_product_pays(F, k)
    x, w, bias, norm = _data(B, F, K_, F)
    if data == "loss in the last piece":  # fp16 takes nothing of the rows before it, and as much as it can of those
        w = torch.exp2(torch.floor(torch.log2(w.abs() + 1e-3))) * w.sign()
        w[-5:] *= 1 + 2.0**-11
    elif data == "cancelling":  # a common offset that the bias takes away
        w *= 1e-3
        x[:, 0], w[:, 0] = 1000.0, 1.0
        bias = bias * 1e-3 - 1000.0
        norm[:] = 1.0
    elif data == "bad columns":
        w[2, 0], w[300, 1], w[F - 3, 1], w[F - 1] = float("nan"), 3e38, float("inf"), 0.0
        norm[F - 2], bias[F - 4] = 0.0, 1e25
    elif data == "no gate":
        bias = norm = None
    whole = I.topk_encode(x, w.t(), bias, norm, k)
    monkeypatch.setattr(I, "PRODUCT_WORKSPACE", workspace)
    before = K.kernel_launch_count()
    pieces = I.topk_encode(x, w.t(), bias, norm, k)
    assert K.kernel_launch_count() - before == 5 + 4 * -(-F // (max(1, workspace // (-(-K_ // 64) * 64 * 1024)) * 256))
    _same(pieces, whole)
    _same(pieces, I.topk_dense(_in_order(x, w), bias, norm, k))


@pytest.mark.parametrize("B,F,K_,k,workspace", [(300, 2561, 128, 20, 1 << 29), (257, 8200, 72, 64, 1)])
def test_products_that_gave_up(B, F, K_, k, workspace):
    """Every row goes through both selections to the products in order, whatever the ends are."""
    x, w, bias, norm = _data(B, F, K_, F)
    out = torch.full((B, F), float("nan"), device=DEV)
    *_, words = K._ext().topk_encode(x, w, bias, norm, k, workspace, out, True)
    for rows in words[4 + 4 + (F + 1) // 2 :].view(2, 1 + B):  # those too wide for the first selection, and those multiplied as a whole
        assert rows[0] == B and torch.equal(rows[1:].sort().values, torch.arange(B, dtype=torch.int32, device=DEV))
    _same(out, I.topk_dense(_in_order(x, w), bias, norm, k))


@pytest.mark.parametrize("B,F,K_,k", [(300, 2056, 768, 16), (129, 1025, 68, 8), (64, 1024, 16384, 2), (40, 1031, 1028, 8)])
@pytest.mark.parametrize("data", ["normal", "limits", "most loss"])
def test_stored_ends_enclose_the_activations(B, F, K_, k, data):
    """The ends and maxima that the selection reads: every end is at most the activation of the sum in order, which is at most the end, 2^-7 of
    it and the width more; norms, scales and losses are those of 64 bits, rounded up."""
    x, w, bias, norm = _data(B, F, K_, K_)
    if data == "limits":  # rows at either end of what a scale covers (the largest magnitude from 2^-40 to 2^30)
        for t, n in ((x, 2), (w, 3)):
            top = t.abs().amax(1)
            t[:n] *= (2.0**-39.9 / top[:n])[:, None]
            t[n : 2 * n] *= (2.0**29.9 / top[n : 2 * n])[:, None]
        bias[:6] = 0.0
    elif data == "most loss":
        x, w = (torch.exp2(torch.floor(torch.log2(t.abs() + 1e-3))) * t.sign() * (1 + 2.0**-11) for t in (x, w))
    out = torch.empty(B, F, device=DEV)
    h, maxima, norms, words = K._ext().topk_encode(x, w, bias, norm, k, 1 << 29, out, False)
    _same(out, I.topk_dense(_in_order(x, w), bias, norm, k))
    wide, todo = words[4 + 4 + (F + 1) // 2 :].view(2, 1 + B)[:, 0].tolist()
    assert wide <= B // 8 and todo == 0, "the ends have been written over: these data say nothing"
    top = words[4:].view(torch.float32)
    xn, _, lost = norms[: 3 * B].view(3, B)
    at = 3 * B + -3 * B % 4
    wn = norms[at : at + F]
    x64, w64 = x.double(), w.double()

    def half(t):  # fp16 with the row's largest magnitude in [2^14, 2^15) and nothing below 2^-14
        scale = torch.exp2(14 - torch.floor(torch.log2(t.abs().amax(1, keepdim=True))))
        s = t * scale
        return torch.where(s.abs() < 2.0**-14, 0.0, s.float().half().double()) / scale

    for n, t in ((xn, x64), (wn, w64)):
        assert ((n >= t.norm(dim=1)) & (n <= 1.002 * t.norm(dim=1))).all()
    loss = lambda t: (half(t) - t).norm(dim=1) / t.norm(dim=1)  # noqa: E731
    assert ((lost >= loss(x64)) & (lost <= 1.004 * loss(x64) + 1e-7)).all()
    assert loss(w64).max() <= top[2] <= 1.004 * loss(w64).max() + 1e-7
    act = ((_in_order(x, w) + bias) * norm).double()
    lo = h.view(-1).view(torch.bfloat16)[: B * F].view(B, F)
    assert lo.isfinite().all()
    lo64 = lo.double()
    rel = (2.1 * K_ + 136) * 2.0**-24 + lost.double() + top[2].double()
    width = 2 * (rel * 1.000002 + 1e-6)[:, None] * xn.double()[:, None] * (wn * norm).double()
    # (the selection's claim is about what is positive; a product of a rounded sum and a gate keeps its order)
    assert ((lo64 <= act) | (act <= 0)).all()
    assert (act <= lo64 + 2.0**-7 * lo64.abs() + width + 1e-37).all()
    assert float(((act - lo64) / (width + 2.0**-7 * lo64.abs())).mean()) > 0.1  # (and is no wider than it need be)
    padded = torch.cat([lo, torch.zeros(B, maxima.shape[1] * 32 - F, dtype=lo.dtype, device=DEV)], 1).view(B, -1, 32)
    bits = maxima.view(torch.int32)
    assert torch.equal((bits & -65536).view(torch.float32), padded.float().nan_to_num(nan=0.0).amax(-1).clamp_min(0.0))
    assert torch.equal((bits & 1).bool(), padded.isnan().any(-1))
