"""The kernels of fp32 inference against the tensor operations they stand for: row lengths around a vector and a CTA, unaligned
rows, every number of features kept, repeated values, NaN, infinities and zero norms; decoders with sparse rows, rows too dense
for the lists, and weights that are not finite; and the calls that have to take the tensor operations as before."""

import pytest
import torch

from language_model_saes_b200 import SAEConfig, SparseAutoEncoder
from language_model_saes_b200.ops import inference as I
from language_model_saes_b200.utils.math import topk

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("F", [1, 7, 64, 2047, 2052, 24576, 50001])
@pytest.mark.parametrize("k", [1, 50, 1024])
@pytest.mark.parametrize("data", ["normal", "few", "repeated", "special"])
@pytest.mark.parametrize("parts", ["both", "none"])
def test_topk_activation(F, k, data, parts):
    g = torch.Generator().manual_seed(F + k)
    h = torch.randn(4, F, generator=g)
    if data == "few":
        h -= 3.0
    elif data == "repeated":
        h = h.sign() * 0.5
        h[:, ::9] = 1.5
    bias, norm = (0.1 * torch.randn(F, generator=g), torch.rand(F, generator=g) + 0.5) if parts == "both" and data != "repeated" else (None, None)
    if data == "special":
        h[0, :: max(1, F // 5)] = float("nan")
        h[0, F // 5 // 2 if F >= 10 else 0] = float("inf")  # selected only if the NaNs leave a place (which of equals is kept is free)
        h[1, F - 1] = float("inf")
        h[2, F // 2] = -float("inf")
        if norm is not None:
            norm[F // 3] = 0.0
    k = min(k, F)
    h, bias, norm = (t.to(DEV) if t is not None else None for t in (h, bias, norm))
    out = I.topk_dense(h, bias, norm, k)
    g_ = h + bias if bias is not None else h
    g_ = g_ * norm if norm is not None else g_
    r = g_ * g_.gt(0).to(g_.dtype)
    want = topk(r, k=k)
    want = want / norm if norm is not None else want
    assert torch.equal(out.isnan(), want.isnan())
    if data == "repeated":  # which of the equal values are kept is free
        assert torch.equal(out.sort(-1).values, want.sort(-1).values)
        assert ((out == 0) | (out == h)).all()
    else:
        assert torch.equal(out.nan_to_num(nan=-1.0), want.nan_to_num(nan=-1.0))


@pytest.mark.parametrize("B,F,d", [(1, 4, 4), (130, 1000, 64), (5, 24576, 768), (3, 4100, 1028), (129, 512, 256)])
@pytest.mark.parametrize("rows", ["sparse", "some dense", "all dense", "at the limit", "inf weight"])
def test_decoder(B, F, d, rows):
    g = torch.Generator().manual_seed(B + F)
    a = torch.randn(B, F, generator=g) * (torch.rand(B, F, generator=g) < 20 / F)
    W = torch.randn(F, d, generator=g)
    if rows == "some dense":
        a[B // 2] = torch.randn(F, generator=g)
        a[0] = 0.0
    elif rows == "all dense":
        a = torch.randn(B, F, generator=g)
    elif rows == "at the limit":  # as many non-zeros as a row that is gathered may have, and one more
        n = min(I.most_gathered(F), 8 * 256 // 2)
        a.zero_()
        a[:, torch.randperm(F, generator=g)[:n]] = 1.5
        a[::2, (a[0] == 0).nonzero()[0]] = -1.0
    elif rows == "inf weight":
        W[F // 2, 1] = float("inf")
    out = I.sparse_decode(a.to(DEV), W.to(DEV)).cpu()
    want = a.double() @ W.double()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    # fp32 sums: 2^-24 of the sum of magnitudes for each of the non-zero terms
    n = (a != 0).sum(1, keepdim=True) + 1
    bound = 2.0**-24 * n * (a.double().abs() @ W.double().abs().nan_to_num(posinf=1.0)) + 1e-30
    ok = want.isfinite()
    assert ((out.double() - want).abs()[ok] <= bound.expand_as(want)[ok]).all()


@pytest.mark.parametrize("rows", ["sparse", "some dense", "all dense", "inf weight"])
@pytest.mark.parametrize("B,F,d", [(130, 1000, 64), (3, 4100, 1028), (129, 512, 256)])
def test_decoder_with_its_bias_is_the_sum_of_both(B, F, d, rows):
    """One rounding of the finished sum, by whichever way a row is made: the same as adding the bias afterwards."""
    g = torch.Generator().manual_seed(F)
    a, W, b = torch.randn(B, F, generator=g), torch.randn(F, d, generator=g), torch.randn(d, generator=g)
    if rows != "all dense":
        a[1 if rows == "some dense" else 0 :] *= torch.rand(B - (rows == "some dense"), F, generator=g) < 20 / F
    if rows == "inf weight":
        W[F // 2, 1] = float("inf")
    b[3] = float("inf")
    a, W, b = a.to(DEV), W.to(DEV), b.to(DEV)
    out, want = I.sparse_decode(a, W, b), I.sparse_decode(a, W) + b
    assert torch.equal(out.nan_to_num(nan=7.0), want.nan_to_num(nan=7.0))


@pytest.mark.parametrize("bias", ["a column", "unaligned", "one value", "as it is"])
def test_decode_takes_a_bias_of_any_layout(bias):
    sae = _sae("topk", 64)
    values = torch.randn(64, device=DEV)
    if bias == "a column":
        sae.b_D = torch.nn.Parameter(values[:, None].repeat(1, 3)[:, 0])
    elif bias == "unaligned":
        sae.b_D = torch.nn.Parameter(torch.cat([values[:1], values])[1:])
    else:
        sae.b_D = torch.nn.Parameter(values[:1].clone() if bias == "one value" else values)
    with torch.no_grad():
        acts = sae.encode(torch.randn(2048, 64, device=DEV))
        assert sae._sparse_inference(acts)
        assert torch.equal(sae.decode(acts), I.sparse_decode(acts, sae.W_D) + sae.b_D)


def _sae(act, expansion=8):
    torch.manual_seed(0)
    cfg = SAEConfig(hook_point_in="h", hook_point_out="h", d_model=64, expansion_factor=expansion, act_fn=act, top_k=10, device=DEV, dtype=torch.float32)
    sae = SparseAutoEncoder(cfg)
    sae.init_parameters(encoder_uniform_bound=0.2, decoder_uniform_bound=0.2, init_log_jumprelu_threshold_value=-1.0)
    return sae


@pytest.mark.parametrize("act", ["topk", "jumprelu"])
def test_model_routes(act):
    sae = _sae(act)
    x = torch.randn(3, 5, 64, device=DEV)
    acts = sae.encode(x)  # with autograd: tensor operations
    rec = sae.decode(acts)
    assert acts.requires_grad and rec.requires_grad
    with torch.no_grad():
        a, r = sae.encode(x), sae.decode(acts.detach())
        a2, h2 = sae.encode(x, return_hidden_pre=True)
        assert a.shape == acts.shape and r.shape == rec.shape and h2.shape == acts.shape
        assert torch.equal(a, acts) and torch.equal(a2, a)
        assert torch.allclose(r, rec, atol=1e-5)
        seen = []
        sae.hook_hidden_pre.add_hook(lambda t, hook: seen.append(t) or t * 0)
        assert not sae.encode(x).any() and len(seen) == 1
        sae.hook_hidden_pre.remove_hooks()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert not sae._rowwise_topk_inference(x) and not sae._sparse_inference(a)
            assert torch.equal(sae.decode(a), a @ sae.W_D + sae.b_D)
        if act == "topk":
            assert torch.allclose(torch.vmap(lambda t: sae.decode(sae.encode(t)))(x), r, atol=1e-5)
            _, tangent = torch.func.jvp(lambda t: sae.decode(sae.encode(t)), (x,), (torch.ones_like(x),))
            assert tangent.any()


@pytest.mark.parametrize("form", ["kernel", "contiguous W_E", "matmul precision"])
def test_encode_takes_the_estimating_product(form, monkeypatch):
    """Above the size from which the split product pays, ``encode`` runs it, and only on the operands it is made for."""
    torch.manual_seed(0)
    cfg = SAEConfig(hook_point_in="h", hook_point_out="h", d_model=512, expansion_factor=16, act_fn="topk", top_k=20, device=DEV, dtype=torch.float32)
    sae = SparseAutoEncoder(cfg)
    sae.init_parameters(encoder_uniform_bound=0.05, decoder_uniform_bound=0.05, init_log_jumprelu_threshold_value=0.0)
    sae.b_E.data.normal_(0.0, 0.1)
    if form == "contiguous W_E":
        sae.W_E = torch.nn.Parameter(sae.W_E.detach().contiguous())
    x = torch.randn(2, 256, 512, device=DEV)
    calls = []
    made = I.topk_encode
    monkeypatch.setattr(I, "topk_encode", lambda *a: calls.append(1) or made(*a))
    before = torch.get_float32_matmul_precision()
    try:
        if form == "matmul precision":
            torch.set_float32_matmul_precision("high")
        with torch.no_grad():
            acts = sae.encode(x)
    finally:
        torch.set_float32_matmul_precision(before)
    assert len(calls) == (form == "kernel") and acts.shape == (2, 256, 8192)
    if form == "matmul precision":  # (tf32 codes may differ by more than ties)
        return
    norm = sae.decoder_norm().double()
    h = (x.double() @ sae.W_E.double() + sae.b_E.double()) * norm
    want = topk(h.clamp_min(0.0), k=20) / norm
    same = (acts != 0) == (want != 0)
    # fp32 sums of 512 terms: a choice may differ where the k-th values are that close, which hardly a row has
    assert (~same).any(-1).float().mean() < 0.01
    bound = 512 * 2.0**-24 * (x.double().abs() @ sae.W_E.double().abs() + sae.b_E.double().abs())
    assert ((acts.double() - want).abs() <= bound + 1e-12)[same].all()


def test_decoder_of_a_dictionary_longer_than_the_batch():
    """More CTAs look through W than rows are gathered: what they find in any part of it counts."""
    B, F, d = 5, 4096, 4096
    a = torch.zeros(B, F, device=DEV)
    a[:, ::200] = 1.0
    W = torch.randn(F, d, device=DEV)
    want = I.sparse_decode(a, W)
    assert torch.allclose(want, W[::200].sum(0).expand(B, d), atol=1e-4)
    for row in (1, F // 2, F - 1):  # (features that are never active: 0 * inf)
        V = W.clone()
        V[row, d - 1 - row % 7] = float("inf")
        out = I.sparse_decode(a, V)
        assert bool(out[:, d - 1 - row % 7].isnan().all()) and int(out.isnan().sum()) == B
        assert torch.allclose(out.nan_to_num(nan=0.0), want.masked_fill(out.isnan(), 0.0), atol=1e-4)
