"""The sparse decoder's per-row loss, the same sum every time and against 64 bits, and entries whose coefficient is zero."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,d", [(5, 64), (300, 768), (37, 1160), (512, 8192)])
def test_row_loss(B, d):
    g = torch.Generator(device=DEV).manual_seed(d)
    F, k = 200, 7
    idx = torch.randint(0, F, (B, k), device=DEV, dtype=torch.int32, generator=g)
    val, W = torch.rand(B, k, device=DEV, generator=g), torch.randn(F, d, device=DEV, generator=g).to(torch.bfloat16)
    label, bias = torch.randn(B, d, device=DEV, generator=g).to(torch.bfloat16), torch.randn(d, device=DEV, generator=g)
    losses = []
    for _ in range(30):
        row = torch.full((B,), 7.0, device=DEV)
        K.sparse_decode_loss(idx, val, W, bias, label, None, 1.0, torch.zeros(1, device=DEV), row_loss=row)
        losses.append(row)
    assert all(torch.equal(losses[0], r) for r in losses)
    want = ((val.double().unsqueeze(-1) * W.double()[idx.long()]).sum(1) + bias - label.double()).square().sum(-1)
    # the reconstruction's k + 1 roundings, doubled by the square, and those of d / 32 terms per lane and the trees above them
    assert torch.allclose(losses[0].double(), want, rtol=2.0**-24 * (2 * (k + 1) * 8 + d / 32 + 16), atol=0)


@pytest.mark.parametrize("d", [64, 2048])
def test_a_row_that_is_not_finite_shows_under_a_zero_coefficient(d):
    idx = torch.tensor([[3, 5, -1], [1, 4, 0]], dtype=torch.int32, device=DEV)
    val = torch.tensor([[1.0, 0.0, 0.0], [1.0, 2.0, 0.0]], device=DEV)
    W = torch.ones(6, d, device=DEV, dtype=torch.bfloat16)
    W[5, 1], W[0, 2] = float("nan"), float("inf")
    out = K.sparse_decode(idx, val, W, None, torch.float32).cpu()
    want = torch.tensor([[1.0], [3.0]]).expand(2, d).clone()
    want[0, 1], want[1, 2] = float("nan"), float("nan")
    assert torch.equal(out.nan_to_num(nan=-1.0), want.nan_to_num(nan=-1.0))
