"""Masking in place with column sums against the plain statement."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

DEVICES = [pytest.param("cuda", marks=pytest.mark.gpu), "cpu"]


@pytest.mark.parametrize("dev", DEVICES)
@pytest.mark.parametrize("rows,d,pad", [(1, 8, 0), (33, 264, 8), (1000, 2056, 8), (70, 12, 4)])
def test_mask_colsum(dev, rows, d, pad):
    gen = torch.Generator(device=dev).manual_seed(rows)
    g = torch.randn(rows, d, device=dev, generator=gen).to(torch.bfloat16)
    wide = torch.randn(rows, d + pad, device=dev, generator=gen) * (torch.rand(rows, d + pad, device=dev, generator=gen) < 0.2)
    mask = wide.to(torch.bfloat16)[:, :d]
    mask[0, 0], mask[-1, -1] = -0.0, float("nan")  # (a NaN is not zero)
    want = torch.where(mask != 0, g, torch.zeros_like(g))
    got, sums = K.mask_colsum_(g.clone(), mask)
    assert torch.equal(got, want)
    exact = want.double().sum(0)
    assert bool(((sums.double() - exact).abs() <= rows * 2.0**-24 * want.double().abs().sum(0)).all())
