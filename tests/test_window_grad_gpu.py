"""The threshold gradient in the epilogue of its product against the plain statement."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K
from language_model_saes_b200.ops import select_kernels as S

pytestmark = pytest.mark.gpu


# one tile; part of a tile of tokens, features and columns; features behind an odd 128-row panel; more panels than CTA pairs; long rows
@pytest.mark.parametrize("B,F,d", [(256, 256, 64), (1, 8, 8), (77, 136, 72), (300, 392, 768), (513, 19 * 1024 + 8, 64), (1030, 600, 2304)])
@pytest.mark.parametrize("add", [0.0, 0.01])
def test_window_gradient_of_product_matches_the_plain_statement(B, F, d, add):
    g = torch.Generator(device="cuda").manual_seed(0)
    dx = torch.randn(B, d, device="cuda", generator=g).to(torch.bfloat16)
    W = torch.randn(F, d, device="cuda", generator=g).to(torch.bfloat16)
    s = torch.randn(B, F, device="cuda", generator=g).to(torch.bfloat16)
    n = 0.5 + torch.rand(F, device="cuda", generator=g)
    theta = 0.2 + torch.rand(F, device="cuda", generator=g)
    start = torch.randn(F, device="cuda", generator=g)
    got = start.clone()
    S.jumprelu_window_grad_of_product(dx, W, s, n, theta, 1.0, got, add)
    K.check_status(torch.device("cuda"))
    G = dx.double() @ W.double().t()
    x = s.float() * n  # (the kernel's own product and differences, so that the same entries are inside)
    hit = (x > 0) & ((x - theta).abs() < 0.5)
    terms = torch.where(hit, G / n.double() + add, torch.zeros((), dtype=torch.float64, device="cuda")) * (-theta.double() / 1.0)
    want = start.double() + terms.sum(0)
    # fp32 sums: of d products per entry, and of the entries of a feature
    size = torch.where(hit, (dx.double().abs() @ W.double().abs().t()) / n.double() + add, torch.zeros((), dtype=torch.float64, device="cuda")).sum(0) * theta.double()
    bound = (d + B + 8) * 2.0**-24 * (size + start.double().abs())
    assert bool(((got.double() - want).abs() <= bound).all()), float(((got.double() - want).abs() / bound.clamp_min(1e-30)).max())
