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


@pytest.mark.parametrize("B,F,d", [(300, 520, 136), (77, 264, 64)])
def test_what_is_not_finite_shows_where_it_is_inside(B, F, d):
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)  # noqa: E731
    dx, W, s = rand(B, d).to(torch.bfloat16), rand(F, d).to(torch.bfloat16), rand(B, F).to(torch.bfloat16)
    n, theta = 0.5 + torch.rand(F, device="cuda", generator=g), 0.2 + torch.rand(F, device="cuda", generator=g)
    dx[3, 5], dx[B - 1, 0] = float("nan"), float("inf")  # (the last token's tile ends with tokens that do not exist)
    W[7, 2], W[F - 1, 3] = float("inf"), float("nan")
    s[11, 20], s[12, 21], s[13, 22] = float("nan"), float("inf"), -float("inf")
    n[30], n[31], theta[40], theta[41] = 0.0, float("inf"), float("nan"), float("inf")
    s[3, 50:400] = s[B - 1, 50:400] = -1.0  # (features without a bad token)
    got = torch.zeros(F, device="cuda")
    S.jumprelu_window_grad_of_product(dx, W, s, n, theta, 1.0, got, 0.01)
    K.check_status(torch.device("cuda"))
    x = s.float() * n
    hit = (x > 0) & ((x - theta).abs() < 0.5)
    zero = torch.zeros((), dtype=torch.float64, device="cuda")
    want = torch.where(hit, (dx.double() @ W.double().t()) / n.double() + 0.01, zero).sum(0) * torch.where(hit.any(0), -theta.double(), zero)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fine = want.isfinite()
    assert int(fine.sum()) > 150 and int((~fine).sum()) > 10
    size = torch.where(hit, (dx.double().abs() @ W.double().abs().t()) / n.double() + 0.01, zero).sum(0) * torch.where(hit.any(0), theta.double().abs(), zero)
    assert bool(((got.double() - want).abs() <= (d + B + 8) * 2.0**-24 * size)[fine].all())
