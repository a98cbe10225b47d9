"""The list kernel of the JumpReLU step against the same arithmetic in 64 bits: the penalty's derivatives where 1 - tanh^2 cancels,
and which entries are active at the threshold itself."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,stretch", [(1, 1.0), (3, 4.0)])
def test_penalty_terms_keep_fp32_precision(H, stretch):
    g = torch.Generator().manual_seed(H)
    B, cap, F = 5, 24, 120
    idx = torch.stack([torch.randperm(F, generator=g)[:cap] for _ in range(B)]).to(torch.int32)
    idx[1, 7:] = -1
    norm = torch.rand(H, F, generator=g) + 0.5
    theta = torch.rand(F, generator=g) * 0.1 + 0.01
    valid, f = idx >= 0, idx.clamp_min(0).long()
    # up to stretch * s * norm of about 4, where sech^2 is 1e-3
    s = torch.rand(B, cap, generator=g) * 2.6 / stretch + 1e-3
    s[0, :] = (theta / norm[0])[f[0]]  # at head 0's threshold: inactive there
    s[2, :] = torch.nextafter((theta / norm[0])[f[2]], torch.tensor(float("inf")))  # just above it: active
    z = lambda *shape: torch.zeros(*shape, device=DEV)  # noqa: E731
    act, dS, pull, dtheta, u_sum = z(H, B, cap), z(B, cap), z(H, F), z(F), z(1)
    n_valid = torch.zeros(1, dtype=torch.int32, device=DEV)
    K._ext().jumprelu_lists(idx.to(DEV), s.to(DEV), norm.to(DEV), theta.to(DEV), stretch, 0.7, 1e-9, act, dS, pull, dtheta, u_sum, n_valid)
    want_dS, want_pull, want_u = torch.zeros(B, cap, dtype=torch.float64), torch.zeros(H, F, dtype=torch.float64), 0.0
    for h in range(H):
        n = norm[h][f]
        active = valid & (s > (theta / norm[h])[f])
        got = act[h].cpu()
        assert torch.equal(torch.where(valid, got, 0.0), torch.where(active, s, 0.0))
        u = torch.tanh(stretch * s.double() * n.double())
        want_u += float(u[active].sum())
        sech2 = (1 - u * u) * active
        want_dS += 0.7 * n.double() * sech2
        want_pull[h].index_add_(0, f.reshape(-1), (0.7 * s.double() * sech2).reshape(-1))
    # the argument's rounding, 2^-23 relative, moves sech^2 by 2 * argument (<= 4) of that; a few more roundings of 2^-24
    tol = 2.0**-24 * (2 * 2 * 4 + 4 + H)
    err = ((dS.cpu().double() - want_dS).abs() / want_dS.clamp_min(1e-30))[valid & (want_dS > 0)]
    assert float(err.max()) <= tol
    assert torch.allclose(pull.cpu().double(), want_pull, rtol=tol + 2.0**-24 * B, atol=0)
    assert abs(float(u_sum) - want_u) <= 2.0**-23 * 8 * want_u and int(n_valid) == int(valid.sum())
