"""Kernels around the low-rank sparse attention step: Adam on transposed projections, and the pre-activation gradient with the attention
backward's row statistics from the codes."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

DEVICES = [pytest.param("cuda", marks=pytest.mark.gpu), "cpu"]
HYPER = (1e-2, 0.9, 0.999, 1e-8)


def _rand(dev, *shape, seed=0):
    return torch.randn(*shape, device=dev, generator=torch.Generator(device=dev).manual_seed(seed))


def _ref(p, m, v, g, step):
    p, m, v = p.double(), m.double(), v.double()
    K.ref_adam(p, g.double(), m, v, *HYPER, step)
    return p, m, v


@pytest.mark.parametrize("dev", DEVICES)
@pytest.mark.parametrize("heads,d,w,sets", [(1, 8, 8, 1), (2, 64, 64, 2), (3, 72, 16, 2), (2, 200, 136, 1), (2, 70, 68, 2), (1, 9, 5, 1)])
def test_adam_on_turned_gradients(dev, heads, d, w, sets):
    params = [_rand(dev, heads, d, w, seed=i) for i in range(sets)]
    moments = [(0.1 * _rand(dev, heads, d, w, seed=10 + i), _rand(dev, heads, d, w, seed=20 + i).square()) for i in range(sets)]
    grads = [_rand(dev, heads * w, d, seed=30 + i) for i in range(sets)]
    shadows = [torch.empty(heads * w, d, dtype=torch.bfloat16, device=dev) for _ in range(sets)]
    want = [_ref(p, m, v, g.view(heads, w, d).permute(0, 2, 1), 3) for p, (m, v), g in zip(params, moments, grads)]
    K.adam_turned(params, moments, grads, shadows, *HYPER, 3)
    for p, (m, v), sh, ref in zip(params, moments, shadows, want):
        for got, r in zip((p, m, v), ref):
            assert torch.allclose(got.double(), r, rtol=1e-5, atol=1e-6)  # a handful of fp32 roundings
        assert torch.equal(sh, p.permute(0, 2, 1).reshape(heads * w, d).to(torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("d,w", [(4, 4), (3, 70)])
def test_adam_on_more_heads_than_a_grid_dimension_holds(d, w):
    heads = 65537
    p, m, g = (_rand("cuda", *s, seed=i) for i, s in enumerate(((heads, d, w), (heads, d, w), (heads * w, d))))
    v, shadow = 0.5 + torch.rand(heads, d, w, device="cuda"), torch.empty(heads * w, d, dtype=torch.bfloat16, device="cuda")
    want = _ref(p, m, v, g.view(heads, w, d).permute(0, 2, 1), 3)
    K.adam_turned([p], [(m, v)], [g], [shadow], *HYPER, 3)
    for got, r in zip((p, m, v), want):  # (second moments of 0.5 and more: an update is of the learning rate's size, as are its roundings)
        assert torch.allclose(got.double(), r, rtol=1e-5, atol=1e-6)
    assert torch.equal(shadow, p.permute(0, 2, 1).reshape(heads * w, d).to(torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("b,s,heads,group,k", [(1, 8, 1, 8, 1), (2, 24, 3, 64, 7), (1, 40, 300, 8, 513), (2, 16, 64, 128, 128)])
def test_pre_activation_gradient_and_statistics_from_codes(b, s, heads, group, k):
    F, T = heads * group, b * s
    g = torch.Generator(device="cuda").manual_seed(0)
    idx = torch.rand(T, F, device="cuda", generator=g).topk(min(k, F), dim=1).indices.to(torch.int32)
    idx[torch.rand(idx.shape, device="cuda", generator=g) < 0.2] = -1  # empty slots, also in front of others
    act, dact = (torch.randn(idx.shape, device="cuda", generator=g) for _ in range(2))
    dz = torch.full((T, F), float("nan"), dtype=torch.bfloat16, device="cuda")
    delta = torch.empty(b, heads, s, device="cuda")
    K._ext().lorsa_dz(idx, act, dact, dz, delta)
    want, z = torch.zeros(T, F + 1, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, F + 1, device="cuda")
    at = torch.where(idx >= 0, idx, F).long()
    want.scatter_(1, at, dact.to(torch.bfloat16))
    z.scatter_(1, at, act)
    assert torch.equal(dz, want[:, :F])
    prod = (want[:, :F].double() * z[:, :F].double()).view(b, s, heads, group)
    bound = (k + 1) * 2.0**-24 * prod.abs().sum(-1).permute(0, 2, 1)
    assert bool(((delta.double() - prod.sum(-1).permute(0, 2, 1)).abs() <= bound).all())
    assert not K._ext().lorsa_dz_fits(200 * 1024, 8) and not K._ext().lorsa_dz_fits(12, 2) and K._ext().lorsa_dz_fits(8192, 128)
