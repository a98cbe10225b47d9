"""The small kernels at both ends of a JumpReLU step against torch operations."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K, select_kernels as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,F", [(1, 8), (1, 1000), (3, 257), (8, 4096)])
def test_thresholds_and_bias_sum(H, F):
    g = torch.Generator(device=DEV).manual_seed(F)
    log_theta, norm, bias = torch.randn(F, device=DEV, generator=g) * 3, torch.rand(H, F, device=DEV, generator=g) + 0.1, torch.randn(H, F, device=DEV, generator=g)
    norm[0, 1], norm[H - 1, 2], log_theta[3] = 0.0, float("nan"), float("nan")
    theta, t_min, total = K._ext().jumprelu_begin(log_theta, norm, bias)
    want = log_theta.double().exp()
    assert torch.allclose(theta.double(), want, rtol=2.0**-23, atol=0.0, equal_nan=True)
    assert torch.equal(t_min.nan_to_num(nan=-1.0), (theta / norm).amin(0).nan_to_num(nan=-1.0))
    assert torch.allclose(total, bias.sum(0), atol=2.0**-23 * H * 4)
    assert len(K._ext().jumprelu_begin(log_theta, norm, None)) == 2


@pytest.mark.parametrize("F,with_lp", [(8, False), (1000, True)])
def test_end_of_a_step(F, with_lp):
    g = torch.Generator(device=DEV).manual_seed(F)
    r = lambda: torch.randn(F, device=DEV, generator=g)  # noqa: E731
    p, m, v, dtheta, theta = r(), r() * 0.1, r().square() * 0.01, r(), r().exp()
    want = [t.clone() for t in (p, m, v)]
    l_rec, u, l_p = (torch.rand((), device=DEV, generator=g) for _ in range(3))
    n = torch.tensor([1234], dtype=torch.int32, device=DEV)
    out = K._ext().jumprelu_end(p, m, v, dtheta, theta, l_rec, u.reshape(1), l_p if with_lp else None, n, 1e-3, 96.0, 32.0, 1e-3, 0.9, 0.999, 1e-8, 3, K.status_buffer(torch.device(DEV)))
    K.adam_flat(want[0], dtheta * theta, want[1], want[2], 1e-3, 0.9, 0.999, 1e-8, 3)
    for a, b in zip((p, m, v), want):
        assert torch.allclose(a, b, rtol=2.0**-20, atol=4e-9)  # (a product that is rounded, or part of a fused one: 2^-20 of a step, lr / (1 - 0.9^3) at most)
    l_s, lp = 1e-3 * u / 96.0, l_p if with_lp else torch.zeros((), device=DEV)
    assert torch.allclose(out, torch.stack([l_rec + l_s + lp, l_s, lp, n[0] / 32.0]), rtol=1e-6)


@pytest.mark.parametrize("B,N,cap", [(5, 800, 8), (700, 1000, 16), (1300, 264, 8), (9, 1001, 8)])
def test_rows_beyond_the_lists_width_are_counted(B, N, cap):
    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(B, N, device=DEV, generator=g).to(torch.bfloat16)
    thr = torch.rand(N, device=DEV, generator=g) + 1.8
    n = torch.full((1,), 5, dtype=torch.int64, device=DEV)
    idx, val = S.column_threshold_rows_to_sparse(x, thr, cap, overflow=n)
    cpu = torch.full((1,), 5, dtype=torch.int64)
    want_idx, want_val = S.column_threshold_rows_to_sparse(x.cpu(), thr.cpu(), cap, overflow=cpu)
    assert torch.equal(idx.cpu(), want_idx) and torch.equal(val.cpu(), want_val) and int(n) == int(cpu) > 5


@pytest.mark.parametrize("with_status", [False, True])
def test_loss_and_status_reach_the_host(with_status):
    from language_model_saes_b200.trainer import _LossReader

    status = torch.tensor([0, 7, 8, 9], dtype=torch.int32, device=DEV) if with_status else None
    reader, seen = _LossReader(), []
    for i in range(7):
        seen.append(reader.push(torch.full((), 0.1 + i, device=DEV), status))
    assert seen[0] is None and all(abs(s - (0.1 + i)) < 1e-6 for i, s in enumerate(seen[1:]))
    assert abs(reader.flush() - 6.1) < 1e-6
    host = torch.empty(5, pin_memory=True)
    assert K._ext().read_back(torch.ones(1, device=DEV), torch.arange(4, dtype=torch.int32, device=DEV), host)
    torch.cuda.synchronize()
    assert host.tolist() == [1.0, 0.0, 1.0, 2.0, 3.0]
    assert not K._ext().read_back(torch.ones(1, device=DEV, dtype=torch.float64), None, host) and not K._ext().read_back(torch.ones(1, device=DEV), None, torch.empty(5))
    bad = torch.tensor([5, 1, 2, 3], dtype=torch.int32, device=DEV)
    with pytest.raises(K.CollectiveTimeout):
        reader.push(torch.ones((), device=DEV), bad)
        reader.flush()
