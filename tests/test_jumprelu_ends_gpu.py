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
    # the last bit of a threshold decides which values pass it: torch's, to the bit (which is up to 2 units in the last place from the exponential)
    assert torch.equal(theta.nan_to_num(nan=-1.0), log_theta.exp().nan_to_num(nan=-1.0))
    assert torch.equal(t_min.nan_to_num(nan=-1.0), (theta / norm).amin(0).nan_to_num(nan=-1.0))
    assert torch.equal(total, bias.sum(0))
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


@pytest.mark.parametrize("B,heads,d,F,cap,shift", [(256, 1, 64, 2048, 64, 2.0), (300, 2, 64, 4104, 64, 2.0), (37, 3, 128, 1000, 1024, 0.0), (512, 1, 192, 18432, 256, 2.6), (129, 1, 64, 264, 8, 1.0)])
def test_lists_by_maxima_are_those_of_the_whole_matrix(B, heads, d, F, cap, shift):
    """Bit for bit, with thresholds that values equal, of nothing, everything, no number, and beyond the range of their reciprocals; with NaNs and infinities
    in the values, and rows that hold more than the list."""
    g = torch.Generator(device=DEV).manual_seed(F)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    x, w, bias = r(B, heads * d).to(torch.bfloat16), (r(heads * F, d) / (heads * d) ** 0.5).to(torch.bfloat16), 0.1 * r(F)
    log_theta, norm = shift + 0.2 * r(F) - 1.5 * (torch.rand(F, device=DEV, generator=g) < 0.02), torch.ones(heads, F, device=DEV)
    log_theta[3:9] = torch.tensor([float("-inf"), float("inf"), float("nan"), -90.0, 87.5, -100.0], device=DEV)
    norm[0, 40], norm[0, 41], norm[0, 42] = -1.0, 0.0, float("inf")
    bias[100], bias[101], bias[3], bias[4] = 3e38, float("nan"), -1e-39, float("inf")
    gate = torch.empty(F, device=DEV)
    theta, t_min, *_ = K._ext().jumprelu_begin(log_theta, norm, None, gate)
    H, maxima = torch.empty(B, F, dtype=torch.bfloat16, device=DEV), torch.full((B, -(-F // 256) * 8), float("nan"), device=DEV)
    K._ext().head_sum_gemm(x, w, bias, heads, F, F, True, K.status_buffer(torch.device(DEV)), H, maxima, gate)
    K.check_status(torch.device(DEV))
    t_min[200:232] = H[0, 200:232].float().abs()  # (equal is not above; the gates of these are not their reciprocals, but the rows' are looked at below)
    gate[200:232] = 1.0 / t_min[200:232]
    K._ext().head_sum_gemm(x, w, bias, heads, F, F, True, K.status_buffer(torch.device(DEV)), H, maxima, gate)
    plain = H.clone()
    K._ext().head_sum_gemm(x, w, bias, heads, F, F, True, K.status_buffer(torch.device(DEV)), H)
    assert torch.equal(plain.view(torch.int16), H.view(torch.int16))
    got = []
    for m in (None, maxima):
        idx, val, over = torch.empty(B, cap, dtype=torch.int32, device=DEV), torch.empty(B, cap, device=DEV), torch.zeros((), dtype=torch.int64, device=DEV)
        assert K._ext().column_lists(H, t_min, idx, val, over, m)
        got.append((idx, val, over))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert torch.equal(got[1][0][0, : min(cap, int((H[0].float() > t_min).sum()))], torch.nonzero(H[0].float() > t_min).flatten()[:cap].int())


@pytest.mark.parametrize("share", [0.01, 0.05, 0.4])
def test_rows_with_far_more_values_than_places_cost_no_more_by_maxima(share):
    """A dictionary before its thresholds have closed: one warp looked at all of a row's groups, 455 us against 335 from the whole matrix at 0.4."""
    B, F, cap, best = 4096, 98304, 256, [1e9, 1e9]
    x = torch.rand(B, F, device=DEV, generator=torch.Generator(device=DEV).manual_seed(0)).to(torch.bfloat16)
    thr = torch.full((F,), 1 - share, device=DEV)
    maxima = (x.view(B, F // 32, 32).amax(2).float() / (1 - share)).contiguous()
    idx, val = (torch.empty(B, cap, dtype=t, device=DEV) for t in (torch.int32, torch.float32))
    for _ in range(6):
        for i, m in enumerate((maxima, None)):
            over = torch.zeros((), dtype=torch.int64, device=DEV)
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda._sleep(100000)
            start.record()
            assert K._ext().column_lists(x, thr, idx, val, over, m)
            end.record()
            end.synchronize()
            best[i] = min(best[i], start.elapsed_time(end))
            assert int(over) == B
    assert best[0] < best[1], best
