"""fp32 products on the bf16 tensor cores at the edges of tiles, panels and slices, against 64 bits; values that bf16 parts cannot
hold; and no more error than the fp32 pipes where the dictionaries use them."""

import pytest
import torch

from language_model_saes_b200.ops import inference as I
from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K_", [(1, 8, 4), (130, 264, 68), (300, 1000, 128), (257, 513, 200), (513, 520, 1160)])
@pytest.mark.parametrize("special", [False, True])
def test_product(M, N, K_, special):
    g = torch.Generator().manual_seed(M + N)
    a, w = torch.randn(M, K_, generator=g), torch.randn(N, K_, generator=g) * 2.0 ** torch.randint(-40, 40, (N, 1), generator=g).float()
    if special:
        a[0, 1] = float("inf")
        a[M // 2, 2] = float("nan")
        w[N // 2, 3] = 3e38
    out = I.product(a.to(DEV), w.to(DEV).t()).cpu()
    K.check_status(torch.device(DEV))
    want = a.double() @ w.double().t()
    assert torch.equal(out.isnan(), want.isnan())
    fits = want.abs() < 3e38
    mass = a.double().abs() @ w.double().abs().t()
    # three parts hold 24 bits; slices are added up in fp32; within one, 96 accumulations of at most 2^-23 of the sum of magnitudes
    bound = 2.0**-24 * (K_ / 128 + 4) * mass + 2.0**-23 * 96 * mass / max(1.0, K_ / 128) + 1e-37
    assert ((out.double() - want).abs()[fits] <= bound[fits]).all()
    assert (out[~fits & ~want.isnan()].abs() > 2.9e38).all()


@pytest.mark.parametrize("K_", [64, 128, 256, 768, 2048])
@pytest.mark.parametrize("offset", [0.0, 1.0])
def test_no_more_error_than_the_fp32_pipes(K_, offset):
    g = torch.Generator(device=DEV).manual_seed(K_)
    a = torch.randn(512, K_, device=DEV, generator=g) + offset
    w = torch.randn(2048, K_, device=DEV, generator=g) / K_**0.5 + offset / K_
    want = a.double() @ w.double().t()
    ours = (I.product(a, w.t()).double() - want).abs()
    pipes = (a @ w.t()).double().sub(want).abs()
    top = want.topk(32, dim=1).indices  # (what a dictionary keeps)
    for pick in (lambda e: e, lambda e: e.gather(1, top)):
        e, f = pick(ours).square().mean().sqrt(), pick(pipes).square().mean().sqrt()
        print(K_, offset, "error", float(e), "fp32 pipes", float(f), "of", float(pick(want).square().mean().sqrt()))
        assert e <= f


@pytest.mark.parametrize("B,F,K_,k", [(3, 520, 68, 5), (300, 4104, 128, 50), (130, 24576, 256, 64), (40, 1000, 64, 700)])
@pytest.mark.parametrize("data", ["normal", "ties", "few", "special"])
def test_selection_is_that_of_sums_in_order(B, F, K_, k, data):
    g = torch.Generator(device=DEV).manual_seed(B + F)
    x, w = torch.randn(B, K_, device=DEV, generator=g), torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    bias, norm = 0.1 * torch.randn(F, device=DEV, generator=g), torch.rand(F, device=DEV, generator=g) + 0.5
    if data == "ties":  # features that differ in the last bits only: any other order of summation would choose others
        w[1::2] = w[::2] * (1 + 2.0**-23 * torch.randint(-2, 3, (F // 2, 1), device=DEV, generator=g))
        norm[1::2], bias[1::2] = norm[::2], bias[::2]
    elif data == "few":
        bias -= 4.0
    elif data == "special":
        x[0, 0], x[1, 1], norm[7] = float("inf"), float("nan"), 0.0
        w[5, 2] = 3e38
    out = I.topk_encode(x, w.t(), bias, norm, k)
    K.check_status(torch.device(DEV))
    h = torch.zeros(B, F, device=DEV, dtype=torch.float64)
    for i in range(K_):  # fp32 sums in order: a product of two fp32 numbers is exact in 64 bits, and so is rounding the sum to 32
        h = (h + x[:, i : i + 1].double() * w[:, i].double()).float().double()
    want = I.topk_dense(h.float(), bias, norm, k)
    if data == "special":  # half of row 0 is +inf: which of them are selected is free, the others become NaN
        assert out[0].isnan().sum() == want[0].isnan().sum() and out[0].isinf().sum() == want[0].isinf().sum()
        out[0] = want[0] = 0.0
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal((out != 0).sum(-1), (want != 0).sum(-1))
    if data == "ties":  # (equal sums: which of them is free)
        assert torch.equal((out * norm).sort(-1).values, (want * norm).sort(-1).values)
    else:
        assert torch.equal(out.nan_to_num(nan=-1.0), want.nan_to_num(nan=-1.0))


def _in_order(x, w):
    """fp32 sums in ascending order, one rounding per term: the sum in 64 bits is rounded to odd first (what it lost goes into its last
    bit), or one step in 2^29 would be rounded twice."""
    h = torch.zeros(x.shape[0], w.shape[0], device=DEV, dtype=torch.float64)
    for i in range(x.shape[1]):
        p = x[:, i : i + 1].double() * w[:, i].double()
        s = h + p
        b = s - h
        lost = (h - (s - b)) + (p - b)
        bits = s.view(torch.int64)
        odd = (bits - ((lost > 0) != (s > 0)).to(torch.int64)) | 1
        h = torch.where((lost != 0) & s.isfinite(), odd, bits).view(torch.float64).float().double()
    return h.float()


@pytest.mark.parametrize("data", ["cancelling", "near zero", "repeated", "out of range", "one bad column"])
@pytest.mark.parametrize("F,K_,k", [(4104, 128, 50), (9001, 260, 700)])
def test_selection_where_the_estimate_says_little(F, K_, k, data):
    g = torch.Generator(device=DEV).manual_seed(F)
    B = 270
    x, w = torch.randn(B, K_, device=DEV, generator=g), torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    bias, norm = 0.1 * torch.randn(F, device=DEV, generator=g), torch.rand(F, device=DEV, generator=g) + 0.5
    if data == "cancelling":  # a common offset that the bias takes away: what is left is a few units in the last place of the sums
        w *= 1e-3
        x[:, 0], w[:, 0] = 1000.0, 1.0
        bias = bias * 1e-3 - 1000.0
        norm[:] = 1.0
    elif data == "near zero":  # the k-th value is within rounding of zero
        bias = -_in_order(x[:1], w)[0].topk(k).values[-1].expand(F).clone()
        x[1:] = x[0] * (1 + 1e-6 * torch.randn(B - 1, 1, device=DEV, generator=g))
        norm[:] = 1.0
    elif data == "repeated":  # more equal features than there is room for, and fewer than that
        w[: F * 3 // 4] = w[0]
        bias[: F * 3 // 4], norm[: F * 3 // 4] = 1.0, 1.0
        x[B // 2 :] = x[0]
    elif data == "out of range":
        x[0] *= 1e-25
        x[1] *= 1e25
        x[2] = 0.0
        w[5] *= 1e-25
        w[7] *= 1e20
        w[9] = 0.0
    else:
        w[11, 3] = float("nan")
        w[13, 4] = float("inf")
    out = I.topk_encode(x, w.t(), bias, norm, k)
    want = I.topk_dense(_in_order(x, w), bias, norm, k)
    differ = (out.nan_to_num(nan=-1.0) != want.nan_to_num(nan=-1.0)).nonzero()
    assert differ.numel() == 0, (differ[:4], len(differ))


@pytest.mark.parametrize("F,k,equal", [(64, 5, 64), (3000, 7, 2400), (24576, 50, 24576), (30001, 1000, 9000)])
def test_of_equal_values_the_first_columns_are_kept(F, k, equal):
    g = torch.Generator().manual_seed(F)
    h = -torch.rand(3, F, generator=g)
    for r in range(3):
        h[r, torch.randperm(F, generator=g)[:equal]] = 0.75
    h[0, F // 2], h[1, F - 1] = 2.0, 3.0
    order = h.clamp_min(0.0).sort(dim=1, descending=True, stable=True).indices[:, :k]
    want = torch.zeros_like(h).scatter_(1, order, h.gather(1, order)).clamp_min(0.0)
    assert torch.equal(I.topk_dense(h.to(DEV), None, None, k).cpu(), want)


def test_rows_with_few_positive_values_cost_no_more_than_others():
    g = torch.Generator(device=DEV).manual_seed(0)
    x, w = torch.randn(1024, 512, device=DEV, generator=g), torch.randn(8192, 512, device=DEV, generator=g) / 512**0.5
    bias, times = torch.zeros(8192, device=DEV), []
    for shift in (0.0, -4.0):  # half of the features positive, hardly any
        for i in range(8):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            I.topk_encode(x, w.t(), bias + shift, None, 50)
            end.record()
            end.synchronize()
            if i == 0 or start.elapsed_time(end) < best:
                best = start.elapsed_time(end)
        times.append(best)
    assert times[1] < 3 * times[0], times  # (summed up as whole rows they took thirty times as long)


@pytest.mark.parametrize("share,factor", [(0.0, 1.0), (1 / 16384, 30.0), (1 / 16384, 1000.0), (0.01, 30.0), (0.01, 1000.0), (0.5, 10.0)])
def test_features_of_large_norm_do_not_widen_the_others_bounds(share, factor):
    """Codes bit for bit, and at most twice the time that a dictionary of equal norms takes (with one bound for all columns every row was
    multiplied in order as a whole: thirty times as long)."""
    g = torch.Generator(device=DEV).manual_seed(0)
    B, F, K_, k = 512, 16384, 4096, 50
    x = torch.randn(B, K_, device=DEV, generator=g)
    bias, norm = 0.02 * torch.randn(F, device=DEV, generator=g), torch.rand(F, device=DEV, generator=g) * 0.1 + 1.0
    even = torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    uneven = even.clone()
    uneven[torch.randperm(F, device=DEV, generator=g)[: int(share * F)]] *= factor
    best = [1e9, 1e9]
    for _ in range(6):
        for i, w in enumerate((even, uneven)):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            out = I.topk_encode(x, w.t(), bias, norm, k)
            end.record()
            end.synchronize()
            best[i] = min(best[i], start.elapsed_time(end))
    assert torch.equal(out[:64], I.topk_dense(_in_order(x[:64], uneven), bias, norm, k))
    assert best[1] < 2 * best[0], best


@pytest.mark.parametrize("B,F,K_,k", [(300, 1001, 128, 20), (257, 4104, 72, 64)])
def test_selection_where_the_product_gave_up(B, F, K_, k):
    g = torch.Generator(device=DEV).manual_seed(F)
    x, w = torch.randn(B, K_, device=DEV, generator=g), torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    bias, norm = 0.1 * torch.randn(F, device=DEV, generator=g), torch.rand(F, device=DEV, generator=g) + 0.5
    h, out = torch.randn(B, F, device=DEV, generator=g) * 100, torch.full((B, F), float("nan"), device=DEV)
    lo = h.view(-1).view(torch.bfloat16)[: B * F].view(B, F)  # what was there before
    xn, top = torch.full((B,), float("nan"), device=DEV), torch.zeros(4 + (F + 1) // 2, dtype=torch.int32, device=DEV)
    status, todo = torch.ones(4, dtype=torch.int32, device=DEV), torch.zeros(1 + B, dtype=torch.int32, device=DEV)
    K._ext().topk_estimate(lo, h, x, w, xn, top, bias, norm, k, status, todo, out)
    assert todo[0] == B and torch.equal(todo[1:].sort().values, torch.arange(B, dtype=torch.int32, device=DEV))
    assert torch.equal(out, I.topk_dense(_in_order(x, w), bias, norm, k))


def test_a_product_that_gave_up_is_made_good_and_stops_nothing_else(monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(0)
    x, w = torch.randn(300, 128, device=DEV, generator=g), torch.randn(1000, 128, device=DEV, generator=g)
    status = torch.ones(4, dtype=torch.int32, device=DEV)  # a wait ran out, and the tensor cores have written nothing
    out = torch.full((300, 1000), float("nan"), device=DEV)
    K._ext().fp32_gemm(x, w, out, status, None, None, None, None, False, 1 << 30)
    want, mass = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert ((out.double() - want).abs() <= 2.0**-24 * 128 * mass).all()

    def shared(device):
        raise AssertionError("the status word of the training kernels")

    monkeypatch.setattr(K, "status_buffer", shared)
    assert torch.isfinite(I.topk_encode(x, w.t(), None, None, 20)).all() and torch.isfinite(I.product(x, w.t())).all()


@pytest.mark.parametrize("M,N,K_", [(257, 1000, 200), (300, 513, 64)])
def test_a_dictionary_in_pieces(M, N, K_, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(N)
    x, w = torch.randn(M, K_, device=DEV, generator=g), torch.randn(N, K_, device=DEV, generator=g)
    w[N - 3, 1], w[2, 0] = 3e38, float("nan")
    bias, norm = torch.randn(N, device=DEV, generator=g), torch.rand(N, device=DEV, generator=g) + 0.5
    whole = I.product(x, w.t()), I.topk_encode(x, w.t(), bias, norm, 9)
    monkeypatch.setattr(I, "PRODUCT_WORKSPACE", 1)  # one tile at a time
    for a, b in zip(whole, (I.product(x, w.t()), I.topk_encode(x, w.t(), bias, norm, 9))):
        assert torch.equal(a.nan_to_num(nan=-1.0), b.nan_to_num(nan=-1.0))
    # the parts of W: 6 bytes an element of one tile instead of all
    monkeypatch.setattr(I, "PRODUCT_WORKSPACE", 1 << 20)
    w = torch.randn(65536, K_, device=DEV, generator=g)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = I.product(x, w.t())
    assert torch.cuda.max_memory_allocated() - before < out.numel() * 4 + x.numel() * 8 + (4 << 20)


@pytest.mark.parametrize("data", ["normal", "spread", "cancelling", "few cancelling rows", "near zero", "repeated", "out of range", "one bad column", "no gate"])
@pytest.mark.parametrize("B,F,K_,k", [(270, 8192, 128, 50), (259, 9001, 260, 64), (256, 33024, 68, 250)])
def test_selection_by_one_fp16_product(B, F, K_, k, data):
    """Codes bit for bit, wherever a row ends up: decided by the fp16 product, by the three products after it, or multiplied as a whole."""
    g = torch.Generator(device=DEV).manual_seed(F)
    assert I.half_product_pays(F, k)
    x, w = torch.randn(B, K_, device=DEV, generator=g), torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    bias, norm = 0.1 * torch.randn(F, device=DEV, generator=g), torch.rand(F, device=DEV, generator=g) + 0.5
    if data == "spread":  # magnitudes from the largest down to what fp16 drops, rows of very different size
        x *= torch.exp2(-24.0 * torch.rand(B, K_, device=DEV, generator=g)) * torch.exp2(20.0 * torch.rand(B, 1, device=DEV, generator=g))
        w *= torch.exp2(-24.0 * torch.rand(F, K_, device=DEV, generator=g)) * torch.exp2(6.0 * torch.rand(F, 1, device=DEV, generator=g) - 12.0)
        bias *= 0.0
    elif "cancelling" in data:  # a common offset that the bias takes away
        w *= 1e-3
        w[:, 0] = 1.0
        x[:, 0] = 1000.0
        if data != "cancelling":
            x[B // 10 :, 0] = 0.0
            x[B // 10 :] *= 1e6
        bias = bias * 1e-3 - 1000.0
        norm[:] = 1.0
    elif data == "near zero":
        bias = -_in_order(x[:1], w)[0].topk(k).values[-1].expand(F).clone()
        x[1:] = x[0] * (1 + 1e-6 * torch.randn(B - 1, 1, device=DEV, generator=g))
        norm[:] = 1.0
    elif data == "repeated":
        w[: F * 3 // 4] = w[0]
        bias[: F * 3 // 4], norm[: F * 3 // 4] = 1.0, 1.0
        x[B // 2 :] = x[0]
    elif data == "out of range":
        x[0] *= 1e-25
        x[1] *= 1e25
        x[2] = 0.0
        w[5] *= 1e-25
        w[7] *= 1e20
        w[9] = 0.0
        bias[11], norm[13], norm[15] = 1e25, 0.0, 1e20
    elif data == "one bad column":
        w[11, 3] = float("nan")
        w[13, 4] = float("inf")
        w[15, 2] = -float("inf")
    elif data == "no gate":
        norm = None
    out = I.topk_encode(x, w.t(), bias, norm, k)
    want = I.topk_dense(_in_order(x, w), bias, norm, k)
    differ = (out.nan_to_num(nan=-1.0) != want.nan_to_num(nan=-1.0)).nonzero()
    assert differ.numel() == 0, (differ[:4], len(differ))


def test_ends_of_one_fp16_product_enclose_the_sums():
    """What the selection relies on, without the selection: every positive sum in order lies between its end and that plus the width."""
    g = torch.Generator(device=DEV).manual_seed(0)
    B, F, K_, k = 512, 8192, 768, 64
    x, w = torch.randn(B, K_, device=DEV, generator=g), torch.randn(F, K_, device=DEV, generator=g) / K_**0.5
    exact = _in_order(x, w)
    half = lambda t: (lambda s: (t * s).half().double() / s.double())(torch.exp2(14 - t.abs().amax(1, keepdim=True).log2().floor()))  # noqa: E731
    error = (half(x) @ half(w).t() - exact.double()).abs()
    rest = lambda t: ((half(t) - t.double()).norm(dim=1) / t.double().norm(dim=1))  # noqa: E731
    bound = (rest(x)[:, None] + rest(w).max() + (2.1 * K_ + 136) * 2.0**-24) * x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)
    assert (error <= bound).all() and float((error / bound).max()) > 0.01  # (and says something)
    assert torch.equal(I.topk_encode(x, w.t(), None, None, k), I.topk_dense(exact, None, None, k))
