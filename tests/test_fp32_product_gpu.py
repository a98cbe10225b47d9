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
