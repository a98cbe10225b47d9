"""Row top-k of stored pre-activations, a warp per row, against a stable sort; and the route that stores them against the GEMM's epilogue."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one group; a CTA and a row; the most groups with one maximum per register (16384 columns) and eight columns more; three per register
@pytest.mark.parametrize("M,N,k", [(1, 8, 1), (9, 264, 64), (4, 4104, 32), (8, 16384, 128), (17, 16392, 128), (5, 40000, 100)])
@pytest.mark.parametrize("data", ["normal", "few positive", "ties", "equal", "nan", "inf"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gated", [False, True])
def test_row_select(M, N, k, data, dtype, gated):
    g = torch.Generator().manual_seed(N + k)
    H = torch.randn(M, N, generator=g)
    gate = torch.rand(N, generator=g) + 0.5 if gated else None
    if data == "few positive":
        H -= 3.3
    elif data == "ties":
        H, gate = (H * 2).round(), torch.ones(N) if gated else None
    elif data == "equal":  # (more candidates than there is room for)
        H, gate = torch.where(torch.rand(M, N, generator=g) < 0.9, 1.5, H * 0.5), torch.ones(N) if gated else None
    elif data == "nan":
        H[:, N // 2], H[-1] = float("nan"), float("nan")
    elif data == "inf":
        H[0, 3], H[-1, :5] = float("inf"), -float("inf")
    H = H.to(dtype)
    v = H.float() * gate if gated else H.float()
    maxima = torch.zeros(M, -(-N // 256) * 256)
    maxima[:, :N] = v
    maxima = maxima.view(M, -1, 32).amax(2)
    key = torch.where(v > 0, v, torch.zeros(()))  # (NaN never enters)
    val, idx = key.sort(dim=1, descending=True, stable=True)
    val, idx = val[:, :k], torch.where(val[:, :k] > 0, idx[:, :k], -1)
    dev = [None if t is None else t.to(DEV) for t in (H, maxima, gate)]
    for sort in (True, False):
        got_idx, got_val = (t.cpu() for t in K.row_select(dev[0], dev[1], k, dev[2], sort=sort))
        if sort:
            assert torch.equal(got_idx, idx.int())
        assert torch.equal(got_idx.sort(1).values, idx.int().sort(1).values)
        got_key = torch.where(got_idx >= 0, got_val * (gate[got_idx.clamp_min(0).long()] if gated else 1.0), torch.zeros(()))
        finite = torch.isfinite(val)
        want = val if sort else val.sort(1, descending=True).values
        got = got_key if sort else got_key.sort(1, descending=True).values
        # a division by the gate and a product with it again: two roundings of 2^-24, the division to two units in the last place
        assert bool(((got - want).abs() <= 6 * 2.0**-24 * want)[finite].all())


# the line at 4096 columns; that of M * K; that of 4096 rows; rows and columns with remainders; a gate off its alignment
@pytest.mark.parametrize("M,N,d,k", [(1, 4088, 64, 1), (1, 4096, 64, 32), (3, 4104, 64, 7), (2048, 4096, 1024, 32), (2049, 4104, 1024, 32), (4096, 8200, 64, 64), (4097, 8192, 64, 8)])
@pytest.mark.parametrize("form", ["plain", "gate", "gate off by one", "no bias", "ties"])
def test_stored_route_is_the_epilogues(M, N, d, k, form):
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w = torch.randn(M, d, device=DEV, generator=g), torch.randn(N, d, device=DEV, generator=g)
    if form == "ties":
        x, w = x.round().clamp(-1, 1), w.round().clamp(-1, 1)
    x, w = x.to(torch.bfloat16), w.to(torch.bfloat16)
    bias = None if form in ("no bias", "ties") else torch.randn(N, device=DEV, generator=g)
    gate = torch.rand(N + 1, device=DEV, generator=g) + 0.5
    gate = gate[:N] if form == "gate" else gate[1:] if form == "gate off by one" else None
    idx, val = K.encoder_topk(x, w, bias, gate, k)
    cand_val, cand_idx, _ = K.encoder_topk_candidates(x, w, bias, gate, k)
    want_idx, want_val = K.topk_merge(cand_val, cand_idx, k, gate)
    K.check_status(torch.device(DEV))
    assert idx.dtype == want_idx.dtype and val.dtype == want_val.dtype
    assert torch.equal(val * (idx >= 0), want_val * (want_idx >= 0))
    assert torch.equal(idx, want_idx)


# the lines at 1024 rows and 128 codes, that of 128 columns a code (one group of eight more and less), the most codes the maxima serve
@pytest.mark.parametrize("M,N,k", [(1023, 8320, 65), (1024, 8320, 65), (1024, 8312, 65), (1025, 16384, 128), (1024, 16512, 129), (130, 65536, 512), (40, 65536 + 8, 513)])
@pytest.mark.parametrize("form", ["gate", "gate off by one", "none"])
def test_stored_hidden_and_its_codes(M, N, k, form):
    g = torch.Generator(device=DEV).manual_seed(N)
    x, w = torch.randn(M, 64, device=DEV, generator=g).to(torch.bfloat16), torch.randn(N, 64, device=DEV, generator=g).to(torch.bfloat16)
    bias, gate = torch.randn(N, device=DEV, generator=g), torch.rand(N + 1, device=DEV, generator=g) + 0.5
    gate = gate[:N] if form == "gate" else gate[1:] if form == "gate off by one" else None
    H, idx, val = K.hidden_topk(x, w, bias, gate, k)
    K.check_status(torch.device(DEV))
    assert torch.equal(H, K.encoder_hidden(x, w, bias))
    assert bool((idx >= 0).all()) and bool((idx.long().sort(1).values.diff(dim=1) > 0).all())
    gated = H.float() * gate if gate is not None else H.float()
    assert torch.equal(gated.gather(1, idx.long()).sort(1, descending=True).values, gated.topk(k, dim=1).values)
    got = H.float().gather(1, idx.long())
    # with a gate: a product with it and a division by it, three units in the last place together
    assert bool(((val - got).abs() <= (4 * 2.0**-24 if gate is not None else 0.0) * got.abs()).all())
