"""The encoder GEMM's top-k epilogue where its buffers change form: single CTAs and CTA pairs, both buffer sizes, ranges too wide
for 16-bit columns, sweeps resumed over chunks, rows with fewer than k positive values, rows of equal values. Inputs are small
integers, so that every product and sum is exact and the selected values have to be equal to plain torch's."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _data(M, N, Kd, kind, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randint(-2, 3, (M, Kd), generator=g).float()
    w = torch.randint(-2, 3, (N, Kd), generator=g).float()
    b = torch.randint(-8, 9, (N,), generator=g).float() / 4
    if kind == "few":
        b -= 3.0 * Kd**0.5 * 2
    elif kind == "equal":  # thousands of equal values, above a few others
        w[:] = w[:1]
        b[:] = 0.25
        b[::97] = 2.0
    elif kind == "rising":  # every column beats all before it: as many entries as there are columns
        w[:] = 0
        b = torch.arange(1, N + 1).float() / 64
    gate = 2.0 ** torch.randint(-1, 2, (N,), generator=g).float() if kind != "rising" else torch.ones(N)
    x[0] = 0.0
    return x.to(torch.bfloat16), w.to(torch.bfloat16), b, gate


def _check(idx, val, x, w, b, gate, k):
    idx, val = idx.cpu(), val.cpu()
    h = x.float() @ w.float().t() + b
    s = h * gate
    want = s.clamp_min(0).topk(min(k, s.shape[1]), dim=1).values
    keep = idx >= 0
    assert torch.equal(keep.sum(1), (want > 0).sum(1))
    safe = idx.clamp_min(0).long()
    got = torch.where(keep, s.gather(1, safe), torch.zeros(()))
    got = got.sort(dim=1, descending=True).values[:, : want.shape[1]]
    assert torch.equal(got, want)
    assert torch.equal(val, torch.where(keep, h.gather(1, safe), torch.zeros(())))  # (gates are powers of two: exact)
    dup = torch.where(keep, safe, -1 - torch.arange(idx.shape[1])).sort(dim=1).values
    assert (dup[:, 1:] != dup[:, :-1]).all()


@pytest.mark.parametrize("M,N,splits", [(1, 8, None), (130, 264, None), (257, 1000, 1), (300, 4104, None), (256, 66056, 1), (130, 8192, 3)])
@pytest.mark.parametrize("k", [1, 32, 33, 64])
@pytest.mark.parametrize("kind", ["normal", "few", "equal", "rising"])
def test_selected_values_are_exact(M, N, splits, k, kind):
    x, w, b, gate = _data(M, N, 72, kind, seed=N + k)
    xd, wd, bd, gd = x.to(DEV), w.to(DEV), b.to(DEV), gate.to(DEV)
    cv, ci, _ = K.encoder_topk_candidates(xd, wd, bd, gd, k, num_splits=splits)
    idx, val = K.topk_merge(cv, ci, k, gd)
    K.check_status(xd.device)
    _check(idx, val, x, w, b, gate, k)


# few rows are dealt to as many ranges as there are SMs: 98 x 64 candidates of four rows fit a CTA of the merge, 99 x 64 do not
@pytest.mark.parametrize("M,N", [(1, 98 * 256), (5, 99 * 256), (128, 148 * 256), (127, 150 * 256 + 40)])
@pytest.mark.parametrize("k", [32, 33, 64])
@pytest.mark.parametrize("kind", ["normal", "few", "equal"])
def test_few_rows_of_a_long_dictionary(M, N, k, kind):
    x, w, b, gate = _data(M, N, 72, kind, seed=N + k)
    idx, val, H = K.encoder_topk(x.to(DEV), w.to(DEV), b.to(DEV), gate.to(DEV), k, return_hidden=True)
    K.check_status(torch.device(DEV))
    _check(idx, val, x, w, b, gate, k)
    assert torch.equal(H.cpu(), (x.float() @ w.float().t() + b).to(torch.bfloat16))


@pytest.mark.parametrize("k", [20, 50, 64])
@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("kind", ["normal", "equal"])
def test_resumed_sweeps(k, compact, kind):
    M, N = 200, 3000
    x, w, b, gate = _data(M, N, 64, kind, seed=k)
    xd, wd, bd, gd = x.to(DEV), w.to(DEV), b.to(DEV), gate.to(DEV)
    state = None
    for lo, hi in ((0, 1024), (1024, 1536), (1536, N)):
        cv, ci, _ = K.encoder_topk_candidates(xd, wd[lo:hi], bd[lo:hi], gd[lo:hi], k, num_splits=2, n_index_offset=lo, resume=state, compact_smem=compact)
        state = (cv, ci)
    idx, val = K.topk_merge(cv, ci, k, gd)
    K.check_status(xd.device)
    _check(idx, val, x, w, b, gate, k)


@pytest.mark.parametrize("M,N", [(5, 8), (129, 264), (300, 1000)])
@pytest.mark.parametrize("gated", [False, True])
def test_stored_hidden_is_exact(M, N, gated):
    x, w, b, gate = _data(M, N, 72, "normal", seed=M)
    H = K.encoder_hidden(x.to(DEV), w.to(DEV), b.to(DEV), gate=gate.to(DEV) if gated else None)
    K.check_status(torch.device(DEV))
    want = (x.float() @ w.float().t() + b) * (gate if gated else 1.0)
    assert torch.equal(H.cpu(), want.to(torch.bfloat16))
