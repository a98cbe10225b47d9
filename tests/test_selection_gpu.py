"""Row top-k and per-column threshold selection where their kernels change path: rows shorter than one vector per thread,
unaligned rows, fewer positive values than asked for, values repeated more often than the candidate buffer holds, k beyond the
bound on group maxima, list widths that overflow within one warp's part; against plain torch on the CPU."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K
from language_model_saes_b200.ops import select_kernels as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,k", [(8, 3), (250, 128), (4099, 65), (8192, 1024), (8192, 1025), (65536, 128), (512, 600)])
@pytest.mark.parametrize("data", ["normal", "few", "repeated"])
@pytest.mark.parametrize("gated", [False, True])
def test_row_topk_paths(N, k, data, gated):
    M = 5
    g = torch.Generator().manual_seed(N + k)
    H = torch.randn(M, N, generator=g)
    if data == "few":
        H -= 3.0
    elif data == "repeated":
        H = H.sign() * 0.5
        H[:, ::7] = 1.5
    H[0] = -1.0  # a row without a positive value
    H = H.to(torch.bfloat16)
    gate = torch.rand(N, generator=g) + 0.5 if gated else None
    if gated and N == 4099:
        gate[::5] *= -2.0
    alive = (torch.rand(N, generator=g) > 0.3) if gated else None
    idx, val = K.row_topk(H.to(DEV), k, gate.to(DEV) if gated else None, alive.to(DEV) if gated else None)
    ref_idx, ref_val = K.ref_topk_codes(H.float(), k, gate, alive)
    idx, val = idx.cpu(), val.cpu()
    assert torch.equal((idx >= 0).sum(1), (ref_idx >= 0).sum(1))
    for b in range(M):
        got = idx[b][idx[b] >= 0].long()
        assert got.unique().numel() == got.numel()
        v = H[b].float()[got]
        # the stored value is (H * gate) / gate: two roundings (and the fast division's two units)
        assert torch.allclose(val[b][idx[b] >= 0], v, rtol=5 * 2**-23, atol=0)
        # which of several equal values is kept is free: the gated values kept are the same
        score = v * gate[got] if gated else v
        ref = ref_idx[b][ref_idx[b] >= 0].long()
        want = H[b].float()[ref] * (gate[ref] if gated else 1.0)
        assert torch.equal(score.sort().values, want.sort().values)
    assert (val[idx < 0] == 0).all()


@pytest.mark.parametrize("B,N,cap", [(3, 64, 8), (37, 2304, 256), (1184, 1000, 64), (1187, 4104, 256), (9, 4100, 512), (6, 520, 1032)])
@pytest.mark.parametrize("level", [1.0, -1.0])
def test_column_threshold_lists(B, N, cap, level):
    g = torch.Generator().manual_seed(B + N)
    x = torch.randn(B, N, generator=g).to(torch.bfloat16)
    thr = level + 0.1 * torch.randn(N, generator=g)
    thr[::3] = x[B // 2, ::3].float()  # equal to the threshold: not above it
    x[1, 5] = float("inf")
    x[2, 6] = float("nan")
    over, ref_over = torch.zeros(1, dtype=torch.int64, device=DEV), torch.zeros(1, dtype=torch.int64)
    idx, val = S.column_threshold_rows_to_sparse(x.to(DEV), thr.to(DEV), cap, overflow=over)
    ref_idx, ref_val = S.column_threshold_rows_to_sparse(x, thr, cap, overflow=ref_over)
    assert torch.equal(idx.cpu(), ref_idx) and torch.equal(val.cpu(), ref_val) and int(over) == int(ref_over)


# bins per thread from one to 64, in whole vectors and not; numbers of bins that are no whole vectors although a thread's share is; a histogram at an odd address
@pytest.mark.parametrize("nbins", [1, 7, 1024, 3072, 4095, 32640, 32641, 32642, 32643, 32767, 65535, 65536])
@pytest.mark.parametrize("shift", [0, 1])
def test_picked_bin(nbins, shift):
    g = torch.Generator().manual_seed(nbins)
    hist = torch.randint(0, 5, (nbins,), generator=g, dtype=torch.int32) * (torch.rand(nbins, generator=g) < 0.3).int()
    hist[0] += 1
    from_top = hist.flip(0).long().cumsum(0)
    total = int(from_top[-1])
    dev = torch.zeros(nbins + 1, dtype=torch.int32, device=DEV)[shift : shift + nbins].copy_(hist)
    for k in {1, total // 3 + 1, total, total + 1}:
        out = torch.zeros(4, dtype=torch.int64, device=DEV)
        K._ext().radix_pick(dev, nbins, k, None, 0, out, None, None)
        i = int(torch.searchsorted(from_top, k))
        want = [nbins - 1 - i, k - int(from_top[i - 1] if i else 0), total, 0] if k <= total else [0, 0, total, 1]
        assert out.tolist() == want, k
