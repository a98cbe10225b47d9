"""Selections that look at the maxima of 32 columns first, against the ones that read the whole matrix."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K
from language_model_saes_b200.ops import select_kernels as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one group; a group and a bit; a whole tile and eight columns more (rows for the single and the paired kernel); many tiles
@pytest.mark.parametrize("M,N", [(1, 8), (130, 40), (256, 264), (300, 4096 + 24), (512, 9000)])
@pytest.mark.parametrize("gated", ["stored", "max", "none"])
def test_maxima_of_stored_pre_activations(M, N, gated):
    g = torch.Generator(device=DEV).manual_seed(N)
    x, w = torch.randn(M, 64, device=DEV, generator=g).to(torch.bfloat16), torch.randn(N, 64, device=DEV, generator=g).to(torch.bfloat16)
    b, gate = torch.randn(N, device=DEV, generator=g), torch.rand(N, device=DEV, generator=g) + 0.5
    b[N // 2] = float("nan")
    H, maxima = K.encoder_hidden_maxima(x, w, b, gate=gate if gated == "stored" else None, max_gate=gate if gated == "max" else None)
    K.check_status(torch.device(DEV))
    assert torch.equal(H.nan_to_num(nan=7.0), K.encoder_hidden(x, w, b, gate=gate if gated == "stored" else None).nan_to_num(nan=7.0))
    v = H.float() * gate if gated == "max" else H.float()
    groups = -(-N // 32)
    pad = torch.zeros(M, groups * 32 - N, device=DEV)  # (columns past the end inside a group count as zero)
    want = torch.cat([v, pad], 1).view(M, groups, 32).amax(2)
    assert torch.equal(maxima[:, :groups].nan_to_num(nan=7.0), want.nan_to_num(nan=7.0))
    assert bool((maxima[:, groups:] <= 0).all())


@pytest.mark.parametrize("M,N,k", [(3, 8200, 64), (40, 16384 + 40, 100), (9, 32768, 256)])
@pytest.mark.parametrize("data", ["normal", "few positive", "ties", "nan"])
def test_row_topk_with_maxima(M, N, k, data):
    g = torch.Generator(device=DEV).manual_seed(N)
    H = torch.randn(M, N, device=DEV, generator=g).to(torch.bfloat16)
    gate = torch.rand(N, device=DEV, generator=g) + 0.5
    if data == "few positive":
        H = (H - 3.3).to(torch.bfloat16)
    elif data == "ties":
        H, gate = (H * 2).round().to(torch.bfloat16), torch.ones(N, device=DEV)
    elif data == "nan":
        H[0, 5], H[1, 100:140] = float("nan"), float("nan")
    groups = -(-N // 256) * 8
    gated = torch.zeros(M, groups * 32, device=DEV)
    gated[:, :N] = H.float() * gate
    maxima = gated.view(M, groups, 32).amax(2).contiguous()
    idx, val = K.row_topk(H, k, gate, maxima=maxima)
    want_idx, want_val = K.row_topk(H, k, gate)
    order, want_order = idx.sort(1), want_idx.sort(1)
    if data != "ties":  # (which of equal values are taken is free)
        assert torch.equal(order.values, want_order.values)
        assert torch.equal(val.gather(1, order.indices), want_val.gather(1, want_order.indices))
    assert torch.equal((val * (idx >= 0)).sort(1).values, (want_val * (want_idx >= 0)).sort(1).values)


@pytest.mark.parametrize("B,N,k", [(1, 8, 1), (5, 40, 3), (70, 4104, 16), (300, 9000, 64)])
@pytest.mark.parametrize("data", ["normal", "ties", "few positive", "huge", "nan"])
def test_batch_level_selection_with_maxima(B, N, k, data):
    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(B, N, device=DEV, generator=g)
    if data == "ties":
        x = (x * 2).round() / 2
    elif data == "few positive":
        x -= 3.5
    elif data == "huge":
        x[0, 0], x[-1, -1] = 3e38, float("inf")
    elif data == "nan":
        x[0, N // 3] = float("nan")
    x = x.to(torch.bfloat16)
    groups = -(-N // 256) * 8
    padded = torch.zeros(B, groups * 32, dtype=torch.bfloat16, device=DEV)
    padded[:, :N] = x
    maxima = padded.view(B, groups, 32).float().amax(2).contiguous()
    thr, n_ties = S.positive_thresholds(x.view(1, 1, -1), k * B, None, return_remaining=True)
    for floor in (0.75 * thr, 2 * thr, torch.full_like(thr, 1e-3)):  # (the second one is too high: the pass is repeated)
        got, got_ties = S.positive_thresholds(x.view(1, 1, -1), k * B, None, return_remaining=True, floor=floor, maxima=maxima)
        assert torch.equal(got, thr) and torch.equal(got_ties, n_ties)
    div = torch.rand(N, device=DEV, generator=g) + 0.5
    for cap in (8, 8 * k):
        counts = [torch.zeros(1, dtype=torch.int64, device=DEV) for _ in range(2)]
        want = S.threshold_rows_to_sparse(x, thr, div, n_ties=n_ties, cap=cap, overflow=counts[0])
        got = S.threshold_rows_to_sparse(x, thr, div, n_ties=n_ties, cap=cap, overflow=counts[1], maxima=maxima)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1].nan_to_num(nan=7.0), want[1].nan_to_num(nan=7.0)) and torch.equal(*counts)


# on both sides of the lines of both rules
@pytest.mark.parametrize("B,N,k", [(512, 65536, 64), (1024, 16384, 64), (1024, 65536, 16), (4096, 8192, 128), (4096, 32768, 64), (8192, 16384, 32)])
def test_maxima_are_used_where_they_pay(B, N, k):
    g = torch.Generator(device=DEV).manual_seed(0)
    x, w = torch.randn(B, 64, device=DEV, generator=g).to(torch.bfloat16), torch.randn(N, 64, device=DEV, generator=g).to(torch.bfloat16)
    H, maxima = K.encoder_hidden_maxima(x, w, None)
    thr, n_ties = S.positive_thresholds(H.view(1, 1, -1), k * B, None, return_remaining=True)
    overflow = torch.zeros(1, dtype=torch.int64, device=DEV)

    def threshold(by_maxima):
        return S.positive_thresholds(H.view(1, 1, -1), k * B, None, return_remaining=True, floor=thr * (0.9 if by_maxima else 0.75), maxima=maxima if by_maxima else None)

    def lists(by_maxima):
        return S.threshold_rows_to_sparse(H, thr, None, n_ties=n_ties, cap=8 * k, overflow=overflow, maxima=maxima if by_maxima else None)

    def best(fn, by_maxima):
        times = []
        for _ in range(8):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda._sleep(200000)  # (so that the launches wait for the GPU and not the other way round)
            start.record()
            fn(by_maxima)
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)

    for fn, rule in ((threshold, S.maxima_pay_for_threshold), (lists, S.maxima_pay_for_lists)):
        taken = rule(B, N, k)
        assert best(fn, taken) < 1.3 * best(fn, not taken), (fn.__name__, taken)


@pytest.mark.parametrize("B,N", [(1, 33), (9, 4100), (5000, 1000), (33, 4133)])
@pytest.mark.parametrize("data", ["normal", "all equal", "one step", "nan"])
def test_lists_in_one_pass_with_quotas_afterwards(B, N, data):
    """Rows that are not whole vectors, more rows than a turn of the quotas takes, rows of equal values that overflow the list before the quota is taken
    out, and quotas that end within a row, at a row's end, at none and at all of them."""
    g = torch.Generator(device=DEV).manual_seed(B)
    x = torch.randn(B, N, device=DEV, generator=g)
    x = (torch.ones_like(x) if data == "all equal" else (x > 1).float() + 1 if data == "one step" else x).to(torch.bfloat16)
    if data == "nan":
        x[B // 2, N // 2] = float("nan")
    groups = -(-N // 256) * 8
    padded = torch.zeros(B, groups * 32, dtype=torch.bfloat16, device=DEV)
    padded[:, :N] = x
    maxima = padded.view(B, groups, 32).float().amax(2).contiguous()
    thr = x.float().nan_to_num(nan=0.0).flatten().topk(max(1, B * N // 50)).values[-1].reshape(1)
    ties = int((x.float() == thr).sum())
    for n_ties in {0, 1, ties // 2, int((x[0].float() == thr).sum()), ties}:
        want_n, got_n = (torch.zeros(1, dtype=torch.int64, device=DEV) for _ in range(2))
        n = torch.tensor([n_ties], device=DEV)
        want = S.threshold_rows_to_sparse(x, thr, None, n_ties=n, cap=24, overflow=want_n)
        got = S.threshold_rows_to_sparse(x, thr, None, n_ties=n, cap=24, overflow=got_n, maxima=maxima)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1].nan_to_num(nan=7.0), want[1].nan_to_num(nan=7.0)) and torch.equal(got_n, want_n), n_ties


def test_quotas_of_more_equal_values_than_31_bits_count():
    """4096 rows of 600000 values equal to the threshold are 2.5e9: the places go to the first row, and to no other."""
    B, N, places = 4096, 600000, 300000
    x = torch.ones(B, N, dtype=torch.bfloat16, device=DEV)
    maxima = torch.ones(B, N // 32, device=DEV)
    nnz, idx = torch.empty(B, dtype=torch.int32, device=DEV), torch.empty(B, 8, dtype=torch.int32, device=DEV)
    over = torch.zeros(1, dtype=torch.int64, device=DEV)
    K._ext().chunk_lists(x, maxima, torch.ones(1, device=DEV), torch.tensor([places], device=DEV), None, nnz, idx, torch.empty(B, 8, device=DEV), over)
    assert int(nnz[0]) == places and not nnz[1:].any() and int(over) == 1
    assert torch.equal(idx[0].cpu(), torch.arange(8, dtype=torch.int32)) and bool((idx[1:] == -1).all())


@pytest.mark.parametrize("M,N,k", [(1, 8, 3), (5, 2048, 512), (300, 4104, 100), (40, 9216, 512), (3, 3000, 1500)])
@pytest.mark.parametrize("data", ["normal", "few positive", "ties", "no gate"])
def test_row_topk_as_a_matrix(M, N, k, data):
    g = torch.Generator(device=DEV).manual_seed(N)
    H = torch.randn(M, N, device=DEV, generator=g).to(torch.bfloat16)
    gate = None if data == "no gate" else torch.rand(N, device=DEV, generator=g) + 0.5
    if gate is not None:
        gate[:: 3] = 0.0
    if data == "few positive":
        H = (H - 3.0).to(torch.bfloat16)
    elif data == "ties":
        H = (H > 0.5).to(torch.bfloat16)
        gate = torch.ones_like(gate)
    out = K.row_topk_dense(H, k, gate)
    idx, act = K.row_topk(H, k, gate)
    want = torch.zeros(M, N + 1, device=DEV).scatter_(1, torch.where(idx >= 0, idx, torch.full_like(idx, N)).long(), act)[:, :N].to(torch.bfloat16)
    if data == "ties" or gate is None:  # (which of equal values are taken is free)
        out, want = out.sort(1).values, want.sort(1).values
    assert torch.equal(out, want)


@pytest.mark.parametrize("counter", [None, "one", "two", "32 bits"])
@pytest.mark.parametrize("where", ["cpu", DEV])
def test_lists_take_the_numbers_as_they_come(counter, where):
    """The number of equal values from the host, counters of other shapes and types: as without maxima."""
    x = torch.randint(0, 4, (40, 512), device=DEV, generator=torch.Generator(device=DEV).manual_seed(0)).to(torch.bfloat16)
    maxima = x.float().view(40, 16, 32).amax(2).contiguous()
    new = {"one": lambda: torch.zeros(1, dtype=torch.int64, device=DEV), "two": lambda: torch.zeros(2, dtype=torch.int64, device=DEV),
           "32 bits": lambda: torch.zeros((), dtype=torch.int32, device=DEV), None: lambda: None}[counter]  # fmt: skip
    thr, n_ties = torch.full((1,), 2.0, device=DEV), torch.tensor(1000, device=where)
    outs = []
    for m in (None, maxima):
        over = new()
        outs.append((*S.threshold_rows_to_sparse(x, thr, None, n_ties=n_ties, cap=136, overflow=over, maxima=m), *([over] if counter else [])))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
