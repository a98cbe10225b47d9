"""Arguments that are pieces of longer tensors and start anywhere, not at a 16-byte boundary: the same results as from copies."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _piece(t: torch.Tensor, off: int) -> torch.Tensor:
    flat = torch.zeros(t.numel() + 8, dtype=t.dtype, device=t.device)
    view = flat[off : off + t.numel()].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("d", [64, 1160])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_decoder_bias(d, off):
    g = torch.Generator(device=DEV).manual_seed(d)
    B, F, k = 37, 300, 9
    idx = torch.randint(0, F, (B, k), device=DEV, dtype=torch.int32, generator=g)
    val, W = torch.rand(B, k, device=DEV, generator=g), torch.randn(F, d, device=DEV, generator=g).to(torch.bfloat16)
    bias, label = torch.randn(d, device=DEV, generator=g), torch.randn(B, d, device=DEV, generator=g).to(torch.bfloat16)
    assert torch.equal(K.sparse_decode(idx, val, W, _piece(bias, off)), K.sparse_decode(idx, val, W, bias))
    out = []
    for b in (bias, _piece(bias, off)):
        loss = torch.zeros(1, device=DEV)
        out.append(K.sparse_decode_loss(idx, val, W, b, label, None, 0.1, loss))
    for a, b in zip(*out):
        assert (a is None and b is None) or torch.equal(a, b)


@pytest.mark.parametrize("k", [8, 50])
@pytest.mark.parametrize("off", [1, 2])
def test_resumed_candidate_lists(k, off):
    g = torch.Generator(device=DEV).manual_seed(k)
    M, N, d = 200, 1040, 64
    x, w = (torch.randn(n, d, device=DEV, generator=g).to(torch.bfloat16) for n in (M, N))
    lo, hi = w[:512].contiguous(), w[512:].contiguous()
    out = []
    for place in (lambda t: t, lambda t: _piece(t, off)):
        val, idx, C = K.encoder_topk_candidates(x, lo, None, None, k, num_splits=1)
        val, idx = place(val), place(idx)
        val, idx, C = K.encoder_topk_candidates(x, hi, None, None, k, num_splits=1, n_index_offset=512, resume=(val, idx))
        i, v = K.topk_merge(val, idx, k, None)
        order = i.sort(dim=1).indices
        out.append((i.gather(1, order), v.gather(1, order)))
    K.check_status(torch.device(DEV))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
