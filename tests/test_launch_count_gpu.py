"""The counter of launches against the kernels that a profiler sees."""

import pytest
import torch

from language_model_saes_b200.ops import inference as I
from language_model_saes_b200.ops import sae_kernels as K
from language_model_saes_b200.ops import select_kernels as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _encode(pieces):
    x, w = torch.randn(300, 128, device=DEV), torch.randn(4096, 128, device=DEV)

    def run():
        workspace, I.PRODUCT_WORKSPACE = I.PRODUCT_WORKSPACE, 1 if pieces else I.PRODUCT_WORKSPACE
        try:
            I.topk_encode(x, w.t(), None, None, 20)
        finally:
            I.PRODUCT_WORKSPACE = workspace

    return run


def _lists():
    x, w = torch.randn(256, 64, device=DEV).to(torch.bfloat16), torch.randn(4096, 64, device=DEV).to(torch.bfloat16)
    thr, n = torch.ones(1, device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV)
    H, maxima = K.encoder_hidden_maxima(x, w, None)
    return lambda: S.threshold_rows_to_sparse(H, thr, None, n_ties=n, cap=64, maxima=maxima)


def _dead():
    from language_model_saes_b200.ops.fused_step import AuxK

    F = 4096
    aux = AuxK(F, 64, 1 / 32, 10.0, DEV)
    W = torch.randn(F, 64, device=DEV).to(torch.bfloat16)
    fired, n, b = torch.zeros(F, dtype=torch.int32, device=DEV), torch.full((), 7, device=DEV), torch.zeros(F, device=DEV)
    return lambda: aux.compact(fired, n, 512, W, W, b, None)


def _groups(n, F):
    groups = K.FeatureGroups(F, n, torch.device(DEV))
    idx = torch.randint(0, F, (n,), dtype=torch.int32, device=DEV)
    return lambda: groups.build(idx)


CASES = {"encode": lambda: _encode(False), "encode in pieces": lambda: _encode(True), "lists": _lists, "dead rows": _dead,
         "few entries": lambda: _groups(1000, 256), "many entries": lambda: _groups(60000, 256), "long dictionary": lambda: _groups(60000, 200000)}  # fmt: skip


@pytest.mark.parametrize("name", CASES)
def test_launches_are_those_of_the_profiler(name):
    run = CASES[name]()
    run()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        before = K.kernel_launch_count()
        run()
        counted = K.kernel_launch_count() - before
        torch.cuda.synchronize()
    seen = [e.name for e in prof.events() if "lmsae::" in e.name]
    assert counted == len(seen) > 0, seen
