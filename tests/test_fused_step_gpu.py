"""The fused kernel training step against the same step written with autograd + torch.optim.Adam."""

import copy

import pytest
import torch

from language_model_saes_b200.models.sae import SAEConfig, SparseAutoEncoder
from language_model_saes_b200.ops import sae_kernels as K
from language_model_saes_b200.ops.fused_step import FusedTopKSAEStep

pytestmark = pytest.mark.gpu


def _model(d=256, expansion=8, k=16, gate=True, bias=True):
    torch.manual_seed(0)
    cfg = SAEConfig(hook_point_in="h", hook_point_out="h", d_model=d, expansion_factor=expansion, act_fn="topk", top_k=k,
                    sparsity_include_decoder_norm=gate, use_decoder_bias=bias, device="cuda", dtype=torch.float32)  # fmt: skip
    sae = SparseAutoEncoder(cfg)
    sae.init_parameters(encoder_uniform_bound=0.06, decoder_uniform_bound=0.06)
    sae.set_decoder_to_fixed_norm(0.7, True)
    sae.init_encoder_with_decoder_transpose()
    sae.set_dataset_average_activation_norm({"h": d**0.5})
    return sae


def _data(n, B, d, rank=32):
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(rank, d, device="cuda", generator=g)
    out = []
    for _ in range(n):
        x = torch.randn(B, rank, device="cuda", generator=g) @ A + 0.1 * torch.randn(B, d, device="cuda", generator=g)
        x = x * (d**0.5 / x.norm(dim=-1).mean())
        out.append(x.to(torch.bfloat16))
    return out


@pytest.mark.parametrize("chunks", [1, 3])
@pytest.mark.parametrize("gate,bias,k", [(True, True, 16), (False, False, 8), (True, True, 50), (True, True, 100)])
def test_fused_matches_autograd(gate, bias, k, chunks):
    # chunks > 1: the update runs per feature chunk on its own stream and the next step's encoder GEMM follows it
    # chunk by chunk; results must not depend on it
    d, B, steps, lr = 256, 512, 12, 1e-3
    ref = _model(d=d, k=k, gate=gate, bias=bias)
    fused_model = copy.deepcopy(ref)
    engine = FusedTopKSAEStep(fused_model, overlap_chunks=chunks)
    assert len(engine.chunks) == chunks
    data = _data(steps, B, d)
    opt = torch.optim.Adam(ref.parameters(), lr=lr)
    ref_losses, fused_losses = [], []
    tokens = torch.zeros(B, dtype=torch.long, device="cuda")
    for x in data:
        opt.zero_grad()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = ref.compute_loss({"h": x.float(), "tokens": tokens})["loss"]
        loss.backward()
        opt.step()
        ref_losses.append(float(loss.detach()))
        fused_losses.append(float(engine.step(x, x, k, lr)))
    engine.join()
    K.check_status(torch.device("cuda"))
    r, f = torch.tensor(ref_losses), torch.tensor(fused_losses)
    assert torch.allclose(r, f, rtol=3e-2), (ref_losses, fused_losses)
    assert f[-1] < f[0]
    # parameters moved the same way
    for name in ("W_D", "W_E", "b_E") + (("b_D",) if bias else ()):
        a, b = getattr(ref, name).detach().float(), getattr(fused_model, name).detach().float()
        cos = torch.nn.functional.cosine_similarity(a.flatten(), b.flatten(), dim=0)
        # biases take Adam steps of size ~lr whose sign flips on near-zero gradients and they start at zero, so their direction is noisy: looser bound
        assert cos > (0.9 if name.startswith("b_") else 0.999), (name, float(cos))


def test_fused_clipping_matches_generic_clip():
    from language_model_saes_b200.optim import clip_grad_norm

    d, B, k, lr = 256, 512, 16, 1e-3
    ref = _model(d=d, k=k)
    fused_model = copy.deepcopy(ref)
    unclipped = FusedTopKSAEStep(copy.deepcopy(ref))
    engine = FusedTopKSAEStep(fused_model)
    (x,) = _data(1, B, d)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = ref.compute_loss({"h": x.float(), "tokens": torch.zeros(B, dtype=torch.long, device="cuda")})["loss"]
    loss.backward()
    params = [p for p in ref.parameters() if p.grad is not None]
    want = clip_grad_norm(params, float("inf"))  # the trainer's norm on the generic path: |g|_2 / sqrt(non-zero entries)
    unclipped.step(x, x, k, lr, clip_grad_norm=1e9)  # a bound far above the norm: measured, nothing scaled
    norm = unclipped.last_grad_norm
    assert torch.allclose(norm, want, rtol=3e-2), (norm, want)
    max_norm = 0.25 * float(norm)
    engine.step(x, x, k, lr, clip_grad_norm=max_norm)
    K.check_status(torch.device("cuda"))
    assert torch.allclose(engine.last_grad_norm, norm, rtol=1e-4)
    # first Adam moments = 0.1 x gradient: the clipped ones are the unclipped ones times max_norm / (norm + 1e-6)
    mom = lambda e: torch.sqrt(sum(st[0].square().sum() for st in e.state.values() if st is not None))  # noqa: E731
    assert torch.allclose(mom(engine), mom(unclipped) * max_norm / (norm + 1e-6), rtol=1e-3)
    cos = torch.nn.functional.cosine_similarity(engine.state["W_D"][0].flatten(), ref.W_D.grad.flatten(), dim=0)
    assert cos > 0.99, float(cos)


def test_fused_row_mask_and_transcoder_label():
    d, B, k = 128, 256, 8
    sae = _model(d=d, k=k)
    engine = FusedTopKSAEStep(sae)
    x, y = _data(2, B, d)
    w = (torch.rand(B, device="cuda") > 0.3).float()
    idx, act = engine.encode(x, k)
    xhat = K.ref_sparse_decode(idx, act, engine.WD_bf16, engine.bD)
    want = (((xhat - y.float()) ** 2).sum(-1) * w).sum() / w.sum()
    got = engine.step(x, y, k, 1e-3, row_weight=w, n_tokens_global=int(w.sum()))
    assert torch.allclose(got, want, rtol=1e-3)


@pytest.mark.parametrize("k_aux", [16, 96])
def test_fused_auxk_matches_autograd(k_aux):
    """Aux-K on the fused path against the autograd path: same dead set, same losses, same parameter motion."""
    from language_model_saes_b200.ops.fused_step import AuxK

    d, B, k, steps, lr, alpha, thr = 256, 512, 16, 6, 1e-3, 1 / 32, 1000
    ref = _model(d=d, k=k)
    F = ref.cfg.d_sae
    with torch.no_grad():
        ref.b_E[: F // 4] -= 0.5  # a quarter of the dictionary rarely fires: it goes dead after two batches
    fused_model = copy.deepcopy(ref)
    engine = FusedTopKSAEStep(fused_model)
    aux = AuxK(F, k_aux, alpha, thr, "cuda")
    counter = torch.zeros(F, dtype=torch.long, device="cuda")

    def update_dead(feature_acts, mask, specs):
        nonlocal counter
        fired = (feature_acts > 0).any(dim=0)
        counter = torch.where(fired, torch.zeros_like(counter), counter + feature_acts.shape[0])
        return counter >= thr

    opt = torch.optim.Adam(ref.parameters(), lr=lr)
    tokens = torch.zeros(B, dtype=torch.long, device="cuda")
    ref_l, ref_a, fus_l, fus_a, n_dead = [], [], [], [], []
    for x in _data(steps, B, d):
        opt.zero_grad()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = ref.compute_loss({"h": x.float(), "tokens": tokens}, auxk_coefficient=alpha, k_aux=k_aux,
                                   update_dead_statistics=update_dead, return_aux_data=True)  # fmt: skip
        out["loss"].backward()
        opt.step()
        ref_l.append(float(out["loss"].detach()))
        ref_a.append(float(out["l_aux"].detach().mean()))
        fus_l.append(float(engine.step(x, x, k, lr, aux=aux)))
        fus_a.append(float(engine.last_aux_loss))
        n_dead.append(int(aux.is_dead.sum()))
        # the two paths round differently (bf16 kernels vs autocast), so a feature on the edge of firing may differ
        assert (aux.is_dead != (counter >= thr)).float().mean() < 0.02
    K.check_status(torch.device("cuda"))
    assert n_dead[-1] > 0 and max(fus_a) > 0, (n_dead, fus_a)
    assert torch.allclose(torch.tensor(ref_l), torch.tensor(fus_l), rtol=3e-2), (ref_l, fus_l)
    assert torch.allclose(torch.tensor(ref_a), torch.tensor(fus_a), rtol=6e-2, atol=1e-3), (ref_a, fus_a)
    for name in ("W_D", "W_E"):
        a, b = getattr(ref, name).detach().float(), getattr(fused_model, name).detach().float()
        assert torch.nn.functional.cosine_similarity(a.flatten(), b.flatten(), dim=0) > 0.999
    # the dead features moved (only the auxiliary loss reaches them) and moved the same way
    dead = aux.is_dead & (counter >= thr)
    moved_ref = (ref.W_D.detach()[dead] - _model(d=d, k=k).W_D.detach()[dead]).flatten()
    moved_fus = (fused_model.W_D.detach()[dead] - _model(d=d, k=k).W_D.detach()[dead]).flatten()
    assert moved_fus.abs().sum() > 0
    assert torch.nn.functional.cosine_similarity(moved_ref, moved_fus, dim=0) > 0.9


@pytest.mark.parametrize("act", ["topk", "batchtopk"])
@pytest.mark.parametrize("weighted", [False, True])
def test_auxk_step_does_not_wait_for_the_gpu(act, weighted):
    from language_model_saes_b200.ops.fused_step import AuxK

    d, B, k = 256, 512, 16
    sae = _model(d=d, k=k)
    sae.cfg.act_fn = act
    sae.activation_function = sae.activation_function_factory(None)
    engine, aux = FusedTopKSAEStep(sae), AuxK(sae.cfg.d_sae, 96, 1 / 32, 1000, "cuda")
    w = torch.ones(B, device="cuda") if weighted else None
    data = _data(5, B, d)
    for x in data[:4]:
        engine.step(x, x, k, 1e-3, row_weight=w, aux=aux)
    torch.cuda.synchronize()
    torch.cuda.set_sync_debug_mode("error")
    try:
        engine.step(data[4], data[4], k, 1e-3, row_weight=w, aux=aux)
    finally:
        torch.cuda.set_sync_debug_mode("default")


@pytest.mark.parametrize("gate,k", [(True, 16), (False, 8)])
def test_fused_batchtopk_matches_autograd(gate, k):
    """Batch-level top-k on the fused path (radix-select threshold + threshold compaction) against the generic model."""
    d, B, steps, lr = 256, 512, 10, 1e-3
    ref = _model(d=d, k=k, gate=gate)
    ref.cfg.act_fn = "batchtopk"
    ref.activation_function = ref.activation_function_factory(None)
    fused_model = copy.deepcopy(ref)
    fused_model.activation_function = fused_model.activation_function_factory(None)
    assert FusedTopKSAEStep.supports(fused_model)[0]
    engine = FusedTopKSAEStep(fused_model)
    assert engine.batch_level
    engine.batch_list_factor = 32  # tiny shapes: a token can hold many times the average number of codes
    data = _data(steps, B, d)
    idx, act = engine.encode(data[0], k)
    n_codes = int((idx >= 0).sum())
    assert n_codes == k * B, n_codes  # exactly k codes per token on average (ties at the bf16 threshold are rationed)
    assert int((idx >= 0).sum(-1).max()) > k  # ... but not k per token
    opt = torch.optim.Adam(ref.parameters(), lr=lr)
    ref_losses, fused_losses = [], []
    tokens = torch.zeros(B, dtype=torch.long, device="cuda")
    for x in data:
        opt.zero_grad()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = ref.compute_loss({"h": x.float(), "tokens": tokens})["loss"]
        loss.backward()
        opt.step()
        ref_losses.append(float(loss.detach()))
        fused_losses.append(float(engine.step(x, x, k, lr)))
    K.check_status(torch.device("cuda"))
    r, f = torch.tensor(ref_losses), torch.tensor(fused_losses)
    assert torch.allclose(r, f, rtol=3e-2), (ref_losses, fused_losses)
    for name in ("W_D", "W_E"):
        a, b = getattr(ref, name).detach().float(), getattr(fused_model, name).detach().float()
        assert torch.nn.functional.cosine_similarity(a.flatten(), b.flatten(), dim=0) > 0.999, name


@pytest.mark.parametrize("weighted,gate,bias", [(False, True, True), (True, True, False), (True, False, True)])
@pytest.mark.parametrize("B,k,expansion,route", [(300, 9, 8, 0), (257, 32, 32, 1), (1024, 70, 40, 2), (300, 100, 64, 3), (300, 100, 8, 4), (300, 300, 8, 4)])
def test_one_native_call_is_the_same_step(B, k, expansion, route, weighted, gate, bias):
    """The step in one native call against the same kernels called one by one (which phase timing asks for), for every way to find the codes."""
    a = _model(k=k, expansion=expansion, gate=gate, bias=bias)
    b = copy.deepcopy(a)
    one, by_one = FusedTopKSAEStep(a), FusedTopKSAEStep(b)
    assert K.topk_route(B, one.F, one.d, k, one.dec_norm if gate else None) == route
    w = (torch.rand(B, device="cuda") < 0.8).float() if weighted else None
    for i, x in enumerate(_data(3, B, 256)):
        by_one.start_phase_timing()
        la = one.step(x, x, k, 1e-5, row_weight=w, n_tokens_global=B if weighted else None)
        lb = by_one.step(x, x, k, 1e-5, row_weight=w, n_tokens_global=B if weighted else None)
        assert by_one.phase_marks and one.t == by_one.t == i + 1
        # (sums of rows' losses by atomics; later steps start from parameters of which some differ by up to twice the learning rate)
        # row_topk takes any of the equal bf16 values that compete for a row's last place: a few rows' losses change by one of k codes
        assert torch.allclose(la, lb, rtol=5e-3 if route >= 3 else 1e-5 if i == 0 else 1e-4)
        # features' entries come in the order of the counting sort's atomics: fp32 sums in another order, and Adam's first steps move a
        # parameter by the learning rate whatever its gradient's size
        for (n, p), q in zip(a.named_parameters(), b.parameters()):
            off = (p - q).abs()
            assert float(off.max()) <= 2.1e-5 * (i + 1) and (route >= 3 or float(off.mean()) <= 1e-6 * (i + 1)), n
    K.check_status(torch.device("cuda"))


@pytest.mark.parametrize("B,k,expansion,route", [(300, 9, 8, 0), (257, 32, 32, 1), (1024, 70, 40, 2), (300, 100, 64, 3), (300, 100, 8, 4), (300, 300, 8, 4)])
def test_moments_of_one_native_call(B, k, expansion, route):
    """The gradients' signs and sizes, which a parameter's first steps do not show. Where equal bf16 values compete for a row's last place (routes 3 and
    4) at most one of its k codes differs: were it so in every row, a smallest one, sqrt(2 / k)
    of a gradient; elsewhere only the order of fp32 sums."""
    a = _model(k=k, expansion=expansion)
    b = copy.deepcopy(a)
    one, by_one = FusedTopKSAEStep(a), FusedTopKSAEStep(b)
    assert K.topk_route(B, one.F, one.d, k, one.dec_norm) == route
    x = _data(1, B, 256)[0]
    by_one.start_phase_timing()
    one.step(x, x, k, 1e-5)
    by_one.step(x, x, k, 1e-5)
    bound = (2.0 / k) ** 0.5 if route >= 3 else 1e-4
    for name, moments in one.state.items():
        for p, q in zip(moments, by_one.state[name]):
            assert float(q.abs().max()) > 0 and float((p - q).norm() / q.norm()) <= 2 * bound, name  # (second moments: twice a gradient's share)


def test_step_under_capture():
    """A captured step replays: what it needs comes from the graph's pool, and nothing in it waits for the host."""
    sae = _model()
    engine = FusedTopKSAEStep(sae)
    x = _data(1, 512, 256)[0]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        first = float(engine.step(x, x, 16, 1e-3))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            loss = engine.step(x, x, 16, 1e-3)
        losses = []
        for _ in range(5):
            graph.replay()
            losses.append(float(loss))
    torch.cuda.synchronize()
    assert losses[0] < first and all(q < p for p, q in zip(losses, losses[1:])), (first, losses)


@pytest.mark.parametrize("F,cap,dead", [(8, 8, 0.5), (1000, 512, 0.2), (5003, 5008, 1.0), (4096, 1024, 0.0), (70000, 2048, 0.01), (70000, 2048, 0.1)])
@pytest.mark.parametrize("gated", [False, True])
def test_dead_rows_match_the_plain_statement(F, cap, dead, gated):
    """Blocks that end within the features, a capacity beyond them, none and all dead, more dead features than there is room for."""
    from language_model_saes_b200.ops.fused_step import AuxK

    g = torch.Generator(device="cuda").manual_seed(F)
    d = 72
    since = torch.randint(0, 90, (F,), device="cuda", generator=g)
    since[torch.rand(F, device="cuda", generator=g) < dead] = 95
    fired = (torch.rand(F, device="cuda", generator=g) < 0.1).int() * 3
    WE, WD = (torch.randn(F, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    bias, gate = torch.randn(F, device="cuda", generator=g), torch.rand(F, device="cuda", generator=g) + 0.1 if gated else None
    n_valid = torch.full((), 7, device="cuda")
    a, b = (AuxK(F, 16, 1 / 32, 100.5, "cuda", counter=since.clone()) for _ in range(2))
    a.capacity = b.capacity = cap
    any_dead, row_of, we, wd, b_dead, g_dead = a.compact(fired, n_valid, cap, WE, WD, bias, gate)
    is_dead = b.update(fired, n_valid)
    b.observe(is_dead.sum())
    assert torch.equal(a.tokens_since_last_activation, b.tokens_since_last_activation) and torch.equal(a.is_dead, is_dead)
    assert int(a.truncated_steps) == int(b.truncated_steps) and float(any_dead) == float(is_dead.any())
    rows = is_dead.nonzero().squeeze(1)[:cap]
    n = rows.numel()
    want = torch.full((F,), -1, dtype=torch.int32, device="cuda")
    want[rows] = torch.arange(n, dtype=torch.int32, device="cuda")
    assert torch.equal(row_of, want)
    assert torch.equal(we[:n], WE[rows]) and torch.equal(wd[:n], WD[rows]) and not we[n:].any() and not wd[n:].any()
    assert torch.equal(b_dead[:n], bias[rows]) and torch.isfinite(b_dead).all() and not g_dead[n:].any()
    assert torch.equal(g_dead[:n], gate[rows] if gated else torch.ones(n, device="cuda"))
