"""Performance cases: training steps of every dictionary family on one GPU, a short training run through the trainer, and
inference with a trained dictionary.

``listed()`` names fixed cases, ``draw(rng)`` gives more of the same ranges. ``prepare`` makes the model, the optimizer
state and the inputs that a training (or analysis) program has in hand, ``run`` is one pass through the public entry
points: the ``step`` of the fused engines (what ``Trainer.fit`` calls per batch), ``Trainer.fit`` itself, or ``encode`` and
``decode`` of a model. Activations are low-rank Gaussian mixtures plus noise with a mean norm of ``sqrt(d_model)``, the
statistics that dataset-wise normalised residual streams are scaled to.
"""

from __future__ import annotations

import math
import os
import tempfile

import torch

from language_model_saes_b200 import (
    CLTConfig,
    Crosscoder,
    CrosscoderConfig,
    CrossLayerTranscoder,
    LorsaConfig,
    LowRankSparseAttention,
    SAEConfig,
    SparseAutoEncoder,
    Trainer,
    TrainerConfig,
)
from language_model_saes_b200.ops.fused_clt import FusedCLTStep
from language_model_saes_b200.ops.fused_crosscoder import FusedCrosscoderStep
from language_model_saes_b200.ops.fused_lorsa import FusedLorsaStep
from language_model_saes_b200.ops.fused_step import AuxK, FusedTopKSAEStep

LR = 1e-4  # a learning rate on its way up a warm-up, as most of the first thousands of steps have it
HOOK = "blocks.6.hook_resid_post"


# --------------------------------------------------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # a dictionary on a toy language model (d_model 64, 4x): nothing but launches and latency
        dict(name="topk_tiny", kind="topk", d=64, F=256, k=8, B=512, masked=False),
        # a small model's residual stream (d_model 512, 8x), the framework's plumbing configuration
        dict(name="topk_small", kind="topk", d=512, F=4096, k=32, B=1024, masked=False),
        # the last, ragged batch of an epoch with padding tokens masked out, at sizes that fit no tile
        dict(name="topk_ragged_masked", kind="topk", d=1160, F=13000, k=37, B=3001, masked=True),
        # a k above what the encoder's fused epilogue holds: early steps of a k schedule, or wide codes
        dict(name="topk_wide_k", kind="topk", d=2048, F=32768, k=128, B=4096, masked=False),
        # an 8-billion-parameter model's residual stream (d_model 4096, 32x): the headline training step
        dict(name="topk_large", kind="topk", d=4096, F=131072, k=50, B=4096, masked=False),
        # batch-level selection with dead features revived by the auxiliary loss
        dict(name="batchtopk_auxk", kind="batchtopk", d=2048, F=65536, k=64, B=4096, k_aux=512, dead=0.1),
        # a JumpReLU dictionary with the tanh sparsity penalty
        dict(name="jumprelu", kind="jumprelu", d=2304, F=18432, B=4096, l0=64),
        # a crosscoder over eight snapshots of one model, all heads on this GPU
        dict(name="crosscoder", kind="crosscoder", heads=8, d=768, F=98304, B=4096, l0=44),
        # a cross-layer transcoder of a 12-layer model (78 decoder matrices)
        dict(name="clt", kind="clt", L=12, d=768, F=24576, k=64, B=2048),
        # low-rank sparse attention in place of one attention layer
        dict(name="lorsa", kind="lorsa", heads=64, group=128, dqk=64, d=768, k=128, batch=2, seq=1024),
        # a training run through the trainer: pinned host batches in, weights out (d_model 768, 32x, k 50)
        dict(name="fit", kind="fit", d=768, F=24576, k=50, B=4096, steps=16),
        # analysis of a trained dictionary: dense feature activations and reconstructions in fp32
        dict(name="forward_topk", kind="forward", act="topk", d=768, F=24576, k=50, B=4096),
    ]


def _log_int(rng, lo: int, hi: int, step: int = 1) -> int:
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v / step + 0.5) * step))


def draw(rng) -> dict:
    most = [work(c) for c in listed()]
    top_b, top_f = max(w["bytes"] for w in most), max(w["flops"] for w in most)
    while True:
        c = _draw(rng)
        w = work(c)
        if w["bytes"] <= top_b and w["flops"] <= top_f:
            return c


def _draw(rng) -> dict:
    kind = rng.choice(["topk", "topk", "fit", "batchtopk", "jumprelu", "crosscoder", "clt", "lorsa", "forward"])
    if kind == "topk":
        F = _log_int(rng, 256, 131072, 8)
        return dict(kind=kind, d=_log_int(rng, 64, 4096, 8), F=F, k=min(_log_int(rng, 8, 128), F // 16), B=_log_int(rng, 256, 8192),
                    masked=rng.random() < 0.3)  # fmt: skip
    if kind == "batchtopk":
        return dict(kind=kind, d=_log_int(rng, 256, 2048, 8), F=_log_int(rng, 4096, 65536, 8), k=_log_int(rng, 16, 64),
                    B=_log_int(rng, 512, 4096), k_aux=rng.choice([256, 512]), dead=rng.choice([0.02, 0.1, 0.2]))  # fmt: skip
    if kind == "jumprelu":
        return dict(kind=kind, d=_log_int(rng, 256, 2304, 64), F=_log_int(rng, 2048, 32768, 8), B=_log_int(rng, 512, 4096), l0=_log_int(rng, 20, 80))
    if kind == "crosscoder":
        return dict(kind=kind, heads=rng.randint(2, 8), d=_log_int(rng, 256, 768, 64), F=_log_int(rng, 4096, 98304, 8), B=_log_int(rng, 512, 4096),
                    l0=_log_int(rng, 20, 60))  # fmt: skip
    if kind == "clt":
        return dict(kind=kind, L=rng.randint(2, 12), d=_log_int(rng, 256, 768, 8), F=_log_int(rng, 2048, 24576, 8), k=_log_int(rng, 16, 64),
                    B=_log_int(rng, 256, 2048))  # fmt: skip
    if kind == "lorsa":
        return dict(kind=kind, heads=rng.choice([8, 12, 16, 32, 48, 64]), group=rng.choice([64, 128]), dqk=64, d=_log_int(rng, 512, 1024, 64),
                    k=_log_int(rng, 32, 128), batch=rng.randint(1, 4), seq=_log_int(rng, 128, 1024, 8))  # fmt: skip
    if kind == "fit":
        return dict(kind=kind, d=_log_int(rng, 256, 1024, 8), F=_log_int(rng, 2048, 24576, 8), k=_log_int(rng, 16, 64), B=_log_int(rng, 512, 4096),
                    steps=rng.randint(8, 16))  # fmt: skip
    return dict(kind=kind, act=rng.choice(["topk", "jumprelu"]), d=_log_int(rng, 64, 2048, 8), F=_log_int(rng, 1024, 32768, 8), k=_log_int(rng, 16, 64),
                B=_log_int(rng, 256, 8192))  # fmt: skip


# --------------------------------------------------------------------------------------------------------------------
# inputs and models
# --------------------------------------------------------------------------------------------------------------------
def _activations(shape: tuple[int, ...], d: int, g: torch.Generator, mix: torch.Tensor) -> torch.Tensor:
    """``[*shape, d]`` bf16: low-rank Gaussian plus isotropic noise, mean norm ``sqrt(d)``."""
    x = torch.randn(*shape, mix.shape[0], device="cuda", generator=g) @ mix
    x += 0.1 * torch.randn(*shape, d, device="cuda", generator=g)
    return (x * (d**0.5 / x.norm(dim=-1).mean())).to(torch.bfloat16)


def _mix(d: int, g: torch.Generator) -> torch.Tensor:
    return torch.randn(min(256, max(16, d // 4)), d, device="cuda", generator=g)


def _expansion(F: int, d: int) -> float:
    """The configurations state ``d_sae`` as ``int(d_model * expansion_factor)``."""
    return (F + 0.5) / d


def _sae(act: str, d: int, F: int, k: int) -> SparseAutoEncoder:
    cfg = SAEConfig(hook_point_in=HOOK, hook_point_out=HOOK, d_model=d, expansion_factor=_expansion(F, d), act_fn=act, top_k=k, device="cuda",
                    dtype=torch.float32)  # fmt: skip
    sae = SparseAutoEncoder(cfg)
    assert sae.W_D.shape == (F, d)
    bound = d**-0.5
    sae.init_parameters(encoder_uniform_bound=bound, decoder_uniform_bound=bound, init_log_jumprelu_threshold_value=0.0)
    sae.set_decoder_to_fixed_norm(1.0, force_exact=True)
    sae.init_encoder_with_decoder_transpose()
    with torch.no_grad():  # what training leaves: decoder norms that differ, biases
        sae.W_D.mul_(1 + 0.05 * torch.randn(F, 1, device="cuda"))
        sae.b_E.normal_(-0.02, 0.02)
        sae.b_D.normal_(0.0, 0.02)
    sae.set_dataset_average_activation_norm({HOOK: d**0.5})
    return sae


@torch.no_grad()
def _set_thresholds(model, sums: torch.Tensor, l0: int) -> None:
    """JumpReLU thresholds at which ``l0`` features per token of the pre-activations ``sums [tokens, F]`` are active, with
    the spread between features that training leaves."""
    F = sums.shape[1]
    t = sums.float().topk(min(l0, F), dim=1).values[:, -1].mean().clamp_min(1e-2).log()
    p = model.activation_function.log_jumprelu_threshold
    p.copy_(t + 0.05 * torch.randn_like(p))


@torch.no_grad()
def prepare(case: dict, seed: int):
    torch.manual_seed(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind, d = case["kind"], case["d"]
    mix = _mix(d, g)
    s = {"kind": kind}
    if kind in ("topk", "batchtopk"):
        B, F, k = case["B"], case["F"], case["k"]
        sae = _sae(kind, d, F, k)
        s.update(sae=sae, k=k, x=_activations((B,), d, g, mix), weight=None, n=None, aux=None)
        if case.get("masked"):
            keep = (torch.rand(B, device="cuda", generator=g) < 0.9).float()
            s["weight"], s["n"] = keep * (B / keep.sum()), B
        if kind == "batchtopk":
            # features that stopped firing: small encoder rows, counters beyond the dead threshold
            dead = torch.rand(F, device="cuda", generator=g) < case["dead"]
            sae.W_E.data.t()[dead] *= 0.1
            threshold = 10_000_000
            counter = torch.where(dead, threshold + 1, 0).to(torch.long)
            s["aux"] = AuxK(F, case["k_aux"], 1 / 32, threshold, sae.W_D.device, counter=counter)
        s["engine"] = FusedTopKSAEStep(sae)
    elif kind == "jumprelu":
        sae = _sae("jumprelu", d, case["F"], 0)
        x = _activations((case["B"],), d, g, mix)
        _set_thresholds(sae, x[:64].float() @ sae.W_E, case["l0"])
        s.update(sae=sae, x=x.unsqueeze(1), engine=FusedCrosscoderStep(sae))
    elif kind == "crosscoder":
        H, F = case["heads"], case["F"]
        cfg = CrosscoderConfig(hook_points=[f"snapshot{h}.{HOOK}" for h in range(H)], d_model=d, expansion_factor=_expansion(F, d), act_fn="jumprelu",
                               device="cuda", dtype=torch.float32)  # fmt: skip
        cc = Crosscoder(cfg)
        assert cc.W_D.shape == (H, F, d)
        bound = d**-0.5
        cc.init_parameters(encoder_uniform_bound=bound, decoder_uniform_bound=bound, init_log_jumprelu_threshold_value=0.0)
        cc.set_decoder_to_fixed_norm(1.0, force_exact=True)
        cc.init_encoder_with_decoder_transpose(1.0 / H)
        cc.W_D.data.mul_(1 + 0.05 * torch.randn(H, F, 1, device="cuda", generator=g))  # the heads' decoder norms differ
        cc.b_E.data.normal_(-0.02 / H, 0.02)
        cc.b_D.data.normal_(0.0, 0.02)
        z = torch.randn(case["B"], mix.shape[0], device="cuda", generator=g)
        cols = []
        for _ in range(H):  # snapshots of one model on the same tokens: correlated activations
            x = z @ (mix + 0.3 * _mix(d, g)) + 0.1 * torch.randn(case["B"], d, device="cuda", generator=g)
            cols.append((x * (d**0.5 / x.norm(dim=-1).mean())).to(torch.bfloat16))
        x = torch.stack(cols, dim=1)
        _set_thresholds(cc, torch.einsum("bhd,hdf->bf", x[:32].float(), cc.W_E.data), case["l0"])
        s.update(sae=cc, x=x, engine=FusedCrosscoderStep(cc))
    elif kind == "clt":
        L, B = case["L"], case["B"]
        cfg = CLTConfig(hook_points_in=[f"blocks.{i}.ln2.hook_normalized" for i in range(L)], hook_points_out=[f"blocks.{i}.hook_mlp_out" for i in range(L)],
                        d_model=d, expansion_factor=_expansion(case["F"], d), act_fn="topk", top_k=case["k"], device="cuda", dtype=torch.float32)  # fmt: skip
        clt = CrossLayerTranscoder(cfg)
        assert clt.b_E.shape == (L, case["F"])
        clt.init_parameters()
        for b in (clt.b_E, *clt.b_D):
            b.data.normal_(0.0, 0.02)
        z = torch.randn(B, mix.shape[0], device="cuda", generator=g)

        def layers():
            out = []
            for _ in range(L):
                v = z @ _mix(d, g) + 0.1 * torch.randn(B, d, device="cuda", generator=g)
                out.append((v * (d**0.5 / v.norm(dim=-1).mean())).to(torch.bfloat16))
            return torch.stack(out)

        xt, y = layers(), layers()
        s.update(sae=clt, k=case["k"], xt=xt, x=xt.transpose(0, 1), y=y, engine=FusedCLTStep(clt))
    elif kind == "lorsa":
        F, T = case["heads"] * case["group"], (case["batch"], case["seq"])
        cfg = LorsaConfig(hook_point_in="blocks.6.ln1.hook_normalized", hook_point_out="blocks.6.hook_attn_out", d_model=d, expansion_factor=_expansion(F, d),
                          n_qk_heads=case["heads"], d_qk_head=case["dqk"], rotary_dim=case["dqk"], n_ctx=case["seq"], act_fn="topk", top_k=case["k"],
                          device="cuda", dtype=torch.float32)  # fmt: skip
        lorsa = LowRankSparseAttention(cfg)
        assert lorsa.W_V.shape[0] == F
        lorsa.init_parameters()
        for b in (lorsa.b_Q, lorsa.b_K, lorsa.b_V, lorsa.b_D):
            b.data.normal_(0.0, 0.02)
        x = _activations(T, d, g, mix)
        y = (x.float().cumsum(1) / torch.arange(1, T[1] + 1, device="cuda").sqrt()[None, :, None]).to(torch.bfloat16)
        s.update(sae=lorsa, k=case["k"], x=x, y=y, engine=FusedLorsaStep(lorsa))
    elif kind == "fit":
        B = case["B"]
        sae = _sae("topk", d, case["F"], case["k"])
        tokens = torch.zeros(B, dtype=torch.long).pin_memory()
        batches = [{HOOK: _activations((B,), d, g, mix).cpu().pin_memory(), "tokens": tokens} for _ in range(case["steps"])]
        cfg = TrainerConfig(total_training_tokens=case["steps"] * B, lr=LR, lr_scheduler_name="constant", log_frequency=1, l1_coefficient=None,
                            k_warmup_steps=0, skip_metrics_calculation=True, n_checkpoints=0,
                            exp_result_path=os.path.join(tempfile.gettempdir(), "lmsae_perf_fit"))  # fmt: skip
        s.update(sae=sae, batches=batches, cfg=cfg)
    else:
        sae = _sae(case["act"], d, case["F"], case["k"])
        x = _activations((case["B"],), d, g, mix).float()
        if case["act"] == "jumprelu":
            _set_thresholds(sae, x[:64] @ sae.W_E, case["k"])
        s.update(sae=sae.eval(), x=x)
    return s


# --------------------------------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------------------------------
def run(s: dict):
    kind, sae = s["kind"], s["sae"]
    if kind == "forward":
        with torch.no_grad():
            acts = sae.encode(s["x"])
            return acts, sae.decode(acts)
    if kind == "fit":
        trainer = Trainer(s["cfg"])
        trainer.fit(sae, s["batches"])
        loss = trainer.last_loss
    elif kind in ("topk", "batchtopk"):
        loss = s["engine"].step(s["x"], s["x"], s["k"], LR, row_weight=s["weight"], n_tokens_global=s["n"], aux=s["aux"])
    elif kind == "clt":
        loss = s["engine"].step(s["x"], s["y"], s["k"], LR, xt=s["xt"])
    elif kind == "lorsa":
        loss = s["engine"].step(s["x"], s["y"], s["k"], LR)
    else:
        loss = s["engine"].step(s["x"], LR, l1_coefficient=1e-3)
    return {"loss": loss, **{n: p.data for n, p in sae.named_parameters()}}


# --------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct implementations are apart
# --------------------------------------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    """Training: parameters and both Adam moments read and written once in fp32 (24 bytes per parameter), inputs and targets
    read once; one dense encoder product (crosscoder and JumpReLU: a second one for the threshold gradient) plus the
    sparse products of decoder, code gradients and weight gradients. Inference: weights and inputs in, activations and
    reconstruction out."""
    kind, d = case["kind"], case["d"]
    if kind in ("topk", "batchtopk", "fit"):
        F, B, k = case["F"], case["B"], case["k"]
        n = case.get("steps", 1)
        b, f = 24.0 * 2 * F * d + 2.0 * B * d, 2.0 * B * F * d + 8.0 * B * k * d
        if kind == "batchtopk":
            dead = case["dead"] * F
            f += 8.0 * B * dead * d  # auxiliary encoder, decoder and two gradients over the dead features
        return {"bytes": n * b, "flops": n * f}
    if kind in ("jumprelu", "crosscoder"):
        F, B, H, k = case["F"], case["B"], case.get("heads", 1), case["l0"]
        return {"bytes": H * (24.0 * 2 * F * d + 2.0 * B * d), "flops": H * (4.0 * B * F * d + 8.0 * B * k * d)}
    if kind == "clt":
        L, F, B, k = case["L"], case["F"], case["B"], case["k"]
        pairs = L * (L + 1) / 2
        return {"bytes": 24.0 * (pairs + L) * F * d + 4.0 * L * B * d, "flops": 2.0 * L * B * F * d + (6.0 * pairs + 2.0 * L) * B * k * d}
    if kind == "lorsa":
        h, q, v, s = case["heads"], case["dqk"], case["group"], case["seq"]
        T, F = case["batch"] * s, h * v
        proj = 2.0 * h * q + F
        attn = 2.0 * case["batch"] * h * s * s / 2 * (q + v + 3 * q + 2 * v)
        return {"bytes": 24.0 * d * (proj + F) + 4.0 * T * d, "flops": 4.0 * T * d * proj + attn + 6.0 * T * case["k"] * d}
    F, B = case["F"], case["B"]
    return {"bytes": 4.0 * (2 * F * d + 2 * B * d + B * F), "flops": 2.0 * B * F * d + 2.0 * B * case["k"] * d}


def tolerance(case: dict) -> dict:
    """Measured: each engine against its own torch statements on the CPU (same bf16 operands, other orders of summation), two
    steps from the same state, d_model 256. Adam's first steps move a parameter by about the learning rate whatever
    its gradient's size, so what differs is the sign of gradients that are zero up to rounding."""
    kind = case["kind"]
    if kind == "forward":
        return {"rel": 1e-5, "max": 1e-3}  # fp32 sums of up to d_model products
    if kind == "lorsa":
        # a constant added to all keys leaves the attention as it is: the gradient of b_K is rounding alone (measured 4.7e-3)
        return {"rel": 2e-2, "max": 0.2}
    return {"rel": 1e-3, "max": 0.06}  # measured 2.3e-4 and 0.016
