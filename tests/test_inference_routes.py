"""The calls that inference's kernels must leave to the tensor operations: symbolic tracing, and whatever listens between them."""

import pytest
import torch

from language_model_saes_b200 import SAEConfig, SparseAutoEncoder
from language_model_saes_b200.hooks import HookPoint


def _sae(act, device="cpu"):
    torch.manual_seed(0)
    cfg = SAEConfig(hook_point_in="h", hook_point_out="h", d_model=16, expansion_factor=4, act_fn=act, top_k=4, device=device, dtype=torch.float32)
    sae = SparseAutoEncoder(cfg)
    sae.init_parameters(encoder_uniform_bound=0.2, decoder_uniform_bound=0.2, init_log_jumprelu_threshold_value=-1.0)
    return sae


class _Decode(torch.nn.Module):
    def __init__(self, sae):
        super().__init__()
        self.sae = sae

    def forward(self, acts):
        return self.sae.decode(acts)


class _Both(_Decode):
    def forward(self, x):
        return self.sae.decode(self.sae.encode(x))


@pytest.mark.parametrize("act", ["relu", "topk", "jumprelu", "batchtopk"])
def test_symbolic_tracing(act):
    decode = _Decode(_sae(act))
    acts = torch.rand(3, 64)
    assert torch.equal(torch.fx.symbolic_trace(decode)(acts), decode(acts))
    if act == "relu":  # (the other activation functions look at values)
        both, x = _Both(decode.sae), torch.randn(3, 16)
        assert torch.equal(torch.fx.symbolic_trace(both)(x), both(x))


def _kinds():
    one = lambda *a: None  # noqa: E731
    M = torch.nn.modules.module
    return {
        "none": lambda hp: None,
        "hook": lambda hp: hp.add_hook(one),
        "backward hook": lambda hp: hp.add_hook(one, dir="bwd"),
        "module hook": lambda hp: hp.register_forward_hook(one),
        "module pre-hook": lambda hp: hp.register_forward_pre_hook(one),
        "module backward hook": lambda hp: hp.register_full_backward_hook(one),
        "own forward": lambda hp: setattr(hp, "forward", lambda x: x),
        "global hook": lambda hp: M.register_module_forward_hook(one),
        "global pre-hook": lambda hp: M.register_module_forward_pre_hook(one),
    }


@pytest.mark.parametrize("kind", list(_kinds()))
def test_what_a_hook_point_calls_silent(kind):
    hp = HookPoint()
    handle = _kinds()[kind](hp)
    try:
        assert hp.is_silent() == (kind == "none")
    finally:
        if kind.startswith("global"):
            handle.remove()
    assert not type("Other", (HookPoint,), {})().is_silent()


@pytest.mark.gpu
@pytest.mark.parametrize("point", ["hook_hidden_pre", "hook_feature_acts"])
@pytest.mark.parametrize("how", ["hook", "pre-hook", "global hook"])
def test_listeners_of_every_kind_are_called(point, how):
    sae, x, seen = _sae("topk", "cuda"), torch.randn(5, 16, device="cuda"), []
    hp = getattr(sae, point)
    if how == "hook":
        handle = hp.register_forward_hook(lambda m, args, out: out * 2)
    elif how == "pre-hook":
        handle = hp.register_forward_pre_hook(lambda m, args: (args[0] * 2,))
    else:
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, args, out: out * 2 if m is hp else None)
    with torch.no_grad():
        heard = sae.encode(x)
        handle.remove()
        plain = sae.encode(x)
    assert plain.any() and torch.allclose(heard, plain * 2)


@pytest.mark.parametrize("B,F,d,kernel", [(256, 1024, 768, False), (4096, 1024, 256, False), (4096, 1024, 768, True), (256, 4096, 512, True),
                                          (4096, 24576, 768, True), (4096, 24578, 768, False), (1, 131072, 1024, False)])  # fmt: skip
def test_decoders_below_the_cost_of_the_launches_are_products(B, F, d, kernel):
    from language_model_saes_b200.ops.inference import sparse_decode_supported

    assert sparse_decode_supported(torch.empty(B, F, device="meta"), torch.empty(F, d, device="meta")) is kernel
