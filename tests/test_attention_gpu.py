"""tcgen05 causal attention with d_v != d_qk against the fp32 torch oracle."""

import pytest
import torch

from language_model_saes_b200.ops import attention as A
from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,h,dqk,dv", [(2, 256, 3, 64, 128), (1, 384, 2, 128, 64), (2, 200, 2, 64, 256), (1, 1024, 4, 64, 128),
                                          (3, 128, 1, 128, 128), (1, 72, 2, 64, 64)])  # fmt: skip
def test_forward_matches_oracle(b, s, h, dqk, dv):
    torch.manual_seed(0)
    dev = torch.device("cuda")
    q = torch.randn(b, s, h, dqk, device=dev).to(torch.bfloat16)
    k = torch.randn(b, s, h, dqk, device=dev).to(torch.bfloat16)
    v = torch.randn(b, s, h, dv, device=dev).to(torch.bfloat16)
    scale = 1.7 / dqk**0.5
    out, lse = A.causal_attention_fwd(q, k, v, scale, want_lse=True)
    K.check_status(dev)
    want, want_lse = A.ref_causal_attention(q, k, v, scale)
    assert out.shape == want.shape and out.dtype == torch.bfloat16
    assert torch.allclose(lse, want_lse, atol=2e-3, rtol=1e-3), float((lse - want_lse).abs().max())
    assert torch.allclose(out.float(), want, atol=2e-2, rtol=2e-2), float((out.float() - want).abs().max())


@pytest.mark.parametrize("b,s,h,dqk,dv", [(2, 256, 2, 64, 128), (1, 384, 2, 128, 64), (1, 200, 2, 64, 256), (1, 512, 3, 64, 64),
                                          (2, 128, 1, 128, 128), (1, 72, 1, 64, 192)])  # fmt: skip
def test_backward_matches_autograd_of_the_oracle(b, s, h, dqk, dv):
    torch.manual_seed(1)
    dev = torch.device("cuda")
    q, k = (torch.randn(b, s, h, dqk, device=dev).to(torch.bfloat16).float().requires_grad_() for _ in range(2))
    v = torch.randn(b, s, h, dv, device=dev).to(torch.bfloat16).float().requires_grad_()
    scale = 1.3 / dqk**0.5
    dout = torch.randn(b, s, h, dv, device=dev).to(torch.bfloat16).float()
    out = A.causal_attention(q, k, v, scale)
    out.backward(dout)
    K.check_status(dev)
    got = [t.grad.clone() for t in (q, k, v)]
    for t in (q, k, v):
        t.grad = None
    want_out, _ = A.ref_causal_attention(q, k, v, scale)
    want_out.backward(dout)
    assert torch.allclose(out, want_out, atol=2e-2, rtol=2e-2)
    for name, g, t in zip("qkv", got, (q, k, v)):
        rel = float((g - t.grad).norm() / t.grad.norm())
        assert rel < 2e-2, (name, rel)
        assert torch.allclose(g, t.grad, atol=0.05 * float(t.grad.abs().max()), rtol=0.05), name


# sequences shorter than, equal to and just past a 128-position block; value widths of one atom up to ones that are streamed (320: five)
@pytest.mark.parametrize("b,s,h,dqk,dv", [(1, 8, 1, 64, 64), (3, 72, 2, 64, 192), (2, 136, 3, 64, 320), (2, 264, 2, 128, 256), (37, 128, 5, 64, 128)])
def test_backward_of_bf16_tensors_stays_inside_each_sequence(b, s, h, dqk, dv):
    """bf16 inputs get bf16 gradients (fp32 sums, rounded once: 2^-9 of a value, on top of the bf16 products' error); a sequence of NaNs
    behind another one does not reach it although their blocks of positions overlap."""
    torch.manual_seed(2)
    q, k = (torch.randn(b, s, h, dqk, device="cuda").to(torch.bfloat16) for _ in range(2))
    v, dout = (torch.randn(b, s, h, dv, device="cuda").to(torch.bfloat16) for _ in range(2))
    for t in (q, k, v, dout):
        if b > 1:
            t[-1] = float("nan")
    n = max(1, b - 1)
    args = [t.clone().requires_grad_() for t in (q, k, v)]
    out = A.causal_attention(*args, 1.3 / dqk**0.5)
    out.backward(dout)
    K.check_status(torch.device("cuda"))
    ref = [t[:n].float().requires_grad_() for t in (q, k, v)]
    want, _ = A.ref_causal_attention(*ref, 1.3 / dqk**0.5)
    want.backward(dout[:n].float())
    assert torch.allclose(out[:n].float(), want, atol=2e-2, rtol=2e-2)
    for name, g, t in zip("qkv", args, ref):
        assert g.grad.dtype == torch.bfloat16
        rel = float((g.grad[:n].float() - t.grad).norm() / t.grad.norm().clamp_min(1e-6))
        assert rel < 2e-2, (name, rel)


@pytest.mark.parametrize("b,s,h,dv", [(1, 8, 1, 8), (2, 24, 3, 64), (1, 40, 5, 136), (2, 16, 2, 256)])
def test_delta_matches_the_plain_sum(b, s, h, dv):
    torch.manual_seed(3)
    x, y = (torch.randn(b, s, h, dv, device="cuda").to(torch.bfloat16) for _ in range(2))
    delta = torch.empty(b, h, s, device="cuda")
    K._ext().attn_delta(x, y, delta)
    want = (x.double() * y.double()).sum(-1).permute(0, 2, 1)
    bound = dv * 2.0**-24 * (x.double() * y.double()).abs().sum(-1).permute(0, 2, 1)  # dv roundings of partial sums
    assert bool(((delta.double() - want).abs() <= bound).all())


def test_lorsa_encode_uses_the_tensor_core_attention_and_matches_the_score_path():
    from language_model_saes_b200.models.lorsa import LorsaConfig, LowRankSparseAttention

    torch.manual_seed(0)
    cfg = LorsaConfig(hook_point_in="in", hook_point_out="out", d_model=128, expansion_factor=4, n_qk_heads=4, d_qk_head=64,
                      n_ctx=64, act_fn="relu", device="cuda", dtype=torch.bfloat16, norm_activation="inference",
                      positional_embedding_type="rotary", rotary_dim=64, attention_kernel="tensor_core")  # fmt: skip
    m = LowRankSparseAttention(cfg)
    m.init_parameters(encoder_uniform_bound=0.2, decoder_uniform_bound=0.2, init_log_jumprelu_threshold_value=0.0)
    x = torch.randn(2, 64, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    before = K.kernel_launch_count()
    fast, hidden_fast = m.encode(x, return_hidden_pre=True)
    assert K.kernel_launch_count() > before  # the tcgen05 forward ran (OV group 128, d_qk 64)
    slow, hidden_slow, _ = m.encode(x, return_hidden_pre=True, return_attention_pattern=True)
    K.check_status(torch.device("cuda"))
    assert torch.allclose(hidden_fast.float(), hidden_slow.float(), atol=3e-2, rtol=3e-2)
    hidden_fast.float().pow(2).sum().backward()
    g_fast = x.grad.clone()
    x.grad = None
    hidden_slow.float().pow(2).sum().backward()
    rel = float((g_fast.float() - x.grad.float()).norm() / x.grad.float().norm())
    assert rel < 5e-2, rel


def test_transposed_values():
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k = (torch.randn(2, 136, 3, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    v = torch.randn(2, 136, 3, 128, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
    vt = v.detach().permute(0, 2, 3, 1).contiguous().requires_grad_()
    a, b = A.causal_attention(q, k, v), A.causal_attention(q, k, vt=vt)
    a.float().square().sum().backward()
    b.float().square().sum().backward()
    K.check_status(torch.device("cuda"))
    assert torch.equal(a, b) and torch.equal(vt.grad, v.grad.permute(0, 2, 3, 1))
    with pytest.raises(ValueError):
        A.causal_attention(q, k)
