"""The row-streaming gradient + Adam kernel at the widths where its layout changes (one to eight warps per row, partial last
chunks), with empty rows, rows longer than one batch of entries and rows long enough to be shared by a whole CTA, against
the wrapper's plain-torch statement on CPU copies."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(d, F, B, k, seed):
    g = torch.Generator().manual_seed(seed)
    idx = torch.stack([torch.randperm(F - 3, generator=g)[:k] for _ in range(B)]).to(torch.int32) + 2
    idx[:, 0] = 0  # a feature with an entry of every token (a long list), and ...
    idx[: K.HEAVY_ROW, 1] = 1  # ... one right at the limit
    idx[5, 2:] = -1
    act = torch.rand(B, k, generator=g) + 0.1
    act[7, :] = 0.0  # listed, but inactive
    dact = torch.randn(B, k, generator=g)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    t = dict(idx=idx, act=act, dact=dact, x=r(B, d).to(torch.bfloat16), dx=(r(B, d) * 0.1).to(torch.bfloat16), WD=r(F, d), WE=r(F, d), b=r(F),
             n=torch.zeros(F), gsq=torch.zeros(1), scale=torch.rand(F, generator=g) * 0.1, acc=torch.zeros(F),
             row_of=torch.where(torch.arange(F) % 5 == 0, torch.arange(F) // 5, -1).to(torch.int32), xD=r(F, d), xE=r(F, d), xb=r(F))  # fmt: skip
    for n, s in (("mD", (F, d)), ("vD", (F, d)), ("mE", (F, d)), ("vE", (F, d)), ("mb", (F,)), ("vb", (F,))):
        t[n] = torch.rand(*s, generator=g) * 0.01
    t["WD16"], t["WE16"] = t["WD"].to(torch.bfloat16), t["WE"].to(torch.bfloat16)
    return t


def _compare(cpu, gpu, names, d):
    for n in names:
        a, b = gpu[n].cpu().float(), cpu[n].float()
        # fp32 sums of at most 200 terms (entries of a row) or d terms (code gradients) of order one, in another order
        tol = 2**-24 * max(200, d) * 4 if n in ("dact", "gsq", "acc") else 2e-5
        assert torch.allclose(a, b, atol=max(tol, 2e-5), rtol=3e-4), (n, float((a - b).abs().max()))


@pytest.mark.parametrize("d", [64, 132, 768, 1024, 1028, 1160, 2052, 4100, 8192])
@pytest.mark.parametrize("sides,mode", [("both", 0), ("both", 1), ("decoder", 2), ("encoder", 0)])
def test_row_kernel_matches_the_plain_statement(d, sides, mode):
    F, B, k = 230, 200, 6
    cpu = _case(d, F, B, k, seed=d)
    gpu = {n: t.clone().to(DEV) for n, t in cpu.items()}

    def run(t, step):
        groups = K.FeatureGroups(F, B * k, t["idx"].device).build(t["idx"])
        D = [t["WD"], t["mD"], t["vD"], t["WD16"]] if sides != "encoder" else [None] * 4
        E = [t["WE"], t["mE"], t["vE"], t["WE16"], t["b"], t["mb"], t["vb"]] if sides != "decoder" else [None] * 7
        both = sides == "both"
        K.sparse_grad_adam(groups, t["act"], t["dact"], t["x"], t["dx"], *D, *E, t["n"] if both else None, None, t["gsq"] if both else None, 1e-3,
                           0.9, 0.999, 1e-8, step, True, extra=(t["row_of"], t["xD"], t["xE"], t["xb"]) if both else None,
                           wd_self_scale=t["scale"] if sides == "decoder" else None, norm_sq_accum=t["acc"] if sides == "decoder" else None,
                           dact_mode=mode)  # fmt: skip
        return groups

    for step in (1, 2):
        run(cpu, step)
        groups = run(gpu, step)
        K.check_status(torch.device(DEV))
        assert int(groups.heavy[0]) == 1 and int(groups.heavy[1]) == 0
        assert groups.sched.tolist() == [0, 0]  # ready for the next launch
    _compare(cpu, gpu, ["dact", "WD", "mD", "vD", "WE", "mE", "vE", "b", "mb", "vb", "n", "acc"], d)
    assert torch.allclose(gpu["gsq"].cpu(), cpu["gsq"], rtol=1e-3)
    if sides != "encoder":
        assert torch.equal(gpu["WD16"].float(), gpu["WD"].to(torch.bfloat16).float())
    if sides != "decoder":
        assert torch.equal(gpu["WE16"].float(), gpu["WE"].to(torch.bfloat16).float())


def test_gradient_pass_without_an_update_leaves_code_gradients_and_norm_only():
    cpu = _case(260, 230, 200, 6, seed=3)
    gpu = {n: t.clone().to(DEV) for n, t in cpu.items()}
    for t in (cpu, gpu):
        groups = K.FeatureGroups(230, 1200, t["idx"].device).build(t["idx"])
        K.sparse_grad_adam(groups, t["act"], t["dact"], t["x"], t["dx"], t["WD"], t["mD"], t["vD"], t["WD16"], t["WE"], t["mE"], t["vE"], t["WE16"],
                           t["b"], t["mb"], t["vb"], t["n"], None, t["gsq"], 1e-3, 0.9, 0.999, 1e-8, 1, False, dact_mode=1)  # fmt: skip
    _compare(cpu, gpu, ["dact", "WD", "mD", "WE", "vE", "b", "n"], 260)
    assert torch.allclose(gpu["gsq"].cpu(), cpu["gsq"], rtol=1e-3)


@pytest.mark.parametrize("d", [768, 1160, 4100])
@pytest.mark.parametrize("sides,mode", [("both", 0), ("both", 1), ("decoder", 2), ("encoder", 0)])
def test_rows_whose_copies_were_not_waited_for_stay_as_they_are(d, sides, mode):
    cpu = _case(d, 230, 200, 6, seed=d)
    t = {n: v.clone().to(DEV) for n, v in cpu.items()}
    groups = K.FeatureGroups(230, 1200, t["idx"].device).build(t["idx"])
    D = [t["WD"], t["mD"], t["vD"], t["WD16"]] if sides != "encoder" else [None] * 4
    E = [t["WE"], t["mE"], t["vE"], t["WE16"], t["b"], t["mb"], t["vb"]] if sides != "decoder" else [None] * 7

    def run(**kw):
        K.sparse_grad_adam(groups, t["act"], t["dact"], t["x"], t["dx"], *D, *E, t["n"] if sides == "both" else None, None, None, 1e-3, 0.9, 0.999,
                           1e-8, 1, True, norm_sq_accum=t["acc"] if sides == "decoder" else None, dact_mode=mode, **kw)  # fmt: skip

    K.check_status(torch.device(DEV))
    run(wait_cycles=0)
    with pytest.raises(K.KernelStatusError):
        K.check_status(torch.device(DEV))
    for n in cpu:
        assert torch.equal(t[n].cpu(), cpu[n]), n
    assert groups.sched.tolist() == [0, 0]
    run()  # the next launch works as ever
    K.check_status(torch.device(DEV))
    assert not torch.equal((t["WD"] if sides != "encoder" else t["WE"]).cpu(), cpu["WD"] if sides != "encoder" else cpu["WE"])


@pytest.mark.parametrize("d", [4, 64, 124, 128, 132, 256, 260, 508, 512, 516])
@pytest.mark.parametrize("F,B,f_range", [(230, 200, None), (40, 200, None), (9000, 300, None), (230, 200, (1, 117))])
def test_both_sides_in_one_pass_match_the_plain_statement(d, F, B, f_range):
    """Widths at which the groups of warps change, one group per row and several rows per draw, a range of the features."""
    k = 6
    cpu = _case(d, F, B, k, seed=d + F)
    if F == 40:  # all rows shared by a CTA, lists of 32 and a few more entries with gaps
        cpu["idx"][:, 1:] = torch.arange(B).unsqueeze(1) % 34 + torch.arange(1, k)
    if F == 9000:
        cpu["idx"][0::3] = -1
    gpu = {n: t.clone().to(DEV) for n, t in cpu.items()}
    lo = f_range[0] if f_range else 0

    def run(t, step):
        groups = K.FeatureGroups(F, B * k, t["idx"].device).build(t["idx"])
        K.sparse_grad_adam(groups, t["act"], t["dact"], t["x"], t["dx"], t["WD"], t["mD"][lo:], t["vD"][lo:], t["WD16"], t["WE"], t["mE"][lo:], t["vE"][lo:],
                           t["WE16"], t["b"], t["mb"][lo:], t["vb"][lo:], t["n"], t["gsq"].add_(0.5) if F == 230 else None, None, 1e-3, 0.9, 0.999, 1e-8,
                           step, True, f_range, state_f0=lo, extra=(t["row_of"], t["xD"], t["xE"], t["xb"]) if F != 40 else None,
                           wd_self_scale=t["scale"] if F != 40 else None, dact_mode=1)  # fmt: skip
        return groups

    for step in (1, 2):
        run(cpu, step)
        groups = run(gpu, step)
        K.check_status(torch.device(DEV))
        assert groups.sched.tolist() == [0, 0]  # ready for the next launch
    _compare(cpu, gpu, ["dact", "WD", "mD", "vD", "WE", "mE", "vE", "b", "mb", "vb", "n"], d)
    for n, m in (("WD16", "WD"), ("WE16", "WE")):
        assert torch.equal(gpu[n].float(), gpu[m].to(torch.bfloat16).float())


@pytest.mark.parametrize("d", [64, 512])
def test_one_pass_rows_whose_copies_were_not_waited_for_stay_as_they_are(d):
    test_rows_whose_copies_were_not_waited_for_stay_as_they_are(d, "both", 1)


@pytest.mark.parametrize("d", [64, 768, 1160])
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("L,F", [(1, 230), (3, 230), (4, 41)])
def test_encoder_sides_of_several_layers_in_one_launch(d, shared, L, F):
    """Layers with entries of their own and layers that share them, with lists long enough to be shared by a CTA in more than one layer."""
    B, k, g = 200, 6, torch.Generator().manual_seed(d + L)
    n = F if shared else L * F
    idx = torch.randint(0, n, (B, k), generator=g).to(torch.int32)
    idx[:, 0] = 3
    idx[:150, 1] = n - 2  # (the last layer's, or every layer's)
    idx[5, 2:] = -1
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    cpu = dict(idx=idx, dact=r(B, k), x=r(L, B, d).to(torch.bfloat16), W=r(L, F, d), b=r(L, F), S=torch.zeros(L, F, d, dtype=torch.bfloat16))
    for name, shape in (("m", (L, F, d)), ("v", (L, F, d)), ("mb", (L, F)), ("vb", (L, F))):
        cpu[name] = torch.rand(*shape, generator=g) * 0.01
    gpu = {n_: t.clone().to(DEV) for n_, t in cpu.items()}
    for t in (cpu, gpu):
        for step in (1, 2):
            groups = K.FeatureGroups(n, B * k, t["idx"].device).build(t["idx"])
            K.layers_encoder_adam(groups, t["dact"], t["dact"], t["x"], t["W"], t["m"], t["v"], t["S"], t["b"], t["mb"], t["vb"], shared, 1e-3, 0.9, 0.999, 1e-8, step)
    K.check_status(torch.device(DEV))
    assert int(groups.heavy[0]) == 2 and groups.sched.tolist() == [0, 0]
    _compare(cpu, gpu, ["W", "m", "v", "b", "mb", "vb"], d)
    assert torch.equal(gpu["S"].float(), gpu["W"].to(torch.bfloat16).float())


@pytest.mark.parametrize("d", [132, 768, 1160, 4100, 8192])
def test_long_lists_are_cut_evenly(d):
    """Lists just long enough to be shared, of one entry more or less than whole pieces of 32 for every group, and of every token."""
    B, F, g = 1300, 60, torch.Generator().manual_seed(d)
    lengths = [65, 66, 127, 479, 480, 481, 639, 640, 641, 769, 1281, 1300]
    idx = torch.full((B, len(lengths)), -1, dtype=torch.int32)
    for i, n in enumerate(lengths):
        idx[torch.randperm(B, generator=g)[:n], i] = 3 * i
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    cpu = dict(idx=idx, act=r(*idx.shape), dact=torch.zeros(idx.shape), x=r(B, d).to(torch.bfloat16), dx=r(B, d).to(torch.bfloat16), n=torch.zeros(F))
    for s in "DE":
        cpu |= {"W" + s: r(F, d), "S" + s: torch.zeros(F, d, dtype=torch.bfloat16), "m" + s: r(F, d) * 0.01, "v" + s: torch.rand(F, d, generator=g) + 1}
    cpu |= {"b": r(F), "mb": torch.zeros(F), "vb": torch.ones(F)}
    gpu = {n: t.clone().to(DEV) for n, t in cpu.items()}
    for t in (cpu, gpu):
        groups = K.FeatureGroups(F, idx.numel(), t["idx"].device).build(t["idx"])
        K.sparse_grad_adam(groups, t["act"], t["dact"], t["x"], t["dx"], t["WD"], t["mD"], t["vD"], t["SD"], t["WE"], t["mE"], t["vE"], t["SE"], t["b"], t["mb"],
                           t["vb"], t["n"], None, None, 1e-3, 0.9, 0.999, 1e-8, 1, True, dact_mode=1)  # fmt: skip
    K.check_status(torch.device(DEV))
    assert int(groups.heavy[0]) == len(lengths)
    # code gradients: d products of order one, added up in another order. Encoder moments: 0.1 of a sum of up to 1300 products of order sqrt(d), each
    # addition rounding a partial sum of about sqrt(1300 d); decoder moments the same with d = 1.
    assert torch.allclose(gpu["dact"].cpu(), cpu["dact"], atol=2**-24 * d * 4, rtol=1e-4)
    for n, scale in (("mD", 1.0), ("mE", d**0.5)):
        atol = 0.1 * 2**-24 * 1300 * 1300**0.5 * scale + 1e-6
        assert torch.allclose(gpu[n].cpu(), cpu[n], atol=atol, rtol=1e-4), (n, float((gpu[n].cpu() - cpu[n]).abs().max()))
    assert torch.allclose(gpu["mb"].cpu(), cpu["mb"], atol=0.1 * 2**-24 * 1300 * (1300 * d) ** 0.5, rtol=1e-4)


@pytest.mark.parametrize("d", [4, 64, 128, 132, 256, 260, 512])
@pytest.mark.parametrize("B", [1000, 1024, 1025])
def test_long_lists_in_one_pass(d, B):
    """Whole pieces of 32 for each of 8, 15 and 16 groups and one entry more or less, and a list of every token: the longest that two warps a row take in
    one pass, and the first that they leave to the other kernel."""
    g = torch.Generator().manual_seed(d)
    lengths = [65, 127, 255, 256, 257, 479, 480, 481, 511, 512, 513, 769, B]
    F, idx = 3 * len(lengths), torch.full((B, len(lengths)), -1, dtype=torch.int32)
    for i, n in enumerate(lengths):
        idx[torch.randperm(B, generator=g)[:n], i] = 3 * i
    idx[5, idx[5] < 0] = 1  # (a short list)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    cpu = dict(idx=idx, act=r(*idx.shape), dact=torch.zeros(idx.shape), x=r(B, d).to(torch.bfloat16), dx=r(B, d).to(torch.bfloat16), n=torch.zeros(F))
    for s in "DE":
        cpu |= {"W" + s: r(F, d), "S" + s: torch.zeros(F, d, dtype=torch.bfloat16), "m" + s: r(F, d) * 0.01, "v" + s: torch.rand(F, d, generator=g) + 1}
    cpu |= {"b": r(F), "mb": torch.zeros(F), "vb": torch.ones(F)}
    gpu = {n: t.clone().to(DEV) for n, t in cpu.items()}
    for t in (cpu, gpu):
        groups = K.FeatureGroups(F, idx.numel(), t["idx"].device).build(t["idx"])
        K.sparse_grad_adam(groups, t["act"], t["dact"], t["x"], t["dx"], t["WD"], t["mD"], t["vD"], t["SD"], t["WE"], t["mE"], t["vE"], t["SE"], t["b"], t["mb"],
                           t["vb"], t["n"], None, None, 1e-3, 0.9, 0.999, 1e-8, 1, True, dact_mode=1)  # fmt: skip
    K.check_status(torch.device(DEV))
    assert int(groups.heavy[0]) == len(lengths) and groups.sched.tolist() == [0, 0]
    # code gradients: d products of order one, added up in another order. Encoder moments: 0.1 of a sum of up to B products of order sqrt(d), each
    # addition rounding a partial sum of about sqrt(B d); decoder moments the same with d = 1.
    assert torch.allclose(gpu["dact"].cpu(), cpu["dact"], atol=2**-24 * d * 4, rtol=1e-4)
    for n, scale in (("mD", 1.0), ("mE", d**0.5), ("mb", d**0.5)):
        atol = 0.1 * 2**-24 * B * B**0.5 * scale + 1e-6
        assert torch.allclose(gpu[n].cpu(), cpu[n], atol=atol, rtol=1e-4), (n, float((gpu[n].cpu() - cpu[n]).abs().max()))
    assert torch.equal(gpu["SD"].float(), gpu["WD"].to(torch.bfloat16).float()) and torch.equal(gpu["SE"].float(), gpu["WE"].to(torch.bfloat16).float())
    assert torch.allclose(gpu["n"], gpu["WD"].norm(dim=1), rtol=1e-5)


@pytest.mark.parametrize("d", [128, 512])
def test_popular_features_cost_no_more_than_a_pass_per_side(d):
    """Popular features beside rare ones take no longer than where both sides are one after the other (which a gradient norm asks for). One CTA had the
    longest list to itself for 1.7 times as long at 512."""
    F, B, k, g = 8 * d, 4096, 32, torch.Generator(device=DEV).manual_seed(d)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    idx = torch.multinomial((1 / (torch.arange(F, device=DEV) + 5.0)).repeat(B, 1), k, generator=g).int()
    act, x, dx = r(B, k).abs(), r(B, d).to(torch.bfloat16), r(B, d).to(torch.bfloat16)
    WD, WE, vD, vE = r(F, d), r(F, d), r(F, d).abs() + 1, r(F, d).abs() + 1
    mD, mE, b, mb, vb, norm = (torch.zeros(*s, device=DEV) for s in ((F, d), (F, d), (F,), (F,), (F,), (F,)))
    SD, SE, dact, norm_sq, best = WD.to(torch.bfloat16), WE.to(torch.bfloat16), torch.empty_like(act), torch.zeros(1, device=DEV), [1e9, 1e9]
    groups = K.FeatureGroups(F, B * k, torch.device(DEV)).build(idx)
    for _ in range(12):
        for i in range(2):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda._sleep(100000)  # (the launch is on its way when the first event is)
            start.record()
            K.sparse_grad_adam(groups, act, dact, x, dx, WD, mD, vD, SD, WE, mE, vE, SE, b, mb, vb, norm, None, norm_sq if i else None, 1e-4, 0.9, 0.999, 1e-8, 1,
                               True, dact_mode=1)  # fmt: skip
            end.record()
            end.synchronize()
            best[i] = min(best[i], start.elapsed_time(end))
    K.check_status(torch.device(DEV))
    assert best[0] < 1.15 * best[1], best
