"""The launch at the end of a step: column sums of bf16 matrices as bias gradients, Adam on the biases, and the mean loss."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

DEVICES = [pytest.param("cuda", marks=pytest.mark.gpu), "cpu"]
HYPER = (1e-2, 0.9, 0.999, 1e-8)


def _rand(dev, *shape, seed=0):
    return torch.randn(*shape, device=dev, generator=torch.Generator(device=dev).manual_seed(seed))


def _ref(p, m, v, g, step):
    p, m, v = p.double(), m.double(), v.double()
    K.ref_adam(p, g.double(), m, v, *HYPER, step)
    return p, m, v


# one row, a row block and one more row, no multiple of anything; 8 columns, a column block and a bit, several matrices, 18 of them;
# the most rows whose partial sums are added up one by one, one more, and as many row blocks as there can be
@pytest.mark.parametrize("dev", DEVICES)
@pytest.mark.parametrize("rows,widths", [(1, [8]), (64, [256]), (65, [264, 8]), (3001, [768, 40, 2312]), (700, [64] * 18), (40, [12]), (4096, [8]), (4097, [264]), (33000, [72, 8])])
def test_bias_update(dev, rows, widths):
    mats = [_rand(dev, rows, w, seed=i).to(torch.bfloat16) for i, w in enumerate(widths)]
    params = [_rand(dev, w, seed=50 + i) for i, w in enumerate(widths)]
    moments = [(torch.zeros(w, device=dev), torch.zeros(w, device=dev)) for w in widths]
    want = [(p.clone(), m.clone(), v.clone()) for p, (m, v) in zip(params, moments)]
    loss, loss2, weight = torch.zeros(1, device=dev), torch.zeros(1, device=dev), torch.rand(rows, device=dev)
    update = K.BiasUpdate(widths, torch.device(dev))
    for step in range(1, 4):  # (the arrival counters serve every step)
        loss.fill_(7.5)
        loss2.fill_(0.5)
        mean, part = update(mats, params, moments, *HYPER, step, loss, loss2, weight, 0.5)
        den = float(weight.double().sum()) * 0.5
        assert float(mean) == pytest.approx(8.0 / den, rel=1e-5) and float(part) == pytest.approx(0.5 / den, rel=1e-5)
        assert float(loss) == 0.0 and float(loss2) == 0.0
        loss.fill_(3.0)
        want = [_ref(*w, a.double().sum(0), step) for w, a in zip(want, mats)]
    assert float(update([], [], [], *HYPER, 1, loss, loss_den=4.0)) == 0.75 and float(loss) == 0.0
    for p, (m, v), (wp, wm, wv), a in zip(params, moments, want, mats):
        # a sum of `rows` terms in fp32; Adam turns a gradient's sign, and rounding alone may decide the sign of a sum near zero
        err = rows * 2.0**-23 * a.double().abs().sum(0)
        sure = a.double().sum(0).abs() > 8 * err
        assert bool(((m.double() - wm).abs() <= 1e-5 * wm.abs() + err).all())
        assert torch.allclose(p.double()[sure], wp[sure], rtol=1e-4, atol=1e-5)


@pytest.mark.gpu
def test_many_rows_of_few_columns_take_no_longer_than_separate_launches():
    rows, d = 262144, 128
    a, p, m, v, loss = _rand("cuda", rows, d).to(torch.bfloat16), *(torch.zeros(d, device="cuda") for _ in range(3)), torch.zeros(1, device="cuda")
    update, best = K.BiasUpdate([d], torch.device("cuda")), [1e9, 1e9]

    def separate():
        loss.zero_()
        K.adam_flat(p, K.colsum_bf16(a), m, v, *HYPER, 1)

    for _ in range(8):
        for i, fn in enumerate((separate, lambda: update([a], [p], [(m, v)], *HYPER, 1, loss))):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            fn()
            end.record()
            end.synchronize()
            best[i] = min(best[i], start.elapsed_time(end))
    assert best[1] < 1.5 * best[0], best  # (with 64 row blocks: four times as long)
