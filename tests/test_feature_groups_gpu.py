"""Grouping codes by feature around the limits of its kernels, with empty slots and features of every token."""

import pytest
import torch

from language_model_saes_b200.ops import sae_kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,k,F", [(1, 1, 1), (37, 3, 5), (512, 8, 256), (512, 16, 4097), (512, 16, 8192), (512, 16, 8193), (513, 16, 100), (1024, 32, 4096)])
def test_groups(B, k, F):
    g = torch.Generator().manual_seed(B + F)
    idx = torch.randint(-1, F, (B, k), generator=g).to(torch.int32)
    idx[:, 0] = F // 2
    groups = K.FeatureGroups(F, idx.numel(), torch.device("cuda"))
    for _ in range(2):  # (buffers are used again)
        groups.build(idx.cuda())
        counts = torch.bincount(idx[idx >= 0].long(), minlength=F)
        off = groups.offsets.cpu()
        assert torch.equal(groups.counts.cpu().long(), counts) and torch.equal(off.long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
        e = groups.entries.cpu()[: int(off[-1])].long()
        assert torch.equal(idx.reshape(-1)[e], torch.repeat_interleave(torch.arange(F, dtype=torch.int32), counts)) and e.unique().numel() == e.numel()
        heavy = groups.heavy.cpu()
        want = torch.nonzero(counts > K.HEAVY_ROW).flatten()
        assert int(heavy[0]) == want.numel() and torch.equal(heavy[1 : 1 + want.numel()].sort().values.long(), want)


# the most features that one scan launch takes, one more (three launches), and as many as twelve layers of 24576 have; a feature of every token in
# the last part of the scan
@pytest.mark.parametrize("F", [(1 << 17) - 1, 1 << 17, (1 << 17) + 1, 294912])
def test_long_dictionaries(F):
    g = torch.Generator().manual_seed(F)
    groups = K.FeatureGroups(F, 700 * 16, torch.device("cuda"))
    for B in (700, 150, 700):  # (buffers are used again)
        idx = torch.randint(-1, F, (B, 16), generator=g).to(torch.int32)
        idx[:, 0], idx[:, 1] = F - 1, F // 2
        groups.build(idx.cuda())
        counts = torch.bincount(idx[idx >= 0].long(), minlength=F)
        off = groups.offsets.cpu()
        assert torch.equal(groups.counts.cpu().long()[:F], counts) and torch.equal(off.long()[: F + 1], torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
        e = groups.entries.cpu()[: int(off[F])].long()
        assert torch.equal(idx.reshape(-1)[e], torch.repeat_interleave(torch.arange(F, dtype=torch.int32), counts)) and e.unique().numel() == e.numel()
        heavy, want = groups.heavy.cpu(), torch.nonzero(counts > K.HEAVY_ROW).flatten()
        assert want.numel() == 2 and int(heavy[0]) == 2 and torch.equal(heavy[1:3].sort().values.long(), want)


# one launch up to 45056 entries and 148 * 4096 features: both sides of the lines, blocks of 32 features and of 4096, tails of a vector and of a tile,
# all entries in one block's features, all in one feature, none, and an address that vectors cannot take
@pytest.mark.parametrize("n,F", [(0, 40), (3, 33), (4095, 33), (4097, 4736), (45055, 4737), (45056, 100), (45057, 100), (45056, 606208), (9000, 606209)])
def test_few_entries(n, F):
    g = torch.Generator().manual_seed(n + F)
    groups = K.FeatureGroups(F, 45057, torch.device("cuda"))
    spread, narrow = torch.randint(-1, F + 3, (n,), generator=g), torch.randint(max(0, F - 20), F, (n,), generator=g)
    for flat in (spread, narrow, torch.full((n,), F - 1), torch.full((n,), -1), spread):
        for shift in (0, 1):
            idx = torch.zeros(n + 1, dtype=torch.int32, device="cuda")[shift : shift + n].copy_(flat)
            groups.build(idx)
            valid = flat[(flat >= 0) & (flat < F)]
            counts = torch.bincount(valid, minlength=F)
            off = groups.offsets.cpu()
            assert torch.equal(groups.counts.cpu().long(), counts) and torch.equal(off.long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
            e = groups.entries.cpu()[: int(off[-1])].long()
            assert torch.equal(flat[e], torch.repeat_interleave(torch.arange(F), counts)) and e.unique().numel() == e.numel()
            heavy, want = groups.heavy.cpu(), torch.nonzero(counts > K.HEAVY_ROW).flatten()
            assert int(heavy[0]) == want.numel() and torch.equal(heavy[1 : 1 + want.numel()].sort().values.long(), want) and int(heavy[-1]) == 0
