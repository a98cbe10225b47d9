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


@pytest.mark.parametrize("n", [65 * 3, 45056, 65 * 800])
def test_what_the_list_of_long_rows_held_does_not_matter(n):
    """The sort by itself with a list buffer that nobody zeroed and that has room for exactly the rows there can be, all of which are long; then the
    one-launch form with a counter after a list that filled its buffer."""
    F = n // 65 + 3
    flat = torch.arange(n, dtype=torch.int32, device="cuda") % (n // 65)
    new = lambda size: torch.full((size,), -(2**31) + 12345, dtype=torch.int32, device="cuda")  # noqa: E731
    places = torch.zeros(1, dtype=torch.int32, device="cuda")
    heavy = new(1 + n // 65)
    for counter in (None, places, None, places):
        counts, offsets, cursor, entries, sums = new(F), new(F + 1), new(F), new(n), new((F + 4095) // 4096)
        K._ext().csc_build(flat, F, counts, offsets, cursor, entries, sums, heavy, counter)
        want = torch.bincount(flat.long(), minlength=F)
        long_rows = torch.nonzero(want > K.HEAVY_ROW).flatten()
        assert torch.equal(counts.long(), want) and torch.equal(offsets[1:].long(), want.cumsum(0)) and int(places) == 0
        assert long_rows.numel() == n // 65 == int(heavy[0]) and torch.equal(heavy[1:].sort().values.long(), long_rows)
        assert torch.equal(flat[entries.long()], torch.repeat_interleave(torch.arange(F, dtype=torch.int32, device="cuda"), want))
