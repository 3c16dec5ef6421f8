"""csa_sort_pairs where the records are split into buckets by their top bits and finished inside blocks: sizes around the edges of the choice
between one block, one split, two splits and digit passes, and keys whose buckets or bins are uneven, against a stable comparison sort."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from cascade_b200 import api
    c = api.Context(0)
    yield c
    c.close()


def _check(ctx, keys, vals, b0, b1):
    from cascade_b200 import api
    k0, v0 = keys.clone(), vals.clone()
    ko, vo = api.sort_pairs(ctx, keys, vals, b0, b1)
    mk = k0 ^ (-(1 << 63)) if b1 - b0 >= 64 else (k0 >> b0) & ((1 << (b1 - b0)) - 1)
    order = torch.sort(mk, stable=True).indices
    assert torch.equal(k0[order], ko)
    assert torch.equal(v0[order], vo)


def _random(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-(1 << 62), 1 << 62, (n,), device="cuda", dtype=torch.int64, generator=g) * 2 + (torch.arange(n, device="cuda") & 1)


# one block up to 8192; buckets of about 1024, in blocks of 2048, 4096 or 8192; one split up to 2^19, then two
@pytest.mark.parametrize("n", [2, 33, 2047, 2049, 8191, 8192, 8193, 16385, 262_144, (1 << 19) - 1, (1 << 19) + 1, 3_000_001])
@pytest.mark.parametrize("bits", [(0, 64), (0, 32), (5, 45)])
@pytest.mark.parametrize("value", [torch.int32, torch.int64])
def test_sizes_at_the_edges(ctx, n, bits, value):
    keys = _random(n + 1, n)[n & 1:][:n]          # odd sizes start on an odd 8-byte boundary
    _check(ctx, keys, torch.arange(n, device="cuda", dtype=value), *bits)


@pytest.mark.parametrize("n", [5000, 300_000, 2_000_003])
@pytest.mark.parametrize("kind", ["equal", "few", "low_bits_only", "one_large_bucket", "buckets_of_thousands", "few_keys_a_bucket", "equal_keys_in_a_bucket", "all_ones"])
def test_uneven_keys(ctx, n, kind):
    """Buckets too large for a block (all records then go through the digit passes), buckets of up to 8192, and bins of hundreds
    of records, which go through the network; the order of equal keys is the one they came in."""
    r = _random(n, n)
    index = torch.arange(n, device="cuda")
    if kind == "equal":
        keys = torch.full((n,), 0x1234_5678_9ABC_DEF0, device="cuda", dtype=torch.int64)
    elif kind == "few":
        keys = (r & 3) << 50
    elif kind == "low_bits_only":
        keys = r & 0xFFFFF
    elif kind == "one_large_bucket":
        keys = torch.where(index % 3 == 0, r & 0xFFFF, r)
    elif kind == "buckets_of_thousands":        # every key in one of n / 5000 places
        keys = (((r >> 8) & 0x7FFFFFFF) % max(1, n // 5000)) * ((1 << 62) // max(1, n // 5000)) + (r & 0xFFFF)
    elif kind == "few_keys_a_bucket":           # the bits behind the bucket's take three values
        keys = (r & ~0x0000_FFFF_FFFF_FFFF) | ((r >> 3) & 0xFFFF) % 3
    elif kind == "equal_keys_in_a_bucket":
        keys = r & ~0x0000_FFFF_FFFF_FFFF
    else:                                       # filler keys of a partial tile and of the network have all bits set
        keys = torch.where(index % 5 == 0, torch.full_like(r, -1), r)
    for bits in ((0, 64), (0, 40)):
        _check(ctx, keys.clone(), torch.arange(n, device="cuda", dtype=torch.int32), *bits)


# one block; buckets in blocks of 2048 to 8192; above 2^21 records a sample is looked at before the keys are counted
@pytest.mark.parametrize("n", [300, 4097, 8191, 8192, 262_144, 2_200_001])
@pytest.mark.parametrize("kind", ["a_run_a_key", "runs_that_differ_low", "top_bits_and_three_values", "two_far_bits", "one_odd_key"])
@pytest.mark.parametrize("value", [torch.int32, torch.int64])
def test_many_records_of_a_few_keys(ctx, n, kind, value):
    """Bins that hold hundreds of records: a block orders them by the digits in which its keys differ, equal keys as they came."""
    r = _random(n, n + 1)
    index = torch.arange(n, device="cuda")
    if kind == "a_run_a_key":                   # 300 records of every key, the keys spread evenly
        keys = (index // 300) * 0x1E37_79B9_7F4A_7C15
    elif kind == "runs_that_differ_low":        # the same with 8 low bits of their own
        keys = ((index % max(1, n // 300)) * 0x1E37_79B9_7F4A_7C15 & ~0xFF) | (r & 0xFF)
    elif kind == "top_bits_and_three_values":
        keys = (r & ~((1 << 49) - 1)) | ((r >> 3) & 0xFF) % 3
    elif kind == "two_far_bits":                # the lowest and the highest bit: no digit holds both
        keys = (r & 1) | (r & 2) << 62
    else:
        keys = torch.full_like(r, 0x0123_4567_89AB_CDEF)
        keys[n // 2] += 1 << 20
    for bits in ((0, 64), (1, 50)):
        _check(ctx, keys.clone(), torch.arange(n, device="cuda", dtype=value), *bits)


@pytest.mark.parametrize("n", [100_000, 3_000_001])
def test_which_way_the_keys_go(ctx, n):
    """By the launches: four of them look at the keys; then one or two splits and the buckets, or a pass for each digit that differs."""
    from cascade_b200 import api
    r, vals = _random(n, 3), torch.arange(n, device="cuda", dtype=torch.int32)
    splits = 1 if n <= 1 << 19 else 2

    def launches(keys):
        before = ctx.launches
        api.sort_pairs(ctx, keys, vals.clone())
        return ctx.launches - before - 4

    assert launches(r.clone()) == splits + 1
    assert launches(torch.full_like(r, 5)) == 0
    assert launches(r & 0xFF_FFFF) == 3
    assert launches(r & ~((1 << 56) - 1)) == 1
    assert launches(torch.where(vals % 2 == 0, r, torch.zeros_like(r))) == 8
