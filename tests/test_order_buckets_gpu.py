"""csa_sort_pairs of lists long enough that a bucket's words are ordered by threads' windows: buckets for each of the block's capacities, keys whose first bits tell them apart or do not,
equal ones, and keys uneven inside a bucket, against a stable comparison sort."""
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


# buckets of 525 records on average where the keys fill their range, of more where they fill a part: up to 2044, 2556 and 4092 a block, beyond them the larger blocks
@pytest.mark.parametrize("part", [1, 4, 6, 9])
@pytest.mark.parametrize("bits,value", [((0, 64), torch.int32), ((0, 32), torch.int32), ((5, 45), torch.int64)])
@pytest.mark.parametrize("kind", ["spread", "odd_place", "sorted", "pairs", "few_bits_behind", "heap_in_one"])
def test_long_lists(ctx, part, bits, value, kind):
    n, (b0, b1) = 4_300_001, bits
    g = torch.Generator(device="cuda").manual_seed(part)
    width = b1 - b0
    r = torch.randint(0, 1 << 62, (n + 1,), device="cuda", dtype=torch.int64, generator=g)
    keys = (r % ((1 << min(width, 62)) // part)) << (b0 + max(0, width - 62))
    if kind == "sorted":
        keys = torch.sort(keys).values
    elif kind == "pairs":                                   # every key twice or four times: equal ones stay in their order
        keys[n // 4: n // 2] = keys[: n // 2 - n // 4]
        keys = keys[torch.randperm(n + 1, device="cuda", generator=g)]
    elif kind == "few_bits_behind":                         # the first bits of a word are the same for many keys of a bucket, the last ones tell
        keys = (keys >> (b1 - 17) << (b1 - 17)) | ((r & 3) << b0)
    elif kind == "heap_in_one":                             # one value in some hundred places, and as many keys right behind it
        keys[:900] = keys[0]
        keys[900:1500] = keys[0] + (torch.arange(600, device="cuda") << b0)
    keys = keys[1:] if kind == "odd_place" else keys[:n].clone()          # an odd place starts on an odd 8-byte boundary
    _check(ctx, keys, torch.arange(n, device="cuda", dtype=value), b0, b1)


@pytest.mark.parametrize("part", [1, 6])
@pytest.mark.parametrize("bits,value", [((0, 64), torch.int32), ((0, 32), torch.int32), ((5, 45), torch.int64)])
@pytest.mark.parametrize("heaps", [280, 20_000])
def test_heaps_of_equal_keys(ctx, part, bits, value, heaps):
    """Buckets that turn out to be uneven, one in thirty and nearly all: the last are not tried once that is known."""
    n, (b0, b1) = 4_300_001, bits
    g = torch.Generator(device="cuda").manual_seed(part)
    keys = torch.randint(0, 1 << 31, (n,), device="cuda", dtype=torch.int64, generator=g) << 32
    keys += torch.randint(0, 1 << 32, (n,), device="cuda", dtype=torch.int64, generator=g)
    if part > 1 and b1 < 64:
        keys = (keys & ~((1 << b1) - 1)) | ((keys & ((1 << b1) - 1)) // 9 * part)
    keys[:40 * heaps] = keys[:heaps].repeat(40)
    _check(ctx, keys, torch.arange(n, device="cuda", dtype=value), b0, b1)


# buckets of 2441 records on average: the largest of the blocks where a word holds all of a key that is compared, the kernel before it where it does not or keys stand many times; of 4091: beyond both
@pytest.mark.parametrize("n", [40_000_003, (1 << 26) - 77])
@pytest.mark.parametrize("bits,value", [((0, 32), torch.int32), ((9, 41), torch.int64), ((0, 64), torch.int32)])
@pytest.mark.parametrize("kind", ["spread", "pairs", "eights"])
def test_the_longest_lists(ctx, n, bits, value, kind):
    g = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(-(1 << 62), 1 << 62, (n,), device="cuda", dtype=torch.int64, generator=g)
    if kind == "pairs":                 # two of a key here and there, which stay in their order
        keys[: n // 100] = keys[n // 2: n // 2 + n // 100]
    elif kind == "eights":
        keys = keys[torch.randint(0, n // 8, (n,), device="cuda", generator=g)]
    _check(ctx, keys, torch.arange(n, device="cuda", dtype=value), *bits)
