"""The resident build at the edges of its kernels' tiles and of its dispatch (one split or two, small and wide tiles), and on
texts that take its rarer paths: children that do not fit a block, groups of more than 256 tied suffixes, bins with many
records, suffixes that end inside the symbols compared. Each array byte for byte against the oracle's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from cascade_b200 import api
    c = api.Context(0)
    yield c
    c.close()


def _check(ctx, oracle, T):
    from cascade_b200 import api
    T = np.ascontiguousarray(T, dtype=np.uint16)
    n = len(T)
    Td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    sa, st = api.build_sa(ctx, Td, n, 8)
    assert np.array_equal(sa[:5 * n].cpu().numpy(), oracle.build_sa40(T)[:5 * n])
    return st


def _zipf(n, seed, sigma=50257):
    rng = np.random.default_rng(seed)
    return np.minimum(rng.zipf(1.2, n), sigma).astype(np.uint16)


# tile of 128 threads: 1984 positions; child: 2048 suffixes; batch of the local sort: 8192; window of a list: 1792 + 256;
# second split above 2^21, wide tiles (8128 positions) from 2^19 on
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 1983, 1984, 1985, 2047, 2048, 2049, 3968, 3969, 4096, 4097, 8191, 8192, 8193, 16385, (1 << 21) - 1, 1 << 21, (1 << 21) + 1,
                               (1 << 22) - 1, (1 << 22) + 1])
def test_sizes_at_the_edges(ctx, oracle, n):
    _check(ctx, oracle, _zipf(n, n))


@pytest.mark.parametrize("n", [257, 1793, 2049, 8193, 70_001, 2_200_000])
@pytest.mark.parametrize("kind", ["one", "two", "period", "phrase", "stretch", "zeros_at_the_end", "copies", "phrase_of_thousands", "wide"])
def test_texts_of_the_rarer_paths(ctx, oracle, n, kind):
    rng = np.random.default_rng(n)
    if kind == "one":                   # one group of everything, halved by every generation
        T = np.full(min(n, 70_001), 7)
    elif kind == "two":
        T = rng.integers(0, 2, n) * 9
    elif kind == "period":              # a few huge groups
        T = np.resize(rng.integers(0, 5, 7), min(n, 70_001))
    elif kind == "phrase":              # a phrase of 12 symbols every 30: groups of thousands, and bins with as many records
        T = rng.integers(0, 60000, n)
        for k in range(12):
            T[k + 5::30] = 1000 + k
    elif kind == "phrase_of_thousands":     # at 2.2 million a child of some 6300 suffixes: for the larger blocks of the local sort alone
        T = rng.integers(0, 60000, n)
        for k in range(6):
            T[k + 5::350][:len(T) // 350] = 1000 + k
    elif kind == "stretch":             # copies of a long stretch: groups below and above 256 members, many generations
        T = rng.integers(0, 3000, n)
        L = max(8, n // 700)
        for a in range(0, n - L, 2 * L):
            T[a:a + L] = T[:L]
    elif kind == "zeros_at_the_end":    # suffixes that differ from others by their end alone
        T = rng.integers(0, 3, n)
        T[-min(n, 300):] = 0
    elif kind == "copies":              # near-duplicate documents of an odd length: nearly all suffixes tied, in groups that mostly agree
        base = rng.integers(0, 200, (5, 331))
        T = base[rng.integers(0, 5, n // 331 + 1)].ravel()[:n].copy()
        T[rng.random(n) < 0.004] = 60000
    else:
        T = rng.integers(0, 65536, n)
    st = _check(ctx, oracle, T)
    assert st.n == len(T) and 1 <= st.partitions <= 8 and 0 < st.max_partition <= len(T)


@pytest.mark.parametrize("shared", [6, 30, 90])
@pytest.mark.parametrize("spread", [1, 40])
def test_groups_about_as_large_as_the_small_ones_may_be(ctx, oracle, shared, spread):
    """Phrases that begin alike and then fall apart into groups of 1 to 2049 members, around the 256 up to which a group is small, at any place
    of a tile of the list: most are found in one large group first, and the stretch that they share is longer or shorter than what is
    compared in the text."""
    rng = np.random.default_rng(shared + spread)
    sizes = [1, 2, 31, 32, 33, 254, 255, 256, 257, 258, 511, 512, 513, 2047, 2048, 2049] + [int(x) for x in rng.integers(200, 300, spread)]
    begin = rng.integers(1, 60000, shared)
    pieces = []
    for c in sizes:
        end = rng.integers(1, 60000, 5)
        pieces += [np.concatenate([begin, end, rng.integers(1, 60000, int(rng.integers(1, 4)))]) for _ in range(c)]
    rng.shuffle(pieces)
    st = _check(ctx, oracle, np.concatenate(pieces))
    assert st.generations >= 2, "no group was ranked"


@pytest.mark.parametrize("n", [300, 5000, 70_001])
def test_nothing_but_zeros_and_zeros_behind_a_text(ctx, oracle, n):
    """The padding behind a text is zeros as well: large groups whose members end inside the symbols that they share."""
    _check(ctx, oracle, np.zeros(n))
    T = np.random.default_rng(n).integers(0, 2, n)
    T[n // 2:] = 0
    _check(ctx, oracle, T)


def _pairs_text(n, medium, oversize, seed):
    """Random symbols, and pairs of symbols that stand together many times: a child of 4097 to 8192 suffixes for each of the `medium`
    pairs, one of more than 8192 for each of the `oversize` ones, spread over the whole array."""
    rng = np.random.default_rng(seed)
    T = rng.integers(0, 65000, n, dtype=np.uint16)
    sizes = np.concatenate([rng.integers(4300, 7500, medium), rng.integers(8600, 9500, oversize)])
    rng.shuffle(sizes)
    slots = 2 * rng.permutation((n - 2) // 2)[:sizes.sum()]
    which = np.repeat(np.arange(len(sizes)), sizes)
    T[slots] = 100 + 255 * which
    T[slots + 1] = 101 + 255 * which
    return T


def test_blocks_that_go_on_behind_a_child_left_to_others(ctx, oracle):
    """More chunks of the local sort than blocks (4736), so that blocks take two or three: chunks that end in a child too large for the block
    stand among their first, middle and last ones. Resident, and as one part straight from the text."""
    from cascade_b200 import api
    T = _pairs_text(21_000_003, 230, 24, 5)
    n = len(T)
    want = oracle.build_sa40(T)[:5 * n]
    Tp = np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)])
    Td = torch.from_numpy(Tp.view(np.int16)).cuda().view(torch.uint16)
    for _ in range(3):
        sa, st = api.build_sa(ctx, Td, n, 8)
        assert np.array_equal(sa[:5 * n].cpu().numpy(), want)
        assert st.sort_passes > 2, "no child went through the radix sort"
    for _ in range(3):
        sa, st = api.build_sa_streamed(ctx, Tp, n, 8)
        assert np.array_equal(sa[:5 * n], want)
        assert st.sort_passes > 2 and st.host_parts == 0, "not straight from the text, or no child went through the radix sort"


def _held_by_a_build(T):
    """Device memory that a new context holds after one build, and the build's statistics."""
    from cascade_b200 import api
    n = len(T)
    Td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    out = torch.zeros(5 * n + api.SA_PAD_BYTES, dtype=torch.uint8, device="cuda")
    held = 0
    for _ in range(2):              # the first build loads the kernels' code, too
        torch.cuda.empty_cache()
        c = api.Context(0)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        _, st = api.build_sa(c, Td, n, 8, out=out)
        torch.cuda.synchronize()
        held = free - torch.cuda.mem_get_info()[0]
        c.close()
    return held, st


def test_a_few_oversize_children_take_no_ranking_memory():
    """20 bytes a suffix and a sixteenth of head-room, tables, and buffers for one suffix in 64: not the 16 bytes a suffix that ranks need."""
    T = _pairs_text(21_000_003, 230, 24, 5)
    held, st = _held_by_a_build(T)
    assert st.sort_passes > 2, "no child went through the radix sort"
    assert held < 24 * len(T), held / len(T)


def test_a_build_that_ranks_fits_what_it_says_it_needs(ctx):
    """With no more device memory free than csa_build_device_bytes, a text whose repeats need ranks is built: the first buffer's head-room is not
    taken from what the ranks need later."""
    from cascade_b200 import api
    n = 120_000_007
    piece = torch.randint(1, 60000, (1000,), dtype=torch.int32, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).to(torch.int16)
    Td = torch.zeros(n + api.TEXT_PAD, dtype=torch.int16, device="cuda")
    Td[:n] = piece.repeat(n // 1000 + 1)[:n]
    Td = Td.view(torch.uint16)
    out = torch.zeros(5 * n + api.SA_PAD_BYTES, dtype=torch.uint8, device="cuda")
    _held_by_a_build(np.resize(np.arange(1, 1000, dtype=np.uint16), 300_000))        # the kernels' code is on the device
    c = api.Context(0)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    need = c.L.csa_build_device_bytes(n, 8) + (16 << 20)
    rest = torch.empty(torch.cuda.mem_get_info()[0] - need, dtype=torch.uint8, device="cuda")
    _, st = api.build_sa(c, Td, n, 8, out=out)
    assert st.generations > 10, "no ranks were needed"
    c.close()
    del rest
    torch.cuda.empty_cache()
    assert api.validate_sa(ctx, Td, n, out)["ok"]


def test_repeats_of_two_thousand_million_symbols_above_2_31_positions(ctx):
    """A text of 2.26e9 symbols with a period of 1.5e8: its suffixes share up to 2.1e9 symbols, and a step of 61 * 2^25, the next after one that tells
    2.05e9 of them, no longer fits a sort key of two ranks."""
    from cascade_b200 import api
    n, period = 2_260_000_000, 150_000_000
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 130e9:
        pytest.skip("needs 130 GB of device memory")
    T = torch.zeros(n + api.TEXT_PAD, dtype=torch.int16, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(3)
    for at in range(0, period, 1 << 24):
        k = min(1 << 24, period - at)
        T[at:at + k] = torch.randint(-(1 << 15), 1 << 15, (k,), device="cuda", dtype=torch.int32, generator=g).to(torch.int16)
    at = period
    while at < n:               # of the text so far: always from a multiple of the period
        k = min(at, n - at)
        T[at:at + k] = T[:k]
        at += k
    T = T.view(torch.uint16)
    c = api.Context(0)
    out, st = api.build_sa(c, T, n, 8)
    c.close()
    assert st.generations > 20
    assert api.validate_sa(ctx, T, n, out)["ok"]
