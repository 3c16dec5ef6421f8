"""Large query batches, whose queries are dealt into slots by where they fall in the sample table, against the oracle and against the same
batch in pieces that are searched in their own order."""
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


def _index(ctx, T, stride, shift=0):
    """The array (host), and an index. shift: symbols by which the text's address misses a 16-byte boundary (bytes for the array: four times as many)."""
    from cascade_b200 import api
    n = len(T)
    whole = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    sa40 = api.build_sa(ctx, whole, n)[0].cpu().numpy()
    td = torch.zeros(n + shift + api.TEXT_PAD, dtype=torch.int16, device="cuda")
    td[shift:shift + n] = torch.from_numpy(T.view(np.int16)).cuda()
    sd = torch.zeros(len(sa40) + 4 * shift, dtype=torch.uint8, device="cuda")
    sd[4 * shift:] = torch.from_numpy(np.ascontiguousarray(sa40)).cuda()
    return sa40, api.SuffixIndex(ctx, td.view(torch.uint16)[shift:], sd[4 * shift:], n, stride)


def _patterns(T, q, rng, longest):
    """Pieces of the text (some past its end), random symbols, zeros, empty ones: off, sym."""
    n = len(T)
    m = rng.integers(0, longest + 1, q)
    at = rng.integers(0, n, q)
    off = np.concatenate([[0], np.cumsum(m)]).astype(np.int64)
    within = np.arange(off[-1]) - np.repeat(off[:-1], m)
    source = np.repeat(at, m) + within
    sym = np.where(source < n, T[np.minimum(source, n - 1)], 0).astype(np.uint16)
    other = np.repeat(rng.integers(0, 4, q) == 0, m)
    sym = np.where(other, rng.integers(0, 400, len(sym)), sym).astype(np.uint16)
    return off, sym


def _find(idx, off, sym, q, first=0):
    o = torch.from_numpy(off[first:first + q + 1].copy()).cuda()
    s = torch.from_numpy(np.concatenate([sym[off[first]:off[first + q]], np.zeros(8, np.uint16)]).view(np.int16)).cuda()
    return idx.find(o, s, q).cpu().numpy().view(np.uint64)


# from 2^19 queries and 2^22 keys in the table on; the directory has 4096 keys
@pytest.mark.parametrize("n,stride,q,longest", [(1 << 22, 1, 1 << 19, 16), ((1 << 22) + 1, 1, (1 << 19) + 1, 5), (((1 << 22) + 3) * 3 - 1, 3, 600_001, 40)])
@pytest.mark.parametrize("shift", [0, 3])
def test_large_batches_against_the_oracle(ctx, oracle, n, stride, q, longest, shift):
    rng = np.random.default_rng(n + q)
    T = np.minimum(rng.zipf(1.3, n), 350).astype(np.uint16)
    T[n // 2:n // 2 + 3000] = 7             # keys that many entries of the directory share
    T[n - 20:] = 0                          # suffixes that end inside what looks equal to a pattern
    sa, idx = _index(ctx, T, stride, shift)
    off, sym = _patterns(T, q, rng, longest)
    launches = ctx.launches
    got = _find(idx, off, sym, q)
    assert ctx.launches == launches + 4, "not dealt"
    assert np.array_equal(got, oracle.find_batch(T, sa, off, sym))


def test_one_pattern_and_nothing_but_empty_ones(ctx, oracle):
    """All queries in one slot, before, inside and behind everything."""
    rng = np.random.default_rng(4)
    n, q = 1 << 22, 1 << 19
    T = rng.integers(5, 300, n).astype(np.uint16)
    sa, idx = _index(ctx, T, 1)
    for pattern in ([], [0], [65535, 1], [int(x) for x in T[100:103]], [int(x) for x in T[200:220]]):
        off = np.arange(q + 1, dtype=np.int64) * len(pattern)
        sym = np.tile(np.array(pattern, np.uint16), q)
        want = np.array(oracle.find_one(T, sa, np.array(pattern, np.uint16)), np.uint64)
        assert np.array_equal(_find(idx, off, sym, q).reshape(q, 2), np.tile(want, (q, 1))), pattern


def test_a_batch_of_more_than_one_share(ctx):
    """2^22 queries are dealt at a time; the rest of the batch starts at offsets and symbols further on. Against pieces that are searched in their own order."""
    rng = np.random.default_rng(9)
    n, q = 1 << 22, (1 << 22) + 40_001
    T = np.minimum(rng.zipf(1.3, n), 350).astype(np.uint16)
    _, idx = _index(ctx, T, 1)
    off, sym = _patterns(T, q, rng, 6)
    got = _find(idx, off, sym, q)
    step = 300_000
    for first in range(0, q, step):
        c = min(step, q - first)
        assert np.array_equal(got[2 * first:2 * (first + c)], _find(idx, off, sym, c, first)), first
