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


def _index(ctx, T, sa40, stride, shift=0):
    """shift: symbols by which the text's address misses a 16-byte boundary (bytes for the array: four times as many)."""
    from cascade_b200 import api
    n = len(T)
    td = torch.zeros(n + shift + api.TEXT_PAD, dtype=torch.int16, device="cuda")
    td[shift:shift + n] = torch.from_numpy(T.view(np.int16)).cuda()
    sd = torch.zeros(len(sa40) + 4 * shift, dtype=torch.uint8, device="cuda")
    sd[4 * shift:] = torch.from_numpy(np.ascontiguousarray(sa40)).cuda()
    return api.SuffixIndex(ctx, td.view(torch.uint16)[shift:], sd[4 * shift:], n, stride)


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


# from 32768 queries and 16384 keys in the table on; the directory has 4096 keys
@pytest.mark.parametrize("n,stride,q,longest", [(16_384, 1, 32_768, 16), (16_383, 1, 32_768, 16), (70_001, 1, 40_001, 5), (70_001, 4, 32_769, 40), (300_007, 7, 100_003, 16)])
@pytest.mark.parametrize("shift", [0, 3])
def test_large_batches_against_the_oracle(ctx, oracle, n, stride, q, longest, shift):
    rng = np.random.default_rng(n + q)
    T = np.minimum(rng.zipf(1.3, n), 350).astype(np.uint16)
    T[n // 2:n // 2 + 3000] = 7             # keys that many entries of the directory share
    T[n - 20:] = 0                          # suffixes that end inside what looks equal to a pattern
    sa = oracle.build_sa40(T)
    off, sym = _patterns(T, q, rng, longest)
    assert np.array_equal(_find(_index(ctx, T, sa, stride, shift), off, sym, q), oracle.find_batch(T, sa, off, sym))


def test_one_pattern_and_nothing_but_empty_ones(ctx, oracle):
    """All queries in one slot, before, inside and behind everything."""
    rng = np.random.default_rng(4)
    n, q = 50_000, 60_000
    T = rng.integers(5, 300, n).astype(np.uint16)
    sa = oracle.build_sa40(T)
    idx = _index(ctx, T, sa, 2)
    for pattern in ([], [0], [65535, 1], [int(x) for x in T[100:103]], [int(x) for x in T[200:220]]):
        off = np.arange(q + 1, dtype=np.int64) * len(pattern)
        sym = np.tile(np.array(pattern, np.uint16), q)
        want = np.array(oracle.find_one(T, sa, np.array(pattern, np.uint16)), np.uint64)
        assert np.array_equal(_find(idx, off, sym, q).reshape(q, 2), np.tile(want, (q, 1))), pattern


def test_a_batch_of_more_than_one_share(ctx, oracle):
    """2^22 queries are dealt at a time; the rest of the batch starts at offsets and symbols further on."""
    rng = np.random.default_rng(9)
    n, q = 60_000, (1 << 22) + 40_001
    T = np.minimum(rng.zipf(1.3, n), 350).astype(np.uint16)
    idx = _index(ctx, T, oracle.build_sa40(T), 3)
    off, sym = _patterns(T, q, rng, 6)
    got = _find(idx, off, sym, q)
    step = 30_000                           # searched in their own order
    for first in range(0, q, step * 7):
        c = min(step, q - first)
        assert np.array_equal(got[2 * first:2 * (first + c)], _find(idx, off, sym, c, first)), first
    c = 1000
    assert np.array_equal(got[2 * (q - c):], _find(idx, off, sym, c, q - c))
