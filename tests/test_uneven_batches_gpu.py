"""Texts whose symbols depend on the ones before, and texts of which most stand several times: their suffixes lie unevenly in a batch of the local sort, and it orders them all the same (CSA_DEBUG tells how many
batches went where). Arrays byte for byte against the oracle's, large ones by the validator."""
import re

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


def _zipf(rng, size):
    return np.minimum(rng.zipf(1.3, size), 50257)


def _dependent(n, share, seed, successors=32):
    """A share of the symbols is drawn from 32 successors of the one before."""
    rng = np.random.default_rng(seed)
    lanes = 512 if n < 4_000_000 else 1 << 16
    out = _zipf(rng, (-(-n // lanes), lanes))
    table = _zipf(rng, (50258, successors))
    for s in range(1, len(out)):
        out[s] = np.where(rng.random(lanes) < share, table[out[s - 1], rng.integers(0, successors, lanes)], out[s])
    return out.T.ravel()[:n]


def _copies(n, copies, seed, length=500):
    """Passages that stand `copies` times each, over three quarters of the text."""
    rng = np.random.default_rng(seed)
    T = _zipf(rng, n)
    places = rng.permutation(n // length)[:3 * (n // length) // 4]
    for k in range(0, len(places) - copies + 1, copies):
        passage = _zipf(rng, length)
        for p in places[k:k + copies]:
            T[p * length:(p + 1) * length] = passage
    return T


def _build(ctx, T, monkeypatch, capfd):
    from cascade_b200 import api
    monkeypatch.setenv("CSA_DEBUG", "1")
    n = len(T)
    Td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, T.dtype)]).astype(np.uint16).view(np.int16)).cuda().view(torch.uint16)
    sa, _ = api.build_sa(ctx, Td, n, 8)
    m = re.search(r"(\d+) of (\d+) batches crowded, (\d+) runs left, (\d+) of (\d+) first", capfd.readouterr().err)
    crowded, batches, left, uneven, tried = map(int, m.groups())
    return Td, sa, dict(crowded=crowded, batches=batches, left=left, uneven=uneven, tried=tried)


def _check(oracle, T, sa):
    n = len(T)
    assert np.array_equal(sa[:5 * n].cpu().numpy(), oracle.build_sa40(T.astype(np.uint16))[:5 * n])


# one split, two splits with one batch a block, several batches a block
@pytest.mark.parametrize("n", [100_003, 300_000, 2_500_003])
@pytest.mark.parametrize("share", [0.1, 0.3, 0.6, 0.9])
def test_symbols_that_depend_on_the_one_before(ctx, oracle, monkeypatch, capfd, n, share):
    T = _dependent(n, share, n)
    _, sa, at = _build(ctx, T, monkeypatch, capfd)
    _check(oracle, T, sa)
    if n >= 300_000 and share >= 0.3:           # of one block in eight
        assert at["uneven"] > 0, "even batches: nothing is shown"
    if share < 0.9 and n > 1 << 21:     # texts of one split leave them all to the last kernel; children of more suffixes than a batch holds, some sixty of 2.5e6, go to it too, and where there are any, batches beside them until it has 148
        assert at["crowded"] + at["left"] < at["batches"] / 4 + 148 < at["batches"]


@pytest.mark.parametrize("copies", [2, 3, 5, 8, 15, 16, 17, 40, 60, 300])
@pytest.mark.parametrize("n", [200_001, 2_300_003])
def test_passages_that_stand_several_times(ctx, oracle, monkeypatch, capfd, n, copies):
    T = _copies(n, copies, n + copies)
    _, sa, at = _build(ctx, T, monkeypatch, capfd)
    _check(oracle, T, sa)
    if copies <= 3 and n > 1 << 21:
        assert at["crowded"] + at["left"] < at["batches"] / 4 + 148 < at["batches"]
    if copies == 60 and n > 2_000_000:
        assert at["crowded"] > at["batches"] / 2, "not left for its copies"


@pytest.mark.parametrize("kind", ["dependent", "copies", "mixed"])
def test_blocks_of_several_batches(ctx, monkeypatch, capfd, kind):
    """More batches than the local sort has blocks; mixed: even, uneven and copied stretches by turns."""
    from cascade_b200 import api
    n = 24_000_001
    if kind == "dependent":
        T = _dependent(n, 0.3, 7)
    elif kind == "copies":
        T = _copies(n, 4, 8, 3000)
    else:
        T = np.concatenate([_dependent(n // 3, 0.5, 9), _copies(n // 3, 50, 10), _zipf(np.random.default_rng(11), n - 2 * (n // 3))])
    Td, sa, at = _build(ctx, T, monkeypatch, capfd)
    assert at["batches"] > 3552 or kind == "mixed"
    assert api.validate_sa(ctx, Td, n, sa)["ok"]


# the smallest and the largest batches, and slots that begin at each place of a group of four: few symbols, so that children hold from nothing to more than a batch
@pytest.mark.parametrize("n", [16_385, 17_001, 30_002, 50_003, 65_536, 131_071])
@pytest.mark.parametrize("symbols", [3, 20, 150, 4000])
def test_short_texts_of_few_symbols_that_depend(ctx, oracle, monkeypatch, capfd, n, symbols):
    T = _dependent(n, 0.7, n + symbols, 4) % symbols
    _, sa, _ = _build(ctx, T, monkeypatch, capfd)
    _check(oracle, T, sa)


# the first and the last sizes of plans of two splits: parents and children double at 1537 suffixes a child, from 2^26 on at 2049; children are the smallest behind such a size and the largest before it
@pytest.mark.parametrize("n", [12_591_103, 12_591_104, 25_182_208, 50_364_415, 50_364_416, (1 << 26) - 1, 1 << 26, 2049 << 15])
def test_at_the_edges_of_the_plans(ctx, n):
    from cascade_b200 import api
    g = torch.Generator(device="cuda").manual_seed(n)
    steps = 512
    lanes = -(-n // steps)

    def zipf(*shape):
        u = torch.rand(shape, device="cuda", generator=g, dtype=torch.float64).clamp_(min=1e-12)
        return u.pow_(-1 / 0.3).clamp_(max=50257).to(torch.int64)

    table, out = zipf(50258, 32), torch.empty((steps, lanes), dtype=torch.int16, device="cuda")
    now = zipf(lanes)
    for s in range(steps):
        out[s] = now.to(torch.int16)
        followed = torch.rand(lanes, device="cuda", generator=g) < 0.5
        now = torch.where(followed, table[now, torch.randint(0, 32, (lanes,), device="cuda", generator=g)], zipf(lanes))
    T = torch.zeros(n + api.TEXT_PAD, dtype=torch.int16, device="cuda")
    T[:n] = out.t().reshape(-1)[:n]
    T = T.view(torch.uint16)
    sa, _ = api.build_sa(ctx, T, n, 64)
    assert api.validate_sa(ctx, T, n, sa)["ok"]


# blocks of one batch each, the last one of a block, whose tied records are fewer or more than a block keeps (1024 of some 2900): symbols all as frequent, so that bins are small
@pytest.mark.parametrize("share", [0.2, 0.3, 0.35, 0.4, 0.5])
def test_ties_of_a_blocks_last_batch(ctx, monkeypatch, capfd, share):
    from cascade_b200 import api
    n = 6_000_011
    rng = np.random.default_rng(int(100 * share))
    pairs = np.repeat(rng.integers(0, 50000, (int(n * share) // 46, 23)), 2, axis=0)
    rng.shuffle(pairs)
    T = np.concatenate([rng.integers(0, 50000, n - pairs.size), pairs.ravel()])
    Td, sa, at = _build(ctx, T, monkeypatch, capfd)
    assert at["batches"] < 3552 and api.validate_sa(ctx, Td, n, sa)["ok"]
