"""Builds of texts whose tied groups lead to one another (from 2^22 tied suffixes on), each array checked exactly by csa_validate_sa."""
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


def _check(ctx, T):
    from cascade_b200 import api
    T = np.ascontiguousarray(T, dtype=np.uint16)
    n = len(T)
    Td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    sa, st = api.build_sa(ctx, Td, n, 8)
    v = api.validate_sa(ctx, Td, n, sa)
    assert v["ok"], v
    return st


@pytest.mark.parametrize("copies,mutate,cut", [(2, 0, 0), (3, 1e-5, 1), (40, 1e-3, 17), (250, 1e-3, 0), (40, 0.05, 3)])
def test_a_text_that_occurs_many_times(ctx, copies, mutate, cut):
    """Groups of 2 to 250: rows of followers as long as the text, rows that end where the copies differ, at every few symbols, and at the text's end."""
    rng = np.random.default_rng(copies)
    base = rng.integers(1, 60000, 5_200_000 // copies).astype(np.uint16)
    T = np.tile(base, copies)
    hit = rng.random(len(T)) < mutate
    T[hit] = rng.integers(1, 60000, int(hit.sum()))
    st = _check(ctx, T[:len(T) - cut])
    assert st.generations > 1


def test_documents_in_another_order_every_time(ctx):
    """Near-duplicate documents with separators, and some passages that stand in the text too often for a small group."""
    rng = np.random.default_rng(2)
    docs = [np.concatenate([[65535], np.minimum(rng.zipf(1.2, int(rng.integers(20, 4000))), 50000)]).astype(np.uint16) for _ in range(60)]
    T = np.concatenate([docs[int(k)] for k in rng.integers(0, 60, 3000)])[:5_500_001]
    hit = rng.random(len(T)) < 1e-3
    T[hit] = rng.integers(1, 60000, int(hit.sum()))
    _check(ctx, T)
    T[::20000] = 7
    for k in range(0, len(T) - 40, 19000):
        T[k:k + 30] = docs[0][1:31] if len(docs[0]) > 31 else 9
    _check(ctx, T)


@pytest.mark.parametrize("n", [(1 << 24) + 1, (1 << 25) + 12345])
def test_slots_sorted_into_buckets(ctx, n):
    """Above 2^24 suffixes the others' slots go through buckets by their top bits: a last bucket of one slot, and one that is partly there."""
    rng = np.random.default_rng(n)
    docs = rng.integers(1, 60000, (3000, 400)).astype(np.uint16)
    T = docs[rng.integers(0, 3000, n // 400 + 1)].reshape(-1)[:n]
    hit = rng.random(n) < 1e-3
    T[hit] = rng.integers(1, 60000, int(hit.sum()))
    _check(ctx, T)


@pytest.mark.parametrize("length", [6, 200])
def test_a_few_large_groups_beside_many_small_ones(ctx, length):
    """A passage that stands in the text 400 times: its groups are ranked first where that takes a few steps, else they stay large."""
    rng = np.random.default_rng(length)
    T = np.tile(rng.integers(1, 60000, 130_000).astype(np.uint16), 40)
    hit = rng.random(len(T)) < 1e-3
    T[hit] = rng.integers(1, 60000, int(hit.sum()))
    for k in rng.integers(0, len(T) - length, 400):
        T[k:k + length] = np.arange(1, length + 1)
    _check(ctx, T)


# ---- which way a text goes, as the build's own diagnostics (CSA_DEBUG) say it ----------------------------------------------------


def _way(ctx, T, capfd, monkeypatch):
    monkeypatch.setenv("CSA_DEBUG", "1")
    capfd.readouterr()
    _check(ctx, T)
    return capfd.readouterr().err


def _mutated(T, share, rng):
    T = T.copy()
    hit = rng.random(len(T)) < share
    T[hit] = rng.integers(1, 60000, int(hit.sum()))
    return T


def _phrases(n, length, times, rng):
    vocab = rng.integers(1, 60000, (n // (length * times), length)).astype(np.uint16)
    return vocab[rng.integers(0, len(vocab), n // length)].reshape(-1)


def test_near_duplicates_are_followed(ctx, capfd, monkeypatch):
    rng = np.random.default_rng(1)
    err = _way(ctx, _mutated(np.tile(rng.integers(1, 60000, 150_000).astype(np.uint16), 40), 1e-3, rng), capfd, monkeypatch)
    assert "are tied one symbol on" in err and "have a follower" in err and "large groups, h=" not in err and "generation" in err


def test_large_groups_are_ranked_ahead_and_the_others_followed(ctx, capfd, monkeypatch):
    """A passage of six symbols that stands in the text 400 times."""
    rng = np.random.default_rng(2)
    T = _mutated(np.tile(rng.integers(1, 60000, 150_000).astype(np.uint16), 40), 1e-3, rng)
    for k in rng.integers(0, len(T) - 6, 400):
        T[k:k + 6] = np.arange(1, 7)
    err = _way(ctx, T, capfd, monkeypatch)
    assert "large groups, h=" in err and "have a follower" in err


@pytest.mark.parametrize("kind", ["phrases", "far_copies", "two_symbols"])
def test_ties_that_the_text_settles_are_not_ranked(ctx, capfd, monkeypatch, kind):
    """Many tied suffixes whose groups fall apart a symbol on: no inverse array is made to find that out."""
    rng = np.random.default_rng(3)
    if kind == "phrases":
        T = _phrases(40_000_000, 4, 4, rng)
    elif kind == "far_copies":
        T = _mutated(np.tile(rng.integers(1, 60000, 300_000).astype(np.uint16), 20), 0.05, rng)
    else:
        T = rng.integers(0, 2, 40_000_000).astype(np.uint16)
    err = _way(ctx, T, capfd, monkeypatch)
    assert "are tied one symbol on" in err and "have a follower" not in err


def test_ties_that_the_text_settles_need_no_memory_for_ranks(capfd, monkeypatch):
    """Phrases of thirty symbols: nearly all groups are followed, but where the device has no room for the ranks the text alone tells the suffixes apart. A text
    that needs them is refused, and the context goes on."""
    from cascade_b200 import api
    rng = np.random.default_rng(4)
    n = 1 << 24
    texts = [_phrases(n + 30, 30, 4, rng)[:n], np.tile(rng.integers(1, 60000, n // 8).astype(np.uint16), 8)]
    T = [torch.from_numpy(np.concatenate([t, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16) for t in texts]
    out = torch.zeros(5 * n + api.SA_PAD_BYTES, dtype=torch.uint8, device="cuda")
    other = api.Context(0)                          # loads every kernel, so that a full device is not asked for that
    for t in T:
        api.build_sa(other, t, n, 8, out=out)
    other.close()
    ctx = api.Context(0)
    filler = []
    try:
        ordinary = torch.randint(0, 60000, (n + api.TEXT_PAD,), device="cuda", dtype=torch.int32).to(torch.int16)
        ordinary[n:] = 0
        api.build_sa(ctx, ordinary.view(torch.uint16), n, 8, out=out)          # takes the buffers that every build of this length has
        monkeypatch.setenv("CSA_DEBUG", "1")
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        need = 16 * n                                       # what the ranks take at least
        if free > need // 2:
            filler.append(torch.empty(free - need // 2, dtype=torch.uint8, device="cuda"))
        capfd.readouterr()
        api.build_sa(ctx, T[0], n, 8, out=out)
        err = capfd.readouterr().err
        with pytest.raises(api.CascadeError) as refused:
            api.build_sa(ctx, T[1], n, 8, out=out)
        assert refused.value.code == 3
        api.build_sa(ctx, T[0], n, 8, out=out)
        filler.clear()
        torch.cuda.empty_cache()
        v = api.validate_sa(ctx, T[0], n, out)
        assert v["ok"], v
        assert "are tied one symbol on" in err and "have a follower" not in err
    finally:
        ctx.close()
