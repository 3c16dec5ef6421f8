"""The local sort's ways through a batch of children, by how many records share a key and how evenly the keys lie: bins that a thread's window orders, crowded
bins, batches of more tied records than a block keeps, batches of many records of each key, of many keys close together, and large groups. Each array
byte for byte against the oracle's."""
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


def _check(ctx, oracle, T):
    from cascade_b200 import api
    T = np.ascontiguousarray(T, dtype=np.uint16)
    n = len(T)
    Td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    sa, st = api.build_sa(ctx, Td, n, 8)
    assert np.array_equal(sa[:5 * n].cpu().numpy(), oracle.build_sa40(T)[:5 * n])
    return st


# one split, two splits; copies of every piece: 2 to 4 records of a key lie in a window, 5 to 15 make a crowded bin, 16 and more a crowded batch, 300 a large group
@pytest.mark.parametrize("n,copies", [(n, c) for n in (40_000, 300_001) for c in (2, 3, 4, 5, 8, 15, 16, 17, 31, 33, 40, 300)] + [(2_300_003, c) for c in (3, 9, 40)])
def test_pieces_that_stand_so_many_times(ctx, oracle, n, copies):
    rng = np.random.default_rng(n + copies)
    piece = 23
    base = rng.integers(0, 50000, (n // (2 * piece * copies) + 1, piece))
    pieces = np.repeat(base, copies, axis=0)
    rng.shuffle(pieces)
    T = np.concatenate([pieces.ravel()[:n // 2], rng.integers(0, 50000, n - n // 2)])     # half of the text is told apart by its first symbols
    st = _check(ctx, oracle, T)
    assert st.active_after_gen0 > n // 4


@pytest.mark.parametrize("n", [300_000, 2_500_000])
@pytest.mark.parametrize("kind", ["steep", "few_symbols", "one_in_two", "twice"])
def test_keys_that_lie_unevenly(ctx, oracle, n, kind):
    rng = np.random.default_rng(n)
    if kind == "steep":                 # a hundred symbols, each half as frequent as the one before
        T = np.minimum(rng.geometric(0.5, n), 100)
    elif kind == "few_symbols":         # children that hold nearly everything or nothing
        T = np.where(rng.random(n) < 0.9, 5, rng.integers(0, 4, n))
    elif kind == "one_in_two":          # every other symbol is one of three
        T = rng.integers(0, 60000, n)
        T[::2] = rng.integers(0, 3, (n + 1) // 2)
    else:                               # every piece stands twice: more ties than a block keeps
        pieces = rng.integers(0, 60000, (n // 120, 60))
        T = np.concatenate([pieces, rng.permutation(pieces)]).ravel()
    _check(ctx, oracle, T)


# few tied suffixes, which a thread each compares where a group has up to 15 members: pieces shorter and longer than what is compared at once, and a copy that the text's end cuts off
@pytest.mark.parametrize("length", [23, 49, 80, 300])
@pytest.mark.parametrize("copies", [2, 3, 15, 16])
@pytest.mark.parametrize("n", [17_003, 200_001])
def test_few_ties(ctx, oracle, n, copies, length):
    rng = np.random.default_rng(n + copies + length)
    pieces = np.repeat(rng.integers(0, 60000, (8000 // (copies * length) + 1, length)), copies, axis=0)
    T = rng.integers(0, 60000, n)
    for k, at in enumerate(rng.permutation(n // (length + 1) - 1)[:len(pieces)]):
        T[at * (length + 1):][:length] = pieces[k]
    T[-length // 2:] = pieces[0][:length // 2 + length % 2]
    _check(ctx, oracle, T)


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1, 1_000_003])
def test_one_split_by_small_and_by_wide_tiles(ctx, oracle, n):
    rng = np.random.default_rng(n)
    _check(ctx, oracle, np.minimum(rng.zipf(1.2, n), 50257))


def test_a_split_into_a_thousand_children_of_a_parent(ctx):
    """The larger blocks of the second split: from 2^29 suffixes on. Checked by the validator, which looks at every entry."""
    from cascade_b200 import api
    n = (1 << 29) + (1 << 25) + 7
    T = api.gen_corpus_device(ctx, n, 3, 1024)
    sa, _ = api.build_sa(ctx, T, n, 8)
    assert api.validate_sa(ctx, T, n, sa)["ok"]


@pytest.mark.parametrize("n", [1_000_003, 4_000_001, 9_000_001, 13_000_003])
def test_parents_of_few_children(ctx, n):
    """Parts straight from the text, whose parents have two to sixteen children: batches of up to four of them, whose keys give up their last bits."""
    from cascade_b200 import api
    T = api.gen_corpus_device(ctx, n, 9, 512)
    Th = T.cpu()
    sa, st = api.build_sa_streamed(ctx, Th.view(torch.int16).numpy().view(np.uint16), n, 64)
    assert st.host_parts == 0, "not straight from the text"
    assert api.validate_sa(ctx, T, n, torch.from_numpy(sa).cuda())["ok"]


@pytest.mark.parametrize("n", [1_000_003, 4_000_001, 9_000_001])
@pytest.mark.parametrize("copies", [2, 5, 15])
def test_parents_of_few_children_with_ties(ctx, n, copies):
    """The same with a tenth of the text in pieces that stand several times: what the keys' last bits told apart is told by the text."""
    from cascade_b200 import api
    rng = np.random.default_rng(n + copies)
    pieces = np.repeat(rng.integers(0, 50000, (n // (10 * 23 * copies), 23)), copies, axis=0)
    rng.shuffle(pieces)
    T = np.concatenate([rng.integers(0, 50000, n - pieces.size), pieces.ravel()]).astype(np.uint16)
    sa, st = api.build_sa_streamed(ctx, T, n, 64)
    assert st.host_parts == 0 and st.active_after_gen0 > n // 20, "not straight from the text, or no ties"
    Td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    assert api.validate_sa(ctx, Td, n, torch.from_numpy(sa).cuda())["ok"]


@pytest.mark.parametrize("n,by_records", [(2_200_003, 2 * 2_200_003 // 4092 + 2048 // 64 + 32), (4_500_003, 2 * 4_500_003 // 4092 + 4096 // 64 + 64)])
def test_runs_of_nearly_empty_children(ctx, oracle, monkeypatch, capfd, n, by_records):
    """Two alphabets of 32 symbols by turns, one position in a hundred off: parents whose children hold nearly everything or nothing, and more batches than records and segments account for (4.5e6; the list
    has an entry for every child)."""
    rng = np.random.default_rng(n)
    odd = (np.arange(n) & 1).astype(bool) ^ (rng.random(n) < 0.01)
    T = np.where(odd, 65000, 0) + rng.integers(0, 32, n)
    monkeypatch.setenv("CSA_DEBUG", "1")
    _check(ctx, oracle, T)
    batches = int(re.search(r"of (\d+) batches", capfd.readouterr().err).group(1))
    assert batches > by_records or n < 4_000_000
