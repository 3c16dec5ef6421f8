"""Builds in one block, around the sizes and the texts at which a text is left to the general build. Each array byte for byte against the oracle's."""
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


def _check(ctx, oracle, T, p=5):
    """The array; returns whether one launch made it."""
    from cascade_b200 import api
    T = np.ascontiguousarray(T, dtype=np.uint16)
    n = len(T)
    Tp = np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)])
    Td = torch.from_numpy(Tp.view(np.int16)).cuda().view(torch.uint16)
    out = torch.full((5 * n + api.SA_PAD_BYTES,), 0xAB, dtype=torch.uint8, device="cuda")
    sa, st = api.build_sa(ctx, Td, n, p, out=out)
    assert np.array_equal(sa[:5 * n].cpu().numpy(), oracle.build_sa40(T)[:5 * n])
    assert bool((sa[5 * n:] == 0xAB).all()), "written behind the array"
    assert 1 <= st.partitions <= p and 0 < st.max_partition <= n
    assert np.array_equal(api.build_sa_host(ctx, Tp, n, p)[0][:5 * n], sa[:5 * n].cpu().numpy())
    return st.kernel_launches == 1


# 1024 threads, 16 entries packed at a time, 16384 symbols at most; symbols at both ends of the alphabet
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 1023, 1025, 2049, 5000, 16383, 16384, 16385])
@pytest.mark.parametrize("sigma", [4, 300, 65536])
def test_random_texts(ctx, oracle, n, sigma):
    T = np.random.default_rng(n + sigma).integers(0, sigma, n)
    T[0] = sigma - 1
    one = _check(ctx, oracle, T)
    assert one == (n <= 16384) or sigma == 4 or n < 40


@pytest.mark.parametrize("copies", [2, 60, 64, 65, 400])
@pytest.mark.parametrize("length", [5, 40, 300])
def test_repeats(ctx, oracle, copies, length):
    """A passage that stands in the text as many times: bins of up to 64 suffixes, and comparisons that end at the text's end or take too long."""
    rng = np.random.default_rng(copies * length)
    passage = rng.integers(1, 60000, length)
    n = min(16384, copies * (length + 30))
    T = rng.integers(1, 60000, n)
    step = n // copies
    for k in range(copies):
        T[k * step:k * step + min(length, step)] = passage[:min(length, step)]
    T[n - min(length, n):] = passage[:min(length, n)]
    _check(ctx, oracle, T)


@pytest.mark.parametrize("n", [1, 2, 64, 65, 5000])
def test_one_symbol_two_symbols_and_zeros_at_the_end(ctx, oracle, n):
    rng = np.random.default_rng(n)
    for symbol in (0, 7, 65535):
        _check(ctx, oracle, np.full(n, symbol))
    _check(ctx, oracle, rng.integers(0, 2, n) * 65535)
    T = rng.integers(0, 60000, n)
    T[n // 2:] = 0
    _check(ctx, oracle, T)
    T[:] = np.arange(n) % 65536            # every symbol once, in order
    _check(ctx, oracle, T)
    _check(ctx, oracle, T[::-1])


# which of them one launch makes; None: either way
@pytest.mark.parametrize("n", [900, 3001, 16384])
@pytest.mark.parametrize("kind,one", [("a passage twice", True), ("a short passage often", True), ("phrases of four symbols", None), ("phrases forty times", None), ("documents twenty times", None),
                                      ("a period", False), ("two symbols in turn", False), ("zeros at the end of every document", False)])
def test_repetitive_texts(ctx, oracle, n, kind, one):
    """Pairs of suffixes in one bin and comparisons up to the limits and past them: what is given up is made by the general build, from the start."""
    rng = np.random.default_rng(n)
    T = rng.integers(1, 60000, n)
    if kind == "a passage twice":
        T[n // 2:n // 2 + 300] = T[10:310]
    elif kind == "a short passage often":
        for k in range(20):
            T[k * (n // 20):k * (n // 20) + 12] = np.arange(12)
    elif kind == "phrases of four symbols":
        T = rng.integers(1, 60000, (n // 16, 4))[rng.integers(0, n // 16, n // 4 + 1)].reshape(-1)[:n]
    elif kind == "phrases forty times":
        T = rng.integers(1, 60000, (n // 200, 5))[rng.integers(0, n // 200, n // 5 + 1)].reshape(-1)[:n]
    elif kind == "documents twenty times":
        T = np.tile(T[:n // 20 + 1], 20)[:n]
        T[rng.random(n) < 0.02] = 7
    elif kind == "a period":
        T = np.arange(n) % 9
    elif kind == "two symbols in turn":
        T = np.arange(n) % 2 * 65535
    else:
        T[np.arange(n) % 300 > 200] = 0
    way = _check(ctx, oracle, T)
    assert one is None or way == one
