"""Host query batches that two launches answer, from and to pinned and pageable memory, against the oracle."""
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


def _setup(ctx, oracle):
    from cascade_b200 import api
    rng = np.random.default_rng(1)
    n = 30_000
    T = np.minimum(rng.zipf(1.3, n), 200).astype(np.uint16)
    sa = oracle.build_sa40(T)
    td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
    return T, sa, api.SuffixIndex(ctx, td, torch.from_numpy(np.ascontiguousarray(sa)).cuda(), n, 16)


def _batch(T, q, seed):
    rng = np.random.default_rng(seed)
    pats = []
    for i in range(q):
        m, at = int(rng.integers(0, 20)), int(rng.integers(0, len(T) - 20))
        pats.append(T[at:at + m] if i % 3 else rng.integers(0, 210, m).astype(np.uint16))
    off = np.concatenate([[0], np.cumsum([len(x) for x in pats])]).astype(np.uint64)
    return off, np.concatenate(pats + [np.zeros(1, np.uint16)]).astype(np.uint16)


# a block answers 32 queries; up to 256 are read in place; 8193 go through the lanes
@pytest.mark.parametrize("q,max_pos", [(1, 1), (31, 7), (33, 100), (256, 20), (257, 20), (3000, 5), (8192, 40), (8193, 40)])
@pytest.mark.parametrize("pinned", ["all", "none", "inputs", "outputs"])
def test_answers_from_and_to_any_memory(ctx, oracle, q, max_pos, pinned):
    T, sa, idx = _setup(ctx, oracle)
    off, sym = _batch(T, q, q)
    bufs = {"itv": torch.zeros(2 * q, dtype=torch.int64), "cnt": torch.zeros(q, dtype=torch.int32), "pos_off": torch.zeros(q + 1, dtype=torch.int64),
            "pos": torch.full((q * max_pos + 1,), -7, dtype=torch.int64)}
    o, s = torch.from_numpy(off.view(np.int64)), torch.from_numpy(sym.view(np.int16))
    if pinned in ("all", "inputs"):
        o, s = o.pin_memory(), s.pin_memory()
    if pinned in ("all", "outputs"):
        bufs = {k: v.pin_memory() for k, v in bufs.items()}
    itv, cnt, poff, pos, total = idx.query_host(o, s, max_pos, bufs)
    want = oracle.find_batch(T, sa, off, sym)
    rows, counts = oracle.locate_batch(sa, want, max_pos)
    assert np.array_equal(itv.numpy().view(np.uint64), want) and np.array_equal(cnt.numpy().view(np.uint32), counts)
    assert np.array_equal(poff.numpy(), np.concatenate([[0], np.cumsum(counts.astype(np.int64))])) and total == int(counts.sum())
    assert np.array_equal(pos.numpy()[:total].view(np.uint64), np.concatenate([rows[i, :counts[i]] for i in range(q)]))
    assert int(pos[q * max_pos]) == -7


@pytest.mark.parametrize("pinned", [True, False])
def test_counts_alone_and_a_positions_buffer_that_is_too_small(ctx, oracle, pinned):
    from cascade_b200 import api
    T, sa, idx = _setup(ctx, oracle)
    q = 100
    off, sym = _batch(T, q, 5)
    want = oracle.find_batch(T, sa, off, sym)
    itv, _, _, _, total = idx.query_host(off, sym, 0)
    assert np.array_equal(itv, want) and total == 0
    few = torch.full((11,), -7, dtype=torch.int64)
    itv = torch.zeros(2 * q, dtype=torch.int64)
    if pinned:
        few, itv = few.pin_memory(), itv.pin_memory()
    with pytest.raises(api.CascadeError) as e:
        idx.query_host(off, sym, 20, {"pos": few[:10], "itv": itv})
    assert e.value.code == 3 and int(few[10]) == -7 and np.array_equal(itv.numpy().view(np.uint64), want)
    itv, cnt, poff, pos, total = idx.query_host(off, sym, 20)      # and the context goes on as before
    assert np.array_equal(itv, want) and int(poff[q]) == total
    bad = off.copy()
    bad[q] = 0
    bad[0] = 1
    with pytest.raises(api.CascadeError):
        idx.query_host(bad, sym, 20)


@pytest.mark.parametrize("what", ["off", "sym", "itv", "pos"])
def test_buffers_of_which_only_the_first_page_is_pinned(ctx, oracle, what):
    """Such a buffer is pageable memory: neither are its other pages read or written in place nor is the call refused."""
    import mmap
    T, sa, idx = _setup(ctx, oracle)
    q, max_pos = 1000, 5
    off, sym = _batch(T, q, 9)
    sizes = {"off": (q + 1) * 8, "sym": len(sym) * 2, "itv": 2 * q * 8, "pos": q * max_pos * 8}
    assert min(sizes.values()) > 4096
    memory = mmap.mmap(-1, (sizes[what] + 4095) // 4096 * 4096)
    buf = np.frombuffer(memory, dtype=np.uint16 if what == "sym" else np.uint64)[:sizes[what] // (2 if what == "sym" else 8)]
    cudart = torch.cuda.cudart()
    assert int(cudart.cudaHostRegister(buf.ctypes.data, 4096, 0)) == 0
    try:
        o, s, bufs = off, sym, {}
        if what in ("off", "sym"):
            buf[:] = off if what == "off" else sym
            o, s = (buf, sym) if what == "off" else (off, buf)
        else:
            bufs = {what: buf}
        itv, cnt, _, pos, total = idx.query_host(o, s, max_pos, bufs)
        want = oracle.find_batch(T, sa, off, sym)
        rows, counts = oracle.locate_batch(sa, want, max_pos)
        assert np.array_equal(itv, want) and np.array_equal(cnt, counts) and total == int(counts.sum())
        assert np.array_equal(pos[:total], np.concatenate([rows[i, :counts[i]] for i in range(q)]))
    finally:
        assert int(cudart.cudaHostUnregister(buf.ctypes.data)) == 0
