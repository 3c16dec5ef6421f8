"""csa_find on batches of patterns of one symbol (a warp of them has a search of its own), against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# the first and the last symbol of the alphabet in the text and not, symbols that stand once, and one in half of the places; strides past a symbol's run and past the text
@pytest.mark.parametrize("n,stride", [(1, 1), (40, 64), (20_000, 1), (20_000, 32), (20_000, 64)])
@pytest.mark.parametrize("ends", [False, True])
@pytest.mark.parametrize("mixed", [False, True])
def test_every_symbol(oracle, n, stride, ends, mixed):
    from cascade_b200 import api
    ctx = api.Context(0)
    try:
        rng = np.random.default_rng(n + stride)
        T = np.where(rng.random(n) < 0.5, 300, rng.integers(1, 65535, n)).astype(np.uint16)
        if ends:
            T[::7] = 0
            T[::11] = 65535
            T[-1] = 0
        sa = oracle.build_sa40(T)
        td = torch.from_numpy(np.concatenate([T, np.zeros(api.TEXT_PAD, np.uint16)]).view(np.int16)).cuda().view(torch.uint16)
        idx = api.SuffixIndex(ctx, td, torch.from_numpy(np.ascontiguousarray(sa)).cuda(), n, stride)
        pats = [np.array([c], np.uint16) for c in rng.permutation(65536)]
        if mixed:       # warps with another length or an empty pattern among them
            for k in range(0, 65536, 77):
                pats[k] = np.array([300, 300], np.uint16) if k % 2 else np.zeros(0, np.uint16)
        off = np.concatenate([[0], np.cumsum([len(x) for x in pats])]).astype(np.uint64)
        sym = np.concatenate(pats + [np.zeros(8, np.uint16)])
        itv = idx.find(torch.from_numpy(off.view(np.int64)).cuda(), torch.from_numpy(sym.view(np.int16)).cuda().view(torch.uint16), len(pats))
        assert np.array_equal(itv.cpu().numpy().view(np.uint64), oracle.find_batch(T, sa, off, sym))
    finally:
        ctx.close()
