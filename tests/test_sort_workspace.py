"""One workspace of csa_sort_pairs serves every list up to the length that it was sized for: builds size one for their longest list and sort what is left of it."""
import ctypes

import pytest


def test_the_size_never_falls_as_the_list_grows():
    from cascade_b200._lib import lib
    f = lib().csa_sort_workspace_bytes
    # where the number of bucket bits changes (powers of two times 1024), a tile or a launch more, and around 2^26, the most that is sorted by buckets
    edges = [1 << b for b in range(1, 33)] + [4608 * k for k in (1, 2, 3)] + [3 << b for b in range(8, 27)]
    sizes = sorted({n for e in edges for n in range(max(1, e - 3), e + 4)} | {(1 << 26) + d for d in range(1, 700_001, 997)})
    bytes_ = [f(n) for n in sizes]
    assert all(a <= b for a, b in zip(bytes_, bytes_[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("n,sized_for", [(1 << 26, (1 << 26) + 1), ((1 << 26) + 1, (1 << 26) + 1), (5000, (1 << 26) + 1), (3_000_001, 1 << 27)])
def test_a_list_in_the_workspace_of_a_longer_one(n, sized_for):
    import torch
    from cascade_b200 import api
    ctx = api.Context(0)
    try:
        g = torch.Generator(device="cuda").manual_seed(n)
        keys = torch.randint(-(1 << 62), 1 << 62, (n,), device="cuda", dtype=torch.int64, generator=g) * 2
        vals = torch.arange(n, device="cuda", dtype=torch.int32)
        ka, va = torch.empty_like(keys), torch.empty_like(vals)
        k0 = keys.clone()
        wsb = ctx.L.csa_sort_workspace_bytes(sized_for)
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        in_alt = ctypes.c_int(0)
        torch.cuda.synchronize()
        ctx.check(ctx.L.csa_sort_pairs(ctx.h, keys.data_ptr(), ka.data_ptr(), vals.data_ptr(), va.data_ptr(), 4, n, 0, 64, ws.data_ptr(), wsb, ctypes.byref(in_alt)))
        ctx.sync()
        order = torch.sort(k0 ^ (-(1 << 63)), stable=True).indices
        ko, vo = (ka, va) if in_alt.value else (keys, vals)
        assert torch.equal(ko, k0[order]) and torch.equal(vo, order.to(torch.int32))
    finally:
        ctx.close()


@pytest.mark.gpu
def test_a_build_whose_large_groups_shrink_past_the_edge():
    """One symbol 2^26 + 1000 times: the doubling generations sort 2^26 + 1000 suffixes, then what is left of them, fewer than 2^26."""
    import torch
    from cascade_b200 import api
    ctx = api.Context(0)
    try:
        n = (1 << 26) + 1000
        T = torch.full((n + api.TEXT_PAD,), 7, dtype=torch.int16, device="cuda")
        T[n:] = 0
        T = T.view(torch.uint16)
        sa, _ = api.build_sa(ctx, T, n, 8)
        v = api.validate_sa(ctx, T, n, sa)
        assert v["ok"], v
    finally:
        ctx.close()
