"""The forming of the local sort's batches (csrc/batches.hpp, which the kernel and the host code share): every plan's list has room for whatever the children's sizes are."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SORT_MOST, SHORT_BATCH, SEGMENT, SHORT_SEGMENT = 4092, 1024, 64, 8

SHIM = """
#include "batches.hpp"
extern "C" uint64_t room(uint32_t parents, uint32_t children) { return most_batches(parents, children); }
extern "C" uint32_t longest(uint32_t children) { return longest_run(children); }
extern "C" void constants(uint32_t* c) { c[0] = SORT_MOST; c[1] = SHORT_BATCH; c[2] = SEGMENT; c[3] = SHORT_SEGMENT; }
extern "C" uint64_t form(const uint32_t* off, uint32_t children, uint32_t segment, uint32_t most, uint32_t* sizes)
{
    uint64_t batches = 0;
    for(uint32_t s = 0; s < children; s += segment)
        for(uint32_t i = s; i < children && i < s + segment;)
        {
            const uint32_t e = batch_end(off, i, children, segment, most), m = off[e] - off[i];
            if(m && m <= SORT_MOST) sizes[batches++] = m;
            i = e;
        }
    return batches;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("batches")
    src, so = str(d / "shim.cpp"), str(d / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "cascade_b200", "csrc"), src, "-o", so])
    L = ctypes.CDLL(so)
    L.room.restype = L.form.restype = ctypes.c_uint64
    c = (ctypes.c_uint32 * 4)()
    L.constants(c)
    assert tuple(c) == (SORT_MOST, SHORT_BATCH, SEGMENT, SHORT_SEGMENT)
    return L


def _batches(L, sizes, segment, most):
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    out = np.zeros(len(sizes), np.uint32)
    k = L.form(off.ctypes.data_as(ctypes.c_void_p), len(sizes), segment, most, out.ctypes.data_as(ctypes.c_void_p))
    assert out[:k].sum() == sum(np.diff(off)[np.diff(off) <= SORT_MOST])      # every record of a child that a batch may hold is in one
    return int(k)


# children of a parent: all plans of the resident build and of parts straight from the text
@pytest.mark.parametrize("b2", range(0, 12))
@pytest.mark.parametrize("kind", ["even", "every_other", "one_a_run", "full_and_one", "random", "heavy_tail", "empty_ones"])
def test_a_list_has_room_for_every_batch(shim, b2, kind):
    children = 1 << b2
    rng = np.random.default_rng(b2)
    c = shim.longest(children)
    i = np.arange(children)
    sizes = {"even": np.full(children, 1536), "every_other": np.where(i % 2, 1, 2900), "one_a_run": np.where(i % c == 0, 1, 0), "full_and_one": np.where(i % 2, 1, SORT_MOST),
             "random": rng.integers(0, 4000, children), "heavy_tail": np.minimum(rng.zipf(1.3, children), 20000), "empty_ones": np.where(rng.random(children) < 0.7, 0, 1)}[kind]
    for segment, most in ((SEGMENT, SORT_MOST), (SHORT_SEGMENT, SHORT_BATCH)):
        if segment == SHORT_SEGMENT and b2 > 10:
            continue            # one split has at most 1024 children
        assert _batches(shim, sizes, segment, most) <= shim.room(1, children)


@pytest.mark.parametrize("children", [64, 128, 256])
def test_runs_that_end_by_their_number(shim, children):
    """Parents by turns of children with one suffix each, whose runs end by their number, and of children with 2047, no two of which fit a batch: 1024 a child on average, as the plans have it, and more
    batches than records and segments account for."""
    parents = 64
    sparse, dense = np.ones(children, int), np.full(children, SORT_MOST // 2 + 1)
    batches = parents // 2 * (_batches(shim, sparse, SEGMENT, SORT_MOST) + _batches(shim, dense, SEGMENT, SORT_MOST))
    n = parents // 2 * int(sparse.sum() + dense.sum())
    assert batches > 2 * n // SORT_MOST + parents * children // SEGMENT + parents
    assert batches <= shim.room(parents, children)
