"""The merging insert's words are part of a table's scratch: calls on fresh
tables, on tables whose scratch came without them, with them in a scratch that
grows, and without room for them, against the oracle."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


def _records(rng, n, size):
    return rng.integers(0, 256, (n, size), dtype=np.uint8)


def _insert(g, o, n, rng, fault=False):
    """Inserts n pairs from device memory; the kernels launched by it."""
    import torch
    from flash_map import _native

    k, v = _records(rng, n, g.key_size), _records(rng, n, g.value_size)
    dk, dv = torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()
    torch.cuda.synchronize()
    before = _native.launch_count()
    if fault:
        _native.inject_fault(_native.FAULT_ALLOC, 0)
    try:
        assert g.bulk_insert_device(dk, dv, n) == o.bulk_insert(k, v)
    finally:
        _native.inject_fault(_native.FAULT_NONE)
    launches = _native.launch_count() - before
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)
    return launches


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("calls", [(9000,), (100, 9000, 4000), (9000, 100, 3000), (2000, 11000), (6000, 6000, 3000)])
def test_words_with_the_scratch(shape, calls):
    cap = 1 << 14
    rng = np.random.default_rng(len(calls))
    g, o = gpu_map(cap, *shape), O.OracleMap(cap, *shape)
    for n in calls:
        _insert(g, o, n, rng)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
def test_no_room_for_the_words(shape):
    """The first allocation, with the words, fails: the call runs without the merge, and later ones go on."""
    cap = 1 << 14
    rng = np.random.default_rng(5)
    g, o = gpu_map(cap, *shape), O.OracleMap(cap, *shape)
    assert _insert(g, o, 9000, rng, fault=True) < 10
    _insert(g, o, 3000, rng)
    g.clear()
    o.clear()
    assert _insert(g, o, 12000, rng) >= 10  # a larger scratch, with the words


def test_no_second_allocation_in_a_first_merging_call():
    """A fresh table's first merging call takes one block: with the second allocation from there on failing, it merges
    all the same."""
    from flash_map import _native
    import torch

    cap = 1 << 20
    rng = np.random.default_rng(6)
    g, o = gpu_map(cap, 8, 8), O.OracleMap(cap, 8, 8)
    k = _records(rng, cap // 2, 8)
    d = torch.from_numpy(k).cuda()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _native.inject_fault(_native.FAULT_ALLOC, 1)
    try:
        before = _native.launch_count()
        assert g.bulk_insert_device(d, d, len(k)) == o.bulk_insert(k, k)
        assert _native.launch_count() - before >= 10
        g.bulk_insert_device(d, d, len(k))  # and no allocation later either
    finally:
        _native.inject_fault(_native.FAULT_NONE)
    used = free - torch.cuda.mem_get_info()[0]
    assert used < (cap // 2 * 5 // 4 + 1024) * 42 + cap * 4 + (8 << 20)
