"""Paths that serve tables on which an insert has reused a tombstone (or whose
history is not known: loaded tables), and inserts too small beside their table
to be merged: remove groups of every size, removes without an EMPTY slot,
components of more ops than a warp gathers -- plain calls and batches, against
the oracle."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


def _records(rng, n, size):
    return rng.integers(0, 256, (n, size), dtype=np.uint8)


def _keys_at(cap, homes, ks, salt=0):
    """Distinct keys with the given home slots (identity hash)."""
    homes = np.asarray(homes, np.uint64)
    k = np.zeros((len(homes), ks), np.uint8)
    x = (np.arange(len(homes), dtype=np.uint64) + np.uint64(1 + salt)) * np.uint64(cap) + homes
    k[:, :8] = x.view(np.uint8).reshape(-1, 8)
    return k


def _same(g, o):
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)


def _age(g, o, how, rng):
    """Gives both tables a history: 'loaded' (not known) or 'claimed' (an insert has reused a tombstone)."""
    if how == "loaded":
        g.load(*g.snapshot(), g.len())
        return
    cap = o.capacity
    k = _keys_at(cap, rng.integers(0, cap, 40), g.key_size, salt=1 << 40)
    v = _records(rng, 40, g.value_size)
    assert g.bulk_insert(k, v) == o.bulk_insert(k, v)
    assert g.bulk_remove(k) == o.bulk_remove(k)
    k2 = k.copy()
    k2[:, 5] ^= 1  # other keys of the same homes: they take the tombstones
    v2 = _records(rng, 40, g.value_size)
    assert g.bulk_insert(k2, v2) == o.bulk_insert(k2, v2)
    _same(g, o)


def _run_remove(g, o, k, batch):
    """One remove, plain or queued in a (captured) batch."""
    if batch is None:
        assert g.bulk_remove(k) == o.bulk_remove(k)
        return
    import torch

    import flash_map as F

    s = torch.cuda.Stream()
    d = torch.from_numpy(np.ascontiguousarray(k)).cuda()
    torch.cuda.synchronize()
    b = F.FlashMapBatch([F.BatchOp(F.batch.REMOVE, g, len(k), d)])
    if batch == "graph":
        b.capture(s)
    b.run(s)
    assert b.wait() == [(o.bulk_remove(k), 0)]
    b.close()


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("batch,ngroup", [(None, 10), (None, 40), (None, 300), (None, 3000), (None, 9000), ("run", 10),
                                          ("run", 300), ("run", 3000), ("graph", 10), ("graph", 40), ("graph", 300)])
@pytest.mark.parametrize("how", ["loaded", "claimed"])
def test_remove_groups(shape, batch, ngroup, how):
    """Groups between EMPTY slots that a lane, a warp, a block and (9,000 ops, plain calls) the rounds run, with repeats
    and absent keys, beside lone removes."""
    ks, vs = shape
    if ngroup == 9000 and (ks != 8 or how != "claimed"):
        pytest.skip("the rounds take 20 s for a group of this size: once")
    cap = 1 << 15
    rng = np.random.default_rng(ngroup + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    nclu = min(ngroup + ngroup // 4, 12000)
    clu = _keys_at(cap, 2000 + np.arange(nclu) % 200, ks)
    k0 = np.concatenate([clu, _records(rng, cap // 3, ks)])
    v0 = _records(rng, len(k0), vs)
    assert g.bulk_insert(k0, v0) == o.bulk_insert(k0, v0)
    _age(g, o, how, rng)
    absent = _keys_at(cap, np.full(ngroup // 10, 2050), ks, salt=20000)
    grp = np.concatenate([clu[rng.choice(nclu, ngroup - ngroup // 10 - ngroup // 20, replace=False)],
                          clu[rng.integers(0, nclu, ngroup // 20)], absent])
    rest = k0[nclu + rng.choice(len(k0) - nclu, 2000, replace=False)]
    rm = np.concatenate([grp, rest])
    _run_remove(g, o, rm[rng.permutation(len(rm))], batch)
    _same(g, o)
    q = np.concatenate([clu, rest])
    for a, b in zip(g.bulk_get(q), o.bulk_get(q)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128), (12, 20)])
@pytest.mark.parametrize("how", ["removed", "loaded"])
@pytest.mark.parametrize("batch", [None, "run", "graph"])
def test_removes_without_an_empty_slot(shape, how, batch):
    """A filled table has no EMPTY slot, before and after removes: present, repeated and absent keys."""
    ks, vs = shape
    cap = 1 << 12
    rng = np.random.default_rng(ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    k, v = _records(rng, cap, ks), _records(rng, cap, vs)
    assert g.bulk_insert(k, v) == o.bulk_insert(k, v) == cap
    if how == "loaded":
        g.load(*g.snapshot(), g.len())
    for n in (100, 700):
        rm = np.concatenate([k[rng.choice(cap, n, replace=False)], k[rng.integers(0, cap, 30)], _records(rng, 300, ks)])
        _run_remove(g, o, rm, batch)
        _same(g, o)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("nkeys", [63, 64, 65, 70, 200, 1000])
@pytest.mark.parametrize("how", ["clean", "claimed", "loaded"])
def test_components_around_what_a_warp_gathers(shape, nkeys, how):
    """nkeys ops on a few neighbouring homes of a half-full table, in a call below 1/16 of its slots."""
    ks, vs = shape
    cap = 1 << 17
    rng = np.random.default_rng(nkeys)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    k0, v0 = _records(rng, cap // 2, ks), _records(rng, cap // 2, vs)
    assert g.bulk_insert(k0, v0) == o.bulk_insert(k0, v0)
    if how != "clean":
        _age(g, o, how, rng)
    crowd = _keys_at(cap, 5000 + rng.integers(0, 4, nkeys), ks)
    lone = _records(rng, 3000, ks)
    k = np.concatenate([lone[:1500], crowd, lone[1500:]])
    v = _records(rng, len(k), vs)
    assert g.bulk_insert(k, v) == o.bulk_insert(k, v)
    _same(g, o)
