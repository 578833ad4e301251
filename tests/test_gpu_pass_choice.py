"""Which passes a small insert runs on follows from the table's history, size
and load: at most four launches and one wait's worth of work where one set of
passes does it all; and small tables against the oracle at the sizes where the
component pass begins."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


def _records(rng, n, size):
    return rng.integers(0, 256, (n, size), dtype=np.uint8)


def _keys_at(rng, homes, ks):
    k = _records(rng, len(homes), ks)
    k[:, :4] = np.asarray(homes, np.uint32).view(np.uint8).reshape(-1, 4)
    return k


def _same(g, o):
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)


def _insert(g, o, k, rng):
    """Kernels launched by one insert, checked against the oracle."""
    from flash_map import _native

    v = _records(rng, len(k), g.value_size)
    before = _native.launch_count()
    got = g.bulk_insert(k, v)
    n = _native.launch_count() - before
    assert got == o.bulk_insert(k, v)
    return n


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("bits", [4, 6, 8, 9, 10, 11, 12, 14])
@pytest.mark.parametrize("history", ["clean", "removed"])
def test_one_set_of_passes(shape, bits, history):
    """A few new keys, two of them on one home (a component): find, flow and two passes more, no second wait."""
    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    k0 = _keys_at(rng, np.arange(0, cap // 2, 2), ks)
    _insert(g, o, k0, rng)
    if history == "removed":
        assert g.bulk_remove(k0[:3]) == o.bulk_remove(k0[:3])
    n = max(2, min(20, cap // 32))  # below 1/16 of the slots
    homes = rng.integers(0, cap, n)
    homes[:2] = cap // 4
    assert _insert(g, o, _keys_at(rng, homes, ks), rng) <= 4
    _same(g, o)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128), (32, 32)])
@pytest.mark.parametrize("bits", [3, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("load", [0.3, 0.7, 0.9])
def test_small_tables(shape, bits, load):
    """Calls below 1/16 of the slots, to the load and beyond it: lone ops, components, repeats, updates, walks round the
    end of the table, runs longer than a component may be."""
    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits * 10 + int(load * 10) + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    k0 = _keys_at(rng, rng.integers(0, cap, int(cap * load)), ks)
    run = min(cap // 3, 600)
    k0[:run // 2, :4] = rng.integers(cap - run // 4, cap + run // 4 + 1, run // 2, dtype=np.uint32).view(
        np.uint8).reshape(-1, 4)
    _insert(g, o, k0, rng)
    for _ in range(12):
        n = max(1, cap // 20)
        if len(o) + n > cap * 0.96:
            break
        k = _keys_at(rng, rng.integers(0, cap, n), ks)
        k[:n // 3, :4] = rng.integers(cap - 8, cap + 8, n // 3, dtype=np.uint32).view(np.uint8).reshape(-1, 4)
        k[n // 2:n // 2 + n // 6] = k[:n // 6]
        k[n - n // 8:] = k0[rng.integers(0, len(k0), n // 8)] if n // 8 else k[n:]
        _insert(g, o, k, rng)
        _same(g, o)


@pytest.mark.parametrize("load", [0.85, 0.9, 0.93, 0.96])
@pytest.mark.parametrize("n", [3, 40, 400])
def test_near_the_line(load, n):
    """Loads and sizes on both sides of the choice."""
    cap = 1 << 14
    rng = np.random.default_rng(n)
    g, o = gpu_map(cap, 32, 64), O.OracleMap(cap, 32, 64)
    _insert(g, o, _records(rng, int(cap * load), 32), rng)
    for _ in range(3):
        if len(o) + n > cap:
            break
        _insert(g, o, _records(rng, n, 32), rng)
        _same(g, o)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("bits,run", [(6, 20), (10, 300), (12, 900), (14, 700)])
@pytest.mark.parametrize("graph", [False, True])
def test_batched_inserts(shape, bits, run, graph):
    """Queued inserts into a table with a run longer than the component pass takes, before and after a remove."""
    import torch

    import flash_map as F

    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    start = cap - run // 2
    k0 = _keys_at(rng, (start + np.arange(run)) % cap, ks)
    _insert(g, o, k0, rng)
    queue, n = [], max(4, cap // 40)
    for kind in (F.batch.INSERT, F.batch.INSERT, F.batch.REMOVE, F.batch.INSERT):
        k = _keys_at(rng, rng.integers(0, cap, n), ks)
        k[:2, :4] = np.uint32(start).reshape(1).view(np.uint8)  # the whole run is their walk
        if kind == F.batch.REMOVE:
            k[2:] = k0[rng.integers(0, run, n - 2)]
        queue.append((kind, k, _records(rng, n, vs)))
    s = torch.cuda.Stream()
    dev = [(torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()) for _, k, v in queue]
    torch.cuda.synchronize()
    b = F.FlashMapBatch([F.BatchOp(kind, g, n, dk, dv if kind == F.batch.INSERT else None)
                         for (kind, _, _), (dk, dv) in zip(queue, dev)])
    if graph:
        b.capture(s)
    b.run(s)
    want = [(o.bulk_remove(k) if kind == F.batch.REMOVE else o.bulk_insert(k, v), 0) for kind, k, v in queue]
    assert b.wait() == want
    _same(g, o)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("bits,load,part,merged", [(13, 0.0, 4, False), (13, 0.6, 4, True), (16, 0.0, 16, False),
                                                   (16, 0.0, 8, False), (16, 0.85, 16, True), (16, 0.4, 2, True),
                                                   (20, 0.0, 16, False), (20, 0.85, 16, True), (20, 0.0, 2, True)])
def test_merges_where_they_pay(shape, bits, load, part, merged):
    """A merge is ten launches, a direct call four: large calls on either side of the line."""
    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits + part)
    from flash_map import _native
    import torch

    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    if load:
        k, v = _records(rng, int(cap * load), ks), _records(rng, int(cap * load), vs)
        assert g.bulk_insert(k, v) == o.bulk_insert(k, v)
    n = cap // part
    k, v = _records(rng, n, ks), _records(rng, n, vs)
    dk, dv = torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()
    torch.cuda.synchronize()
    before = _native.launch_count()
    assert g.bulk_insert_device(dk, dv, n) == o.bulk_insert(k, v)
    assert (_native.launch_count() - before >= 10) == merged
    _same(g, o)


def test_large_calls_at_high_load():
    """200,000 ops and more keep to the passes for tables without tombstones at every load, entries that are too long
    for the component pass among them."""
    cap = 1 << 22
    rng = np.random.default_rng(11)
    g, o = gpu_map(cap, 8, 8), O.OracleMap(cap, 8, 8)
    k = _records(rng, int(cap * 0.85), 8)
    assert g.bulk_insert(k, k) == o.bulk_insert(k, k)
    for n in (200_000, 199_999):
        k = _records(rng, n, 8)
        k[::50] = k[7]  # one key many times
        _insert(g, o, k, rng)
    _same(g, o)
