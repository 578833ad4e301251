"""Captured batches replayed on tables whose state has changed since the
capture, against the sequential oracle: results, lookups and whole layouts."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8), (32, 128)]


def _records(rng, n, size):
    return rng.integers(0, 256, (n, size), dtype=np.uint8)


def _same(g, o):
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)


class Queue:
    """A batch over tables of both shapes and its replay on oracles."""

    def __init__(self, tables, ops):
        import torch

        import flash_map as F

        self.ops, self.outs, self.stream = ops, [], torch.cuda.Stream()
        batch_ops = []
        for g, kind, k, v in ops:
            dk = torch.from_numpy(k).cuda()
            dv = torch.from_numpy(v).cuda() if v is not None else None
            ov = of = None
            if kind == F.batch.GET:
                ov = torch.zeros((len(k), g.value_size), dtype=torch.uint8, device="cuda")
                of = torch.zeros(len(k), dtype=torch.uint8, device="cuda")
            batch_ops.append(F.BatchOp(kind, g, len(k), dk, dv, ov, of))
            self.outs.append((ov, of))
        torch.cuda.synchronize()
        self.batch = F.FlashMapBatch(batch_ops)
        self.batch.capture(self.stream)

    def check(self, oracle_of):
        """One run against the oracles of the tables."""
        import flash_map as F

        self.batch.run(self.stream)
        got = self.batch.wait()
        for (g, kind, k, v), (ov, of), (res, status) in zip(self.ops, self.outs, got):
            o = oracle_of[g]
            assert status == 0
            if kind == F.batch.INSERT:
                assert res == o.bulk_insert(k, v)
            elif kind == F.batch.REMOVE:
                assert res == o.bulk_remove(k)
            else:
                ev, ef = o.bulk_get(k)
                assert np.array_equal(of.cpu().numpy().astype(bool), ef.astype(bool))
                assert np.array_equal(ov.cpu().numpy(), ev)
        for g, o in oracle_of.items():
            _same(g, o)


def _ops(rng, tables, cap, known):
    """Per table: a merging insert (over 1/16 of the slots), a small insert, a remove, an insert over its tombstones, a
    lookup."""
    import flash_map as F

    ops = []
    for g in tables:
        a, b, c = (_records(rng, n, g.key_size) for n in (cap // 10, 300, 200))
        ops += [(g, F.batch.INSERT, a, _records(rng, len(a), g.value_size)),
                (g, F.batch.INSERT, b, _records(rng, len(b), g.value_size)),
                (g, F.batch.REMOVE, np.concatenate([a[::7], known[g][::5], _records(rng, 50, g.key_size)]), None),
                (g, F.batch.INSERT, c, _records(rng, len(c), g.value_size)),
                (g, F.batch.GET, np.concatenate([a, known[g]]), None)]
    return ops


@pytest.mark.parametrize("by", ["call", "batch"])
def test_replay_after_the_scratch_has_grown(by):
    """A larger plain call, or another batch's, moves a table's scratch between the capture and the replay: the graph
    must not use the old addresses."""
    import flash_map as F

    cap = 1 << 14
    rng = np.random.default_rng(len(by))
    tables = [gpu_map(cap, ks, vs) for ks, vs in SHAPES]
    saved = [gpu_map(cap, ks, vs) for ks, vs in SHAPES]
    known, start = {}, {}
    for g, b in zip(tables, saved):
        k, v = _records(rng, 1000, g.key_size), _records(rng, 1000, g.value_size)
        b.bulk_insert(k, v)
        g.copy_from(b)
        known[g], start[g] = k, (k, v)

    def oracles():
        m = {}
        for g in tables:
            m[g] = O.OracleMap(cap, g.key_size, g.value_size)
            m[g].bulk_insert(*start[g])
        return m

    q = Queue(tables, _ops(rng, tables, cap, known))
    q.check(oracles())
    for n in (6_000, 12_000):  # each above the scratch of the calls before it
        if by == "call":
            for g in tables:
                g.bulk_insert(_records(rng, n, g.key_size), _records(rng, n, g.value_size))
                g.bulk_remove(_records(rng, n, g.key_size))
        else:
            big = [(g, F.batch.INSERT, _records(rng, n, g.key_size), _records(rng, n, g.value_size)) for g in tables]
            other = Queue(tables, big)
            for g, b in zip(tables, saved):
                g.copy_from(b, other.stream)
            other.batch.run(other.stream)
            other.batch.wait()
        for _ in range(2):
            for g, b in zip(tables, saved):
                g.copy_from(b, q.stream)
            q.check(oracles())


@pytest.mark.parametrize("what", ["fits", "hot key", "hot home"])
def test_replay_on_another_history(what):
    """A graph planned for tables without tombstones, with a merged insert (one that the merge takes, or leaves for its
    hot key or hot home), replayed without a rollback: from the second run on the tables hold tombstones, and the third
    finds them reused."""
    import flash_map as F

    cap = 1 << 14
    rng = np.random.default_rng(len(what))
    tables = [gpu_map(cap, ks, vs) for ks, vs in SHAPES]
    ops = []
    for g in tables:
        k = _records(rng, 7000, g.key_size)
        if what == "hot key":
            k[rng.choice(7000, 60, replace=False)] = k[0]
        elif what == "hot home":
            k[rng.choice(7000, 60, replace=False), :4] = k[0, :4]
        small, late = _records(rng, 300, g.key_size), _records(rng, 200, g.key_size)
        small[:100] = k[:100]
        ops += [(g, F.batch.INSERT, k, _records(rng, 7000, g.value_size)),
                (g, F.batch.INSERT, small, _records(rng, 300, g.value_size)),
                (g, F.batch.REMOVE, np.concatenate([k[::3], small[::2], _records(rng, 100, g.key_size)]), None),
                (g, F.batch.INSERT, late, _records(rng, 200, g.value_size)),
                (g, F.batch.REMOVE, np.concatenate([late[::2], k[1::5]]), None),
                (g, F.batch.GET, np.concatenate([k, small, late]), None)]
    q = Queue(tables, ops)
    oracles = {g: O.OracleMap(cap, g.key_size, g.value_size) for g in tables}
    for _ in range(4):
        q.check(oracles)
    for g in tables:  # and from cleared tables again
        g.clear()
        oracles[g].clear()
    q.check(oracles)
