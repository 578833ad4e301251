"""Calls whose path follows from the table's history (no tombstones, none
reused), on tables whose history only the device knows: a batch that was still
queued when the table was cleared has left tombstones, and reused some, behind
the host's back.  The calls must find that out and give the oracle's table."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


def _records(rng, n, size):
    return rng.integers(0, 256, (n, size), dtype=np.uint8)


def _same(g, o):
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("claim", [False, True])
@pytest.mark.parametrize("bits,call", [(14, "insert 100"), (14, "insert 1300"), (12, "insert 300"), (12, "insert 20"),
                                       (9, "insert 20"), (14, "remove 400"), (9, "remove 40"), (14, "batch 100"),
                                       (14, "batch 5000"), (11, "batch 40"), (9, "batch 20")])
def test_call_after_a_clear_that_ran_ahead_of_a_batch(shape, claim, bits, call):
    import torch

    import flash_map as F

    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits * 2 + claim + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    n = cap // 2
    k, v = _records(rng, n, ks), _records(rng, n, vs)
    gone, late, lv = k[::3].copy(), _records(rng, cap // 8, ks), _records(rng, cap // 8, vs)
    s = torch.cuda.Stream()
    dev = [torch.from_numpy(x).cuda() for x in (k, v, gone, late, lv)]
    torch.cuda.synchronize()
    ops = [F.BatchOp(F.batch.INSERT, g, n, dev[0], dev[1]), F.BatchOp(F.batch.REMOVE, g, len(gone), dev[2])]
    if claim:
        ops.append(F.BatchOp(F.batch.INSERT, g, len(late), dev[3], dev[4]))
    b = F.FlashMapBatch(ops)
    b.capture(s)
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)  # the batch starts after the clear
    b.run(s)
    g.clear()
    b.wait()
    o.bulk_insert(k, v)
    o.bulk_remove(gone)
    if claim:
        o.bulk_insert(late, lv)
    _same(g, o)
    kind, m = call.split()
    m = int(m)
    if kind == "batch":  # queued without a graph: its passes are chosen when it runs
        q, w = _records(rng, m, ks), _records(rng, m, vs)
        q[: m // 3] = k[: m // 3]
        dq, dw = torch.from_numpy(q).cuda(), torch.from_numpy(w).cuda()
        torch.cuda.synchronize()
        b2 = F.FlashMapBatch([F.BatchOp(F.batch.INSERT, g, m, dq, dw)])
        b2.run(s)
        assert b2.wait() == [(o.bulk_insert(q, w), 0)]
    elif kind == "insert":
        q = np.concatenate([k[: m // 3], gone[: m // 3], _records(rng, m - m // 3 * 2, ks)])
        q = q[rng.permutation(len(q))]
        w = _records(rng, len(q), vs)
        assert g.bulk_insert(q, w) == o.bulk_insert(q, w)
    else:
        q = np.concatenate([k[rng.integers(0, n, m - 10)], late[:10]])
        assert g.bulk_remove(q) == o.bulk_remove(q)
    _same(g, o)
    assert g.bulk_remove(k[1::2]) == o.bulk_remove(k[1::2])
    more, mv = _records(rng, cap // 10, ks), _records(rng, cap // 10, vs)
    assert g.bulk_insert(more, mv) == o.bulk_insert(more, mv)
    _same(g, o)
