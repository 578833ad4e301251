"""Small inserts into large tables without tombstones (updates told apart,
components and long walks done at once) and lookups of run-time record sizes,
against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


def keys_at(rng, homes, ks, kinds=1 << 31):
    """Keys with the given home slots (identity hash); few kinds make repeats."""
    k = np.zeros((len(homes), ks), np.uint8)
    k[:, :4] = np.asarray(homes, np.uint32).view(np.uint8).reshape(-1, 4)
    k[:, 4:8] = rng.integers(0, kinds, len(homes), dtype=np.uint32).view(np.uint8).reshape(-1, 4)
    return k


def both(g, o, k, vs, rng):
    v = rng.integers(0, 256, (len(k), vs), dtype=np.uint8)
    assert g.bulk_insert(k, v) == o.bulk_insert(k, v)


def same(g, o):
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128), (32, 64), (32, 32), (8, 32)])
@pytest.mark.parametrize("run", [10, 47, 48, 49, 87, 95, 96, 97, 130, 500, 520, 1500])
def test_walks_and_components(shape, run):
    """Runs of OCCUPIED slots of chosen lengths (one entry per home, and several), each met by: one op at its start
    (a walk of the whole run, every entry evicted), a few ops at its start, middle and end, ops with one key several
    times, and updates; the last run goes round the end of the table."""
    ks, vs = shape
    cap = 1 << 16
    rng = np.random.default_rng(run + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    starts = [(run * 3 + 5) * i for i in range(6)] + [cap - run // 2]
    homes = []
    for i, s in enumerate(starts):
        if i % 2 == 0:
            homes += [(s + x) % cap for x in range(run)]             # one entry per home
        else:
            homes += [(s + x // 3 * 3) % cap for x in range(run)]    # threes
    both(g, o, keys_at(rng, homes, ks), vs, rng)
    same(g, o)
    for ops in ([0], [0, 0], [0, run // 2], [0, run // 2, run - 1, run, run + 1], [run - 2] * 5, [0, 1, 2] * 11):
        k = keys_at(rng, [(s + x) % cap for s in starts for x in ops], ks, kinds=3 if len(ops) > 4 else 1 << 31)
        both(g, o, k, vs, rng)
        same(g, o)
    k = keys_at(rng, [starts[0]] * 200 + [starts[1] + run // 2] * 70, ks)  # more than a warp gathers
    both(g, o, k, vs, rng)
    both(g, o, np.concatenate([k[:50], k[:50], keys_at(rng, homes[:100], ks)]), vs, rng)  # updates, twice, and new keys
    same(g, o)


@pytest.mark.parametrize("shape", [(16, 16), (12, 20), (5, 3), (3, 32), (4, 0), (256, 256), (64, 1)])
@pytest.mark.parametrize("mode", [0, 1])
def test_run_time_sizes(shape, mode):
    """Lookups of run-time record sizes: odd counts, values of 16, 4 and 1 byte pieces, no values, buffers off the
    16-byte grid."""
    import torch

    ks, vs = shape
    cap = 1 << 10
    rng = np.random.default_rng(ks * 31 + vs)
    g, o = gpu_map(cap, ks, vs, mode), O.OracleMap(cap, ks, vs, mode)
    k = rng.integers(0, 256, (700, ks), dtype=np.uint8)
    both(g, o, k, vs, rng)
    r = k[::5].copy()
    assert g.bulk_remove(r) == o.bulk_remove(r)
    for n in (1, 31, 32, 33, 1000):
        q = np.concatenate([k, rng.integers(0, 256, (300, ks), dtype=np.uint8)])[rng.integers(0, 1000, n)]
        ov, of = o.bulk_get(q)
        for a, b in zip(g.bulk_get(q), (ov, of)):
            assert np.array_equal(a, b)
        for shift in (0, 4, 1):
            dk = torch.zeros(n * ks + 16, dtype=torch.uint8, device="cuda")
            dv = torch.full((n * vs + 32,), 7, dtype=torch.uint8, device="cuda")
            df = torch.zeros(n, dtype=torch.uint8, device="cuda")
            dk[shift:shift + n * ks] = torch.from_numpy(q.reshape(-1)).cuda()
            g.bulk_get_device(dk[shift:], n, dv[shift:], df)
            torch.cuda.synchronize()
            assert np.array_equal(dv[shift:shift + n * vs].cpu().numpy().reshape(n, vs), ov)
            assert np.array_equal(df.cpu().numpy().astype(bool), of.astype(bool))
            assert (dv[:shift] == 7).all() and (dv[shift + n * vs:] == 7).all()  # nothing beside the records
