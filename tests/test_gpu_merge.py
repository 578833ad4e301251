"""Removes in any order (no tombstone reused yet) against the oracle: counts
and the whole layout, bit for bit."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


def keys_of(rng, n, ks, homes, kinds):
    """n keys over `homes` low words and `kinds` values of the second word: few of either make groups and repeats."""
    k = np.zeros((n, ks), np.uint8)
    k[:, :4] = rng.integers(0, homes, n, dtype=np.uint32).view(np.uint8).reshape(n, 4)
    k[:, 4:8] = rng.integers(0, kinds, n, dtype=np.uint32).view(np.uint8).reshape(n, 4)
    return k


def same(g, o):
    assert g.len() == len(o)
    for a, b in zip(g.snapshot(), o.snapshot()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128), (12, 20)])
@pytest.mark.parametrize("bits", [3, 9, 14])
@pytest.mark.parametrize("load", [0.5, 0.9, 1.0])
def test_remove_any_order(shape, bits, load):
    """Removes with repeats and absent keys before any tombstone is reused, then an insert over the tombstones (the
    any-order removes no longer apply), removes after it, and the same from a cleared table."""
    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    for _ in range(2):
        k = keys_of(rng, int(cap * load), ks, cap, 4)
        v = rng.integers(0, 256, (len(k), vs), dtype=np.uint8)
        assert g.bulk_insert(k, v) == o.bulk_insert(k, v)
        for part in (3, 2):
            r = np.concatenate([k[rng.integers(0, len(k), cap // part)], keys_of(rng, cap // 8 + 1, ks, cap, 4)])
            assert g.bulk_remove(r) == o.bulk_remove(r)
            same(g, o)
        m = cap - len(o)
        k2, v2 = keys_of(rng, m, ks, cap, 4), rng.integers(0, 256, (m, vs), dtype=np.uint8)
        assert g.bulk_insert(k2, v2) == o.bulk_insert(k2, v2)
        same(g, o)
        r = np.concatenate([k, k2])[rng.integers(0, len(k) + m, cap)]
        assert g.bulk_remove(r) == o.bulk_remove(r)
        same(g, o)
        g.clear()
        o.clear()
