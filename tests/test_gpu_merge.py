"""Inserts that are large beside their table (merged into a table without
tombstones in one pass) and removes in any order (no tombstone reused yet),
against the oracle: counts, lookups and the whole layout, bit for bit."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8), (32, 128), (32, 64), (32, 32), (8, 32)]


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


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bits", [10, 11, 15])
@pytest.mark.parametrize("kinds", [1, 3, 1 << 31])
def test_merge(shape, bits, kinds):
    """Calls from a 16th of the table to most of it, up to a load of about 0.97; repeats and updates with few kinds;
    runs that go round the end of the table."""
    ks, vs = shape
    cap = 1 << bits
    rng = np.random.default_rng(bits * 7 + kinds % 5 + ks)
    for part in (0.0626, 0.2, 0.5, 0.95):
        g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
        n = int(cap * part)
        for _ in range(int(0.97 / part)):
            k = keys_of(rng, n, ks, cap if kinds > 3 else cap * 2, kinds)
            if kinds == 1 << 31:
                k[: n // 3, :4] = rng.integers(cap - cap // 8, cap + cap // 8, n // 3, dtype=np.uint32).view(
                    np.uint8).reshape(-1, 4)  # a crowded stretch across the end
            v = rng.integers(0, 256, (n, vs), dtype=np.uint8)
            if len(o) + n > cap:
                break
            assert g.bulk_insert(k, v) == o.bulk_insert(k, v)
        same(g, o)
        q = np.concatenate([k, keys_of(rng, n, ks, cap, kinds)])
        for a, b in zip(g.bulk_get(q), o.bulk_get(q)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128)])
@pytest.mark.parametrize("what", ["hot key", "hot home", "long pool", "full"])
def test_merge_left_to_others(shape, what):
    """Calls that outgrow a bound of the merge run whole on the other paths, updates of the call included."""
    ks, vs = shape
    cap = 1 << 13
    rng = np.random.default_rng(len(what) + ks)
    g, o = gpu_map(cap, ks, vs), O.OracleMap(cap, ks, vs)
    n = cap // 4
    old = keys_of(rng, n, ks, cap, 1 << 31)
    k = keys_of(rng, n, ks, cap, 1 << 31)
    if what == "hot key":
        k[rng.choice(n, 40, replace=False)] = k[0]  # a new key 40 times
    elif what == "hot home":
        old[:70, :4] = old[0, :4]  # 70 stored entries of one home
        k[:40, :4] = old[0, :4]    # and more ops on it
    elif what == "long pool":
        k[:1500, :4] = rng.integers(0, 100, 1500, dtype=np.uint32).view(np.uint8).reshape(-1, 4)
    else:
        old, k = keys_of(rng, cap // 2, ks, cap, 1 << 31), keys_of(rng, cap // 2, ks, cap, 1 << 31)
    k[5:25] = old[5:25]  # updates
    for kk in (old, k):
        v = rng.integers(0, 256, (len(kk), vs), dtype=np.uint8)
        if len(o) + len(kk) > cap:
            kk, v = kk[: cap - len(o)], v[: cap - len(o)]
        assert g.bulk_insert(kk, v) == o.bulk_insert(kk, v)
        same(g, o)


@pytest.mark.parametrize("shape", [(8, 8), (32, 128), (12, 20)])
@pytest.mark.parametrize("bits", [3, 9, 14])
@pytest.mark.parametrize("load", [0.5, 0.9, 1.0])
def test_remove_any_order(shape, bits, load):
    """Removes with repeats and absent keys before any tombstone is reused, then an insert over the tombstones (the
    merge and the any-order removes no longer apply), removes after it, and the same from a cleared table."""
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
