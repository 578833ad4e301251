"""The closed forms behind the merging insert and the any-order removes, on
the sequential oracle (CPU): a model of what a whole insert call does to a
table without tombstones gives the oracle's table, and removes in a shuffled
order give the same table and count while no insert has reused a tombstone."""
import heapq

import numpy as np
import pytest

import oracle as O


def merged(cap, flags, keys, vals, K, V):
    """The table after inserting (K[j], V[j]) in order, without running the ops: (flags, keys, values, new keys)."""
    mask = cap - 1
    occ, dist = (flags & 15) == 1, (flags >> 4).astype(int)
    where = {bytes(keys[x]): x for x in range(cap) if occ[x]}
    first, last = {}, {}
    vals = vals.copy()
    for j, k in enumerate(map(bytes, K)):
        if k in where:
            vals[where[k]] = V[j]  # an update: the last one stays
        else:
            first.setdefault(k, j)
            last[k] = j
    at = {}  # home -> its new ops in index order
    for j in sorted(first.values()):
        at.setdefault(int.from_bytes(bytes(K[j][:8]), "little") & mask, []).append(j)
    carry, c = [0] * cap, 0
    for turn in range(2):  # the second time round from the right start
        for s in range(cap):
            carry[s] = c
            c = max(0, c + len(at.get(s, ())) - (0 if occ[s] else 1))
    start = next((s for s in range(cap) if carry[s] == 0), None)
    if start is None:
        return None  # no EMPTY slot left
    rank, pool = {}, []
    for o in range(cap):
        s = (start + o) & mask
        for a in at.get(s, ()):
            rank[a] = sum(p < a for p in pool)
        for a in at.get(s, ()):
            heapq.heappush(pool, a)
        if not occ[s] and pool:
            heapq.heappop(pool)

    def place(h, pos, m, mine):
        seen, size = 0, m
        for a in at.get(h, ()):
            if pos is not None and size:
                pos = (pos - (rank[a] - seen)) % size
            seen = rank[a]
            if a == mine:
                pos = size
            size += 1
        return (pos - (carry[h] - seen)) % size

    f2, k2, v2 = flags.copy(), keys.copy(), vals.copy()

    def put(dst, h, key, val):
        f2[dst] = ((dst - h) & mask) << 4 | 1
        k2[dst], v2[dst] = key, val

    for x in np.flatnonzero(occ):
        h = int(x - dist[x]) & mask
        i, m = 0, 1
        while i < dist[x] and flags[(x - i - 1) & mask] == (dist[x] - i - 1) << 4 | 1:
            i += 1
        while flags[(x + m) & mask] == (dist[x] + m) << 4 | 1:
            m += 1
        if carry[h]:
            put(int(x - i + carry[h] + place(h, i, i + m, None)) & mask, h, keys[x], vals[x])
    for h, ops in at.items():
        p = m = 0
        while occ[(h + p) & mask] and dist[(h + p) & mask] >= p:
            m += dist[(h + p) & mask] == p
            p += 1
        for a in ops:
            put((h + p - m + carry[h] + place(h, None, m, a)) & mask, h, K[a], V[last[bytes(K[a])]])
    return f2, k2, v2, len(first)


def narrow_keys(rng, n, cap, kinds):
    k = np.zeros((n, 8), np.uint8)
    k[:, :2] = rng.integers(0, cap, n, dtype=np.uint16).view(np.uint8).reshape(n, 2)
    k[:, 4] = rng.integers(0, kinds, n)
    return k


@pytest.mark.parametrize("kinds", [1, 2, 40])
@pytest.mark.parametrize("bits", [3, 5, 8])
def test_merge_is_the_sequential_insert(bits, kinds):
    cap = 1 << bits
    rng = np.random.default_rng(bits * 3 + kinds)
    for _ in range(40):
        m = O.OracleMap(cap, 8, 8, 0)
        for _ in range(4):
            n = int(rng.integers(1, cap // 2 + 1))
            if len(m) + n > cap:
                break
            f, k, v = m.snapshot()
            K, V = narrow_keys(rng, n, cap, kinds), rng.integers(0, 256, (n, 8), dtype=np.uint8)
            want = merged(cap, f, k, v, K, V)
            new = m.bulk_insert(K, V)
            if want is None:
                continue
            f2, k2, v2 = m.snapshot()
            occ = (f2 & 15) == 1
            assert new == want[3] and np.array_equal(f2, want[0])
            assert np.array_equal(k2[occ], want[1][occ]) and np.array_equal(v2[occ], want[2][occ])


@pytest.mark.parametrize("load", [0.5, 0.9, 1.0])
def test_removes_commute_without_a_reused_tombstone(load):
    cap = 1 << 9
    for seed in range(10):
        rng = np.random.default_rng(seed)
        a, b = O.OracleMap(cap, 8, 8, 0), O.OracleMap(cap, 8, 8, 0)
        k = narrow_keys(rng, int(cap * load), cap, 9)
        for m in (a, b):
            m.bulk_insert(k, k)
        for _ in range(3):
            r = np.concatenate([k[rng.integers(0, len(k), 100)], narrow_keys(rng, 50, cap, 9)])
            assert a.bulk_remove(r) == b.bulk_remove(r[rng.permutation(len(r))])
            for x, y in zip(a.snapshot(), b.snapshot()):
                assert np.array_equal(x, y)
