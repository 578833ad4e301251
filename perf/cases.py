"""Workloads of the FlashMap B200 backend, as a program that uses it runs them.

Each case is a dict of plain values; prepare() builds what such a program holds
before the call (tables, keys, buffers, a batch plan), run() makes one pass
through the public API of `flash_map`, exact() says what a pass returns, from
the inputs alone.  Passes start from the same table contents every time: a
cleared table, a checkpoint rolled back on the device, or updates that leave
the table as it is.

Kinds:
  get     device lookups on a filled table
  load    clear, insert calls of `call` keys, lookups of the last call's keys,
          and (with `removes`) a remove and the lookups again
  step    clear, the fill in calls of `call` pairs, a mixed lookup, a remove
  upsert  new values for present keys, then their lookup
  churn   rollback to a checkpoint, then remove / insert / remove / lookup
  batch   rollback of several tables, then one queued batch over them
  host    clear, one insert and one lookup through host arrays
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-map_b200"))
import flash_map as F  # noqa: E402
from flash_map.batch import GET, INSERT, REMOVE  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # one request's keys against a served account table: all latency
        {"name": "get_256", "kind": "get", "k": 32, "v": 128, "bits": 20, "load": 0.75, "n": 256, "hit": 0.8,
         "zipf": 0.9, "murmur": False},
        # the account shape at its stated load factor, half of the queries absent
        {"name": "get_account", "kind": "get", "k": 32, "v": 128, "bits": 24, "load": 0.8, "n": 4_000_000, "hit": 0.5,
         "zipf": 0.0, "murmur": False},
        # skewed lookups (Zipf 1.1, 10% absent) on a nearly full u64 table
        {"name": "get_u64_zipf", "kind": "get", "k": 8, "v": 8, "bits": 25, "load": 0.9, "n": 5_000_000, "hit": 0.9,
         "zipf": 1.1, "murmur": False},
        # a record size without a kernel of its own (16-byte ids to 16-byte records), hashed keys, a ragged count
        {"name": "get_id16", "kind": "get", "k": 16, "v": 16, "bits": 22, "load": 0.7, "n": 999_983, "hit": 0.7,
         "zipf": 0.0, "murmur": True},
        # the smallest of the stated insert sizes: 1K pairs into a table of four times as many
        {"name": "load_1k", "kind": "load", "k": 32, "v": 128, "bits": 12, "n": 1000, "call": 1000, "dup": 0.0,
         "removes": 0},
        # 700K distinct u64 pairs in one call, lookups, a remove of 100K, lookups (the plain small configuration)
        {"name": "load_u64_700k", "kind": "load", "k": 8, "v": 8, "bits": 20, "n": 700_000, "call": 700_000, "dup": 0.0,
         "removes": 100_000},
        # large duplicate-heavy calls (4M keys, 20% repeats) up to about load 0.76
        {"name": "load_u64_4m", "kind": "load", "k": 8, "v": 8, "bits": 24, "n": 16_000_000, "call": 4_000_000,
         "dup": 0.2, "removes": 0},
        # the whole account step: 135 calls of 100K pairs to load 0.8, 8M lookups, a tenth removed
        {"name": "step_account", "kind": "step", "k": 32, "v": 128, "bits": 24, "load": 0.8, "call": 100_000,
         "gets": 8_000_000},
        # a block of account updates: every key present, values overwritten and read back
        {"name": "upsert_account", "kind": "upsert", "k": 32, "v": 128, "bits": 22, "load": 0.7, "n": 100_000},
        # a table that lives: removes and inserts over tombstones from a checkpoint
        {"name": "churn_account", "kind": "churn", "k": 32, "v": 128, "bits": 21, "load": 0.7, "n": 150_000},
        # queued operations of uneven sizes over 16 tables, replayed from a CUDA graph
        {"name": "batch_16", "kind": "batch", "tables": 16, "ops": 64, "lo_bits": 14, "hi_bits": 20, "max_n": 200_000,
         "plan": 5},
        # a million pairs inserted and looked up through host arrays
        {"name": "host_u64_1m", "kind": "host", "k": 8, "v": 8, "bits": 21, "n": 1_000_000},
    ]


SHAPES = [(32, 128), (8, 8), (32, 64), (32, 32), (8, 32), (16, 16)]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["get", "get", "load", "load", "step", "upsert", "churn", "batch", "host"])
    k, v = rng.choice(SHAPES)
    if kind == "get":
        return {"kind": kind, "k": k, "v": v, "bits": rng.randint(16, 24), "load": round(rng.uniform(0.3, 0.9), 3),
                "n": _log(rng, 200, 5_000_000) | 1, "hit": round(rng.uniform(0.3, 1.0), 2),
                "zipf": rng.choice([0.0, 0.9, 1.1]), "murmur": rng.random() < 0.3}
    if kind == "load":
        k, v = rng.choice(SHAPES[:5])
        bits = rng.randint(12, 23)
        n = int((1 << bits) * rng.uniform(0.2, 0.75)) | 1
        return {"kind": kind, "k": k, "v": v, "bits": bits, "n": n, "call": max(1000, n // rng.choice([1, 1, 2, 5])),
                "dup": rng.choice([0.0, 0.0, 0.2]), "removes": rng.choice([0, n // 7])}
    if kind == "step":
        k, v = rng.choice(SHAPES[:5])
        bits = rng.randint(18, 22)
        return {"kind": kind, "k": k, "v": v, "bits": bits, "load": round(rng.uniform(0.4, 0.85), 3),
                "call": _log(rng, max(10_000, (1 << bits) // 50), 200_000), "gets": _log(rng, 10_000, 4_000_000)}
    if kind == "upsert":
        bits = rng.randint(16, 23)
        return {"kind": kind, "k": k, "v": v, "bits": bits, "load": round(rng.uniform(0.4, 0.85), 3),
                "n": _log(rng, 300, min(500_000, 1 << (bits - 2))) | 1}
    if kind == "churn":
        k, v = rng.choice(SHAPES[:5])
        bits = rng.randint(16, 21)
        return {"kind": kind, "k": k, "v": v, "bits": bits, "load": round(rng.uniform(0.4, 0.8), 3),
                "n": _log(rng, 500, (1 << bits) // 12) | 1}
    if kind == "batch":
        return {"kind": kind, "tables": rng.randint(4, 20), "ops": rng.randint(16, 64), "lo_bits": 14,
                "hi_bits": rng.randint(16, 20), "max_n": _log(rng, 20_000, 200_000), "plan": rng.randint(1, 1000)}
    n = _log(rng, 10_000, 1_000_000) | 1
    return {"kind": kind, "k": k, "v": v, "bits": max(12, (2 * n).bit_length()), "n": n}


# -- inputs -------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _bytes(n, size, g):
    """n records of uniform random bytes."""
    if size % 8 == 0:
        return torch.randint(-(1 << 63), (1 << 63) - 1, (n, size // 8), dtype=torch.int64, device=DEV,
                             generator=g).view(torch.uint8).view(n, size)
    return torch.randint(0, 256, (n, size), dtype=torch.uint8, device=DEV, generator=g)


def _picks(n, m, zipf, g):
    """m indices below n, uniform or Zipf(zipf) by rank (the ranks are the insertion order, which is random)."""
    if not zipf:
        return torch.randint(0, n, (m,), device=DEV, generator=g)
    u = torch.rand(m, dtype=torch.float64, device=DEV, generator=g)
    e = 1.0 - zipf
    r = (1.0 + u * ((n + 1.0) ** e - 1.0)) ** (1.0 / e)
    return (r.long() - 1).clamp_(0, n - 1)


def _queries(keys, m, hit, zipf, g):
    """m queries, a share `hit` of them present: the records, and per query its index in keys or -1."""
    idx = _picks(len(keys), m, zipf, g)
    idx[torch.rand(m, device=DEV, generator=g) >= hit] = -1
    q = _bytes(m, keys.shape[1], g)
    return torch.where((idx >= 0)[:, None], keys[idx.clamp(min=0)], q), idx


def _answer(vals, idx):
    """Values and found bytes of the queries idx (-1: absent)."""
    return torch.where((idx >= 0)[:, None], vals[idx.clamp(min=0)], 0), (idx >= 0).to(torch.uint8)


def _table(case, murmur=False, bits=None):
    return F.FlashMap(1 << (bits or case["bits"]), case["k"], case["v"],
                      F.HashStrategy.Murmur3 if murmur else F.HashStrategy.Identity)


def _fill(m, keys, vals):
    """Pairs in calls of 100K keys, fewer calls for the larger tables."""
    step = max(100_000, -(-len(keys) // 64))
    for b in range(0, len(keys), step):
        c = min(step, len(keys) - b)
        m.bulk_insert_device(keys[b:b + c], vals[b:b + c], c)


def _inputs(case, seed):
    """The tensors of a case, from its seed alone."""
    g, kind = _gen(seed), case["kind"]
    k, v = case.get("k"), case.get("v")
    cap = 1 << case["bits"] if "bits" in case else 0
    if kind == "get":
        n = int(cap * case["load"])
        keys, vals = _bytes(n, k, g), _bytes(n, v, g)
        q, idx = _queries(keys, case["n"], case["hit"], case["zipf"], g)
        return {"keys": keys, "vals": vals, "q": q, "idx": idx}
    if kind == "load":
        n, call = case["n"], case["call"]
        distinct = _bytes(n, k, g)
        ids = torch.arange(n, device=DEV)
        if case["dup"]:  # repeats of keys of the same call, anywhere in it
            at = torch.rand(n, device=DEV, generator=g) < case["dup"]
            lo = ids // call * call
            span = (lo + call).clamp(max=n) - lo
            r = lo + (torch.rand(n, device=DEV, generator=g, dtype=torch.float64) * span).long()
            ids = torch.where(at, r, ids)
        last = (n - 1) // call * call
        rem = torch.randperm(n, device=DEV, generator=g)[:case["removes"]]
        absent = _bytes(n - last, k, g)
        return {"keys": distinct[ids].contiguous(), "ids": ids, "vals": _bytes(n, v, g), "last": last, "rem": rem,
                "q": torch.cat([distinct[ids[last:]], absent]).contiguous()}
    if kind == "step":
        n = int(cap * case["load"])
        keys, vals = _bytes(n, k, g), _bytes(n, v, g)
        q, idx = _queries(keys, case["gets"], 0.5, 0.0, g)
        rem = keys[torch.randperm(n, device=DEV, generator=g)[:n // 10]].contiguous()
        return {"keys": keys, "vals": vals, "q": q, "idx": idx, "rem": rem}
    if kind == "upsert":
        n = int(cap * case["load"])
        keys, vals = _bytes(n, k, g), _bytes(n, v, g)
        up = keys[torch.randperm(n, device=DEV, generator=g)[:case["n"]]].contiguous()
        return {"keys": keys, "vals": vals, "up": up, "new": _bytes(case["n"], v, g)}
    if kind == "churn":
        n, m = int(cap * case["load"]), case["n"]
        keys, vals = _bytes(n, k, g), _bytes(n, v, g)
        gone = torch.randperm(n, device=DEV, generator=g)[:2 * m]
        fresh, fvals = _bytes(m, k, g), _bytes(m, v, g)
        q = torch.cat([keys[torch.randint(0, n, (m,), device=DEV, generator=g)], fresh])
        return {"keys": keys, "vals": vals, "rem1": keys[gone[:m]].contiguous(), "fresh": fresh, "fvals": fvals,
                "rem2": torch.cat([keys[gone[m:]], fresh[:m // 4]]).contiguous(), "q": q.contiguous()}
    raise ValueError(kind)


# -- state and passes ---------------------------------------------------------
def _outs(m, v):
    return torch.empty((m, v), dtype=torch.uint8, device=DEV), torch.empty(m, dtype=torch.uint8, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "host":
        r = np.random.default_rng(seed)
        keys = r.integers(0, 256, (case["n"], case["k"]), dtype=np.uint8)
        vals = r.integers(0, 256, (case["n"], case["v"]), dtype=np.uint8)
        return {"case": case, "m": _table(case), "keys": keys, "vals": vals, "q": keys[r.permutation(case["n"])]}
    s = _inputs(case, seed)
    s["case"] = case
    s["m"] = m = _table(case, case.get("murmur", False))
    v = case["v"]
    if kind in ("get", "upsert", "churn"):
        _fill(m, s.pop("keys"), s.pop("vals"))
    if kind == "churn":
        s["live"] = _table(case)
    if kind == "upsert":
        s["ov"], s["of"] = _outs(case["n"], v)
    else:
        s["ov"], s["of"] = _outs(len(s["q"]), v)
    if kind == "load" and case["removes"]:
        s["remk"] = s["keys"][s["rem"]].contiguous()
        s["ov2"], s["of2"] = _outs(len(s["q"]), v)
    torch.cuda.synchronize()
    return s


def _prepare_batch(case, seed):
    """Tables of log-uniform capacities and loads 0.5 to 0.8, alternating u64 and account records; 40% lookups, 40%
    inserts, 20% removes of log-uniform sizes, half of the looked-up and removed keys present."""
    r = np.random.default_rng(case["plan"])  # which tables and ops there are; the seed makes their records
    g = _gen(seed)
    live, saved, known, room = [], [], [], []
    for i in range(case["tables"]):
        c = {"k": 8, "v": 8} if i % 2 == 0 else {"k": 32, "v": 128}
        bits = int(r.integers(case["lo_bits"], case["hi_bits"] + 1))
        m, b = _table(c, bits=bits), _table(c, bits=bits)
        n = int((1 << bits) * r.uniform(0.5, 0.8))
        keys, vals = _bytes(n, c["k"], g), _bytes(n, c["v"], g)
        _fill(b, keys, vals)
        m.copy_from(b)
        live.append(m), saved.append(b), known.append(keys), room.append(int((1 << bits) * 0.88) - n)
    ops, outs = [], []
    for _ in range(case["ops"]):
        t = int(r.integers(case["tables"]))
        m = live[t]
        kind = int(r.choice([GET, INSERT, REMOVE], p=[0.4, 0.4, 0.2]))
        n = int(np.exp(r.uniform(np.log(256), np.log(case["max_n"]))))
        if kind == INSERT:  # up to load 0.88
            n = min(n, room[t])
            if n < 256:
                kind, n = GET, 256
            else:
                room[t] -= n
        if kind == INSERT:
            ops.append(F.BatchOp(kind, m, n, _bytes(n, m.key_size, g), _bytes(n, m.value_size, g)))
            continue
        if kind == REMOVE:
            n = min(n, m.len() // 4)
        q, _idx = _queries(known[t], n, 0.5, 0.0, g)
        if kind == GET:
            ov, of = _outs(n, m.value_size)
            outs.append((ov, of))
            ops.append(F.BatchOp(kind, m, n, q, None, ov, of))
        else:
            ops.append(F.BatchOp(kind, m, n, q))
    stream = torch.cuda.Stream(DEV)
    torch.cuda.synchronize()
    b = F.FlashMapBatch(ops)
    s = {"case": case, "live": live, "saved": saved, "outs": outs, "stream": stream, "batch": b}
    _roll(s)
    b.run(stream)
    b.wait()
    _roll(s)
    b.capture(stream)
    return s


def _roll(s):
    for m, b in zip(s["live"], s["saved"]):
        m.copy_from(b, s["stream"])


def run(s):
    case = s["case"]
    kind = case["kind"]
    m = s.get("m")
    if kind == "get":
        m.bulk_get_device(s["q"], case["n"], s["ov"], s["of"])
        return s["ov"], s["of"]
    if kind == "load" or kind == "step":
        # clear() works on the table's own stream: lookups still queued on the caller's have to be done
        torch.cuda.current_stream().synchronize()
        m.clear()
        keys, vals, call = s["keys"], s["vals"], case["call"]
        new = []
        for b in range(0, len(keys), call):
            c = min(call, len(keys) - b)
            new.append(m.bulk_insert_device(keys[b:b + c], vals[b:b + c], c))
        m.bulk_get_device(s["q"], len(s["q"]), s["ov"], s["of"])
        out = [np.array(new, dtype=np.int64), s["ov"], s["of"]]
        if kind == "step":
            out.append(m.bulk_remove_device(s["rem"], len(s["rem"])))
        elif case["removes"]:
            out.append(m.bulk_remove_device(s["remk"], case["removes"]))
            m.bulk_get_device(s["q"], len(s["q"]), s["ov2"], s["of2"])
            out += [s["ov2"], s["of2"]]
        return out
    if kind == "upsert":
        new = m.bulk_insert_device(s["up"], s["new"], case["n"])
        m.bulk_get_device(s["up"], case["n"], s["ov"], s["of"])
        return new, s["ov"], s["of"]
    if kind == "churn":
        t, n = s["live"], case["n"]
        t.copy_from(m)
        a = t.bulk_remove_device(s["rem1"], n)
        b = t.bulk_insert_device(s["fresh"], s["fvals"], n)
        c = t.bulk_remove_device(s["rem2"], len(s["rem2"]))
        t.bulk_get_device(s["q"], len(s["q"]), s["ov"], s["of"])
        return a, b, c, s["ov"], s["of"]
    if kind == "batch":
        _roll(s)
        s["batch"].run(s["stream"])
        res = np.array(s["batch"].wait(), dtype=np.int64)
        return [res, torch.cat([o[0].view(-1) for o in s["outs"]]), torch.cat([o[1] for o in s["outs"]])]
    m.clear()
    new = m.bulk_insert(s["keys"], s["vals"])
    vals, found = m.bulk_get(s["q"])
    return new, vals, found


def exact(case, seed):
    """What a pass returns, from its inputs (keys are distinct but for the repeats that the inputs place).  None where
    the answer depends on the table's history (inserts over tombstones)."""
    kind = case["kind"]
    if kind in ("churn", "batch"):
        return None
    if kind == "host":
        s = prepare(case, seed)
        order = {bytes(x): i for i, x in enumerate(s["keys"])}
        idx = np.array([order[bytes(x)] for x in s["q"]])
        return case["n"], s["vals"][idx], np.ones(case["n"], bool)
    s = _inputs(case, seed)
    if kind == "get":
        return _answer(s["vals"], s["idx"])
    if kind == "step":
        n, call = len(s["keys"]), case["call"]
        new = np.array([min(call, n - b) for b in range(0, n, call)], dtype=np.int64)
        return [new, *_answer(s["vals"], s["idx"]), len(s["rem"])]
    if kind == "upsert":
        return 0, s["new"], torch.ones(case["n"], dtype=torch.uint8, device=DEV)
    ids, n, call, last = s["ids"], case["n"], case["call"], s["last"]
    new = np.array([len(torch.unique(ids[b:b + call])) for b in range(0, n, call)], dtype=np.int64)
    place = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    place.scatter_reduce_(0, ids, torch.arange(n, device=DEV), "amax")  # the later position of a key wins
    idx = torch.cat([place[ids[last:]], torch.full((n - last,), -1, device=DEV)])
    out = [new, *_answer(s["vals"], idx)]
    if case["removes"]:
        gone = torch.zeros(n, dtype=torch.bool, device=DEV)
        gone[ids[s["rem"]]] = True
        left = idx.clone()
        left[:n - last][gone[ids[last:]]] = -1
        out += [int(gone.sum()), *_answer(s["vals"], left)]
    return out


def work(case):
    """Bytes a pass cannot do without: inputs and outputs once, and per table record touched its key, its value and its
    metadata word (a miss: one metadata sector of 32 bytes).  No floating-point work."""
    kind = case["kind"]
    if kind == "batch":
        per = 0.5 * (16 + 160)
        mean = (case["max_n"] - 256) / math.log(case["max_n"] / 256)
        slots = case["tables"] * ((1 << (case["hi_bits"] + 1)) - (1 << case["lo_bits"])) / (
            case["hi_bits"] - case["lo_bits"] + 1)
        return {"bytes": case["ops"] * mean * 2 * per + 2 * slots * (per + 4), "flops": 0}
    k, v = case["k"], case["v"]
    ins = 2 * (k + v) + 4              # a pair read, a record and its word written

    def get(n, hit):                   # key in, value and found byte out; a hit reads the record
        return n * (k + v + 1 + 32 + hit * (k + v))

    def rem(n):                        # key in, the record's key and metadata read, its word written
        return n * (2 * k + 32 + 4)

    cap = 1 << case["bits"]
    if kind == "get":
        b = get(case["n"], case["hit"])
    elif kind == "load":
        q = 2 * min(case["call"], case["n"])
        b = 4 * cap + case["n"] * ins + get(q, 0.5) + (rem(case["removes"]) + get(q, 0.45) if case["removes"] else 0)
    elif kind == "step":
        n = int(cap * case["load"])
        b = 4 * cap + n * ins + get(case["gets"], 0.5) + rem(n // 10)
    elif kind == "upsert":
        b = case["n"] * ins + case["n"] * (k + 32) + get(case["n"], 1.0)
    elif kind == "churn":
        n = case["n"]
        b = 2 * cap * (k + v + 4) + rem(n) + n * ins + rem(n + n // 4) + get(2 * n, 0.8)
    else:
        b = 4 * cap + case["n"] * ins + get(case["n"], 1.0) + case["n"] * 2 * (k + v)
    return {"bytes": float(b), "flops": 0}
