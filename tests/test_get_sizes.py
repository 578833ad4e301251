"""Lookups of run-time record sizes on both sides of the count from which they
run on a thread per query, against the oracle: pieces of 16, 4 and 1 bytes, no
values, buffers off the 16-byte grid, nothing written beside the outputs."""
import numpy as np
import pytest

import oracle as O
from fm_testutil import gpu_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16), (12, 20), (5, 3), (3, 32), (4, 0), (256, 256), (64, 1), (1, 7)])
@pytest.mark.parametrize("mode", [0, 1])
def test_counts(shape, mode):
    import torch

    ks, vs = shape
    cap = 1 << 12
    rng = np.random.default_rng(ks + vs)
    g, o = gpu_map(cap, ks, vs, mode), O.OracleMap(cap, ks, vs, mode)
    k = rng.integers(0, 256, (int(cap * 0.7) if ks > 1 else 100, ks), dtype=np.uint8)
    v = rng.integers(0, 256, (len(k), vs), dtype=np.uint8)
    assert g.bulk_insert(k, v) == o.bulk_insert(k, v)
    assert g.bulk_remove(k[::9]) == o.bulk_remove(k[::9])
    line = torch.cuda.get_device_properties(0).multi_processor_count * 128
    for n in (1, 33, line - 1, line, line + 1, line + 4099):
        q = rng.integers(0, 256, (n, ks), dtype=np.uint8)
        q[::2] = k[rng.integers(0, len(k), (n + 1) // 2)]
        ov, of = o.bulk_get(q)
        for shift in (0, 4, 1):
            dk = torch.zeros(n * ks + 16, dtype=torch.uint8, device="cuda")
            dv = torch.full((n * vs + 32,), 7, dtype=torch.uint8, device="cuda")
            df = torch.full((n + 8,), 9, dtype=torch.uint8, device="cuda")
            dk[shift:shift + n * ks] = torch.from_numpy(q.reshape(-1)).cuda()
            g.bulk_get_device(dk[shift:], n, dv[shift:], df)
            torch.cuda.synchronize()
            assert np.array_equal(dv[shift:shift + n * vs].cpu().numpy().reshape(n, vs), ov)
            assert np.array_equal(df[:n].cpu().numpy().astype(bool), of.astype(bool))
            assert (dv[:shift] == 7).all() and (dv[shift + n * vs:] == 7).all() and (df[n:] == 9).all()


def test_small_calls_run_on_tiles():
    """The kernels' names by the profiler: a thread per query only for many queries."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    g = gpu_map(1 << 12, 5, 3)
    rng = np.random.default_rng(1)
    k = rng.integers(0, 256, (2000, 5), dtype=np.uint8)
    g.bulk_insert(k, k[:, :3])
    line = torch.cuda.get_device_properties(0).multi_processor_count * 128
    for n, want in ((1000, "k_get<"), (line + 1, "k_get_any")):
        q = torch.from_numpy(rng.integers(0, 256, (n, 5), dtype=np.uint8)).cuda()
        ov, of = torch.zeros((n, 3), dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            g.bulk_get_device(q, n, ov, of)
            torch.cuda.synchronize()
        names = [e.key for e in p.key_averages()]
        if not any("k_" in x for x in names):
            pytest.skip("no kernel records from the profiler")
        assert any(want in x for x in names), names
