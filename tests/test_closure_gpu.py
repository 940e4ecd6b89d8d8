"""TC by searches and heavy-source bit rows (dl_closure.cu, what AUTO runs)
against the sorted runs, exactly: rows to host and device memory, iterations,
per-iteration delta, join and full sizes -- at the limits of the forms: a
warp's 512 targets and 256 levels, a CTA's 4096 targets and 4096 levels, 32
in-edges of a target, 1024 heavy sources to a chunk, 32 chunks to an activity
word."""
import numpy as np
import pytest

from mnmgdatalog_b200 import graphs

pytestmark = pytest.mark.gpu


def _path(n):
    return np.stack([np.arange(n), np.arange(1, n + 1)], 1)


def _cycle(n):
    return np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)


def _fan(n, heads):
    """`heads` sources with an edge each into a root with n targets, which all
    point to one collector (n in-edges) that points on."""
    root, coll = heads, heads + 1
    t = np.arange(n) + heads + 2
    return np.concatenate([np.stack([np.arange(heads), np.full(heads, root)], 1), np.stack([np.full(n, root), t], 1),
                           np.stack([t, np.full(n, coll)], 1), [[coll, heads + 2 + n]]])


def _random(n, m, seed):
    return np.random.default_rng(seed).integers(0, n, (m, 2))


CASES = {
    "path_511": (_path(511), 0), "path_513": (_path(513), 0), "path_257_levels": (_path(257), 0),
    "path_max": (_path(5000), 40), "cycle_512": (_cycle(512), 0), "cycle_4097": (_cycle(4097), 0),
    "fan_31": (_fan(31, 3), 0), "fan_33": (_fan(33, 3), 0), "fan_510": (_fan(509, 5), 0),
    "fan_513": (_fan(513, 40), 0), "fan_4094": (_fan(4094, 3), 0), "fan_4200": (_fan(4200, 1100), 0),
    "random_1023": (_random(1023, 6000, 1), 0), "random_5000": (_random(5000, 15000, 2), 0),
    "random_5000_max3": (_random(5000, 15000, 2), 3), "random_sparse_ids": (_random(6000, 14000, 3) * 977 - 10**6, 0),
    "chung_lu": (graphs.chung_lu(n=30_000, m=100_000, seed=1), 0), "dag": (graphs.dag(n=9000, extra=5000, seed=2), 0),
    "wide_33_chunks": (_random(38_000, 110_000, 4), 5),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tc_searches_equal_sorted_runs(engine, name):
    import torch
    e, stop = CASES[name]
    e = np.ascontiguousarray(e).astype(np.int32)
    want = engine.tc(e, dedup="sort", output="device", max_iterations=stop)
    got = engine.tc(torch.from_numpy(e).cuda(), output="device", max_iterations=stop)
    assert got.iterations == want.iterations and got.nodes >= want.nodes
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    assert got.join_rows_total == want.join_rows_total and got.join_rows_max == want.join_rows_max
    assert torch.equal(got.rows, want.rows)
    if want.output_tuples < 5 * 10**7:
        host = engine.tc(e, max_iterations=stop)
        assert np.array_equal(host.rows, want.rows.cpu().numpy())
