"""TC by searches and heavy-source bit rows (dl_closure.cu, what AUTO runs)
against the sorted runs, exactly: rows to host and device memory, iterations,
per-iteration delta, join and full sizes -- at the limits of the forms: eight
lanes' 255 targets, 96 levels and 48 edges of a row, a warp's 1024 targets and
512 levels, a CTA's 4096 targets and 4096 levels, 32 in-edges of a target, 1024
heavy sources to a chunk, 32 chunks to an activity word."""
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


def _paths(lengths):
    """Disjoint paths; together enough sources for the eight-lane searches."""
    off = np.cumsum([0] + [n + 2 for n in lengths])
    return np.concatenate([_path(n) + o for n, o in zip(lengths, off)])


def _combs(degrees):
    """head -> root -> `d` leaves -> a leaf's own sink or the comb's common one."""
    out, o = [], 0
    for d in degrees:
        t = o + 2 + np.arange(d)
        sink = np.where(np.arange(d) % 2 == 0, o + 2 + d, o + 3 + d + np.arange(d))
        out += [[[o, o + 1]], np.stack([np.full(d, o + 1), t], 1), np.stack([t, sink], 1)]
        o += 3 + 2 * d
    return np.concatenate(out)


def _random(n, m, seed):
    return np.random.default_rng(seed).integers(0, n, (m, 2))


CASES = {
    "path_511": (_path(511), 0), "path_513": (_path(513), 0), "path_1025": (_path(1025), 0),
    "path_max": (_path(5000), 40), "cycle_512": (_cycle(512), 0), "cycle_4097": (_cycle(4097), 0),
    "fan_31": (_fan(31, 3), 0), "fan_33": (_fan(33, 3), 0), "fan_510": (_fan(509, 5), 0),
    "fan_513": (_fan(513, 40), 0), "fan_4094": (_fan(4094, 3), 0), "fan_4200": (_fan(4200, 1100), 0),
    "random_1023": (_random(1023, 6000, 1), 0), "random_5000": (_random(5000, 15000, 2), 0),
    "random_5000_max3": (_random(5000, 15000, 2), 3), "random_sparse_ids": (_random(6000, 14000, 3) * 977 - 10**6, 0),
    "chung_lu": (graphs.chung_lu(n=30_000, m=100_000, seed=1), 0), "dag": (graphs.dag(n=9000, extra=5000, seed=2), 0),
    "paths_reach_255": (_paths([253 + i % 6 for i in range(40)]), 0),
    "paths_levels_96": (_paths([94 + i % 5 for i in range(100)]), 0),
    "paths_max_2": (_paths([60] * 160), 2), "cycles_3": (_cycle(3)[None] + 3 * np.arange(3000)[:, None, None], 0),
    "combs_48": (_combs([45 + i % 6 for i in range(200)]), 0), "combs_63": (_combs([60 + i % 6 for i in range(150)]), 0),
    "wide_33_chunks": (_random(38_000, 110_000, 4), 5),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tc_searches_equal_sorted_runs(engine, name):
    import torch
    e, stop = CASES[name]
    e = np.ascontiguousarray(e).astype(np.int32).reshape(-1, 2)
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
