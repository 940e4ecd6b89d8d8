"""single_join through bit rows (dl_selfjoin.cu) against the sort of its join
output (bitmap_max_gib = 0), and the ranking of node ids (by offset, presence
bits or sort, by the span of the ids): the same graph under a map of its ids
that keeps their order gives the mapped rows."""
import numpy as np
import pytest

from mnmgdatalog_b200 import graphs

pytestmark = pytest.mark.gpu


def _uniform(n, m, seed=0):
    return np.random.default_rng(seed).integers(0, n, (m, 2))


def _star(n):
    a, c = np.arange(n), np.full(n, 7)
    return np.concatenate([np.stack([a, c], 1), np.stack([c, a], 1)])


CASES = {
    "one": [[1, 2]], "loop": [[3, 3]], "chain": [[1, 2], [2, 3]], "extreme_ids": [[-2**31, 2**31 - 1], [2**31 - 1, -2**31]],
    "short_lists": _uniform(31, 200), "row_1024": _uniform(1024, 9000), "row_1025": _uniform(1025, 9000),
    "full": _uniform(1000, 100_000), "long_lists": _uniform(3000, 60_000), "sparse": _uniform(20_000, 400_000),
    "very_sparse": _uniform(5000, 5000), "spread_ids": _uniform(2000, 30_000) * 7919 - 10**6,
    "wide_ids": _uniform(2000, 30_000) * 1_000_003 - 10**9, "star": _star(3000),
    "skewed": np.random.default_rng(1).zipf(1.3, (60_000, 2)) % 9000,
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_single_join_equals_sorted_join(engine, name):
    import torch
    e = np.ascontiguousarray(CASES[name]).astype(np.int32)
    before = engine.tuning()
    try:
        engine.set_tuning(bitmap_max_gib=0)
        want = engine.single_join(e)
    finally:
        engine.set_tuning(before)
    got = engine.single_join(torch.from_numpy(e).cuda(), output="device")
    host = engine.single_join(e)
    assert np.array_equal(got.rows.cpu().numpy(), want.rows) and np.array_equal(host.rows, want.rows)
    for f in ("output_tuples", "nodes", "iterations", "join_rows_total", "join_rows_max"):
        assert getattr(got, f) == getattr(want, f), f
    assert got.deltas.tolist() == want.deltas.tolist()


@pytest.mark.parametrize("prog", ["tc", "sg", "wcc", "single_join"])
@pytest.mark.parametrize("scale,shift", [(1, -70), (1, 2**31 - 3001), (5, -2**31), (4099, 11), (700_001, -2**31)])
def test_results_do_not_depend_on_the_span_of_the_ids(engine, prog, scale, shift):
    e = graphs.lattice3d(side=9, p=0.3, seed=3) if prog == "sg" else graphs.dag(n=3000, extra=900, seed=2)
    plain = engine.run(prog, e, labels=prog == "wcc")
    moved = (e.astype(np.int64) * scale + shift).astype(np.int32)
    got = engine.run(prog, moved, labels=prog == "wcc")
    rows = plain.rows.astype(np.int64) * scale + shift
    if prog == "wcc":  # rows are (component id, 0)
        rows[:, 1] = 0
        assert np.array_equal(got.labels, (plain.labels.astype(np.int64) * scale + shift).astype(np.int32))
    assert np.array_equal(got.rows, rows.astype(np.int32))
    assert got.deltas.tolist() == plain.deltas.tolist()
