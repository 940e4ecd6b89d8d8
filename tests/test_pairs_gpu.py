"""SG as a search over pairs (dl_pairs.cu, what AUTO runs on sparse graphs and
sessions run) against the sorted runs, exactly: rows, iterations and
per-iteration sizes -- with degrees on both sides of the 64 a pair may have,
bases that are empty, runs that stop early, results past the first set's size
(a level repeated on a larger set), and instances of both kinds in a session."""
import numpy as np
import pytest

from mnmgdatalog_b200 import graphs

pytestmark = pytest.mark.gpu


def _tree(n, k):
    return [[i, k * i + 1 + j] for i in range(n) for j in range(k)]


def _hubs(d):
    return [[0, i + 1] for i in range(d)] + [[i + 1, 1000 + i] for i in range(d)]


CASES = {
    "one": [[1, 2]], "loop": [[1, 1], [1, 2]], "siblings": [[1, 2], [1, 3]], "cycle": [[i, (i + 1) % 7] for i in range(7)],
    "tree2": _tree(500, 2), "tree5": _tree(900, 5), "hub_64": _hubs(64), "hub_65": _hubs(65),
    "lattice": graphs.lattice3d(side=12, seed=1), "dense_lattice": graphs.lattice3d(side=14, p=0.3, seed=5),
    "random": np.random.default_rng(0).integers(0, 3000, (5000, 2)), "dag": graphs.dag(n=1500, extra=500, seed=2),
    "wide_ids": graphs.lattice3d(side=10, seed=4) * 1_000_003 - 10**9,
}
STOPS = [0, 1, 4]


def _rows(name):
    return np.ascontiguousarray(CASES[name]).astype(np.int32)


@pytest.mark.parametrize("stop", STOPS)
@pytest.mark.parametrize("name", sorted(CASES))
def test_sg_pairs_equal_sorted_runs(engine, name, stop):
    e = _rows(name)
    want = engine.sg(e, dedup="sort", max_iterations=stop)
    got = engine.sg(e, max_iterations=stop)
    assert got.iterations == want.iterations
    assert got.deltas.tolist() == want.deltas.tolist() and got.full_rows.tolist() == want.full_rows.tolist()
    assert np.array_equal(got.rows, want.rows)
    # the delta rows joined per iteration are counted as on the bit matrix
    assert got.join_rows.tolist() == engine.sg(e, dedup="bitmap", max_iterations=stop).join_rows.tolist()


@pytest.mark.parametrize("stop", STOPS)
@pytest.mark.parametrize("names", [["lattice", "cycle", "tree2", "one"], ["hub_64", "hub_65", "loop", "dense_lattice"]])
def test_sg_batch_equals_sorted_runs(engine, names, stop):
    sets = [_rows(k) for k in names] + [np.zeros((0, 2), np.int32)]
    for e, got in zip(sets, engine.run_batch("sg", sets, max_iterations=stop)):
        want = engine.sg(e, dedup="sort", max_iterations=stop)
        assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows)


def test_sg_session_of_both_kinds(engine):
    """Searched instances and instances on the sorted runs advance side by side."""
    order = [["lattice", "hub_65"], ["dag", "tree5"], ["hub_65", "lattice"], ["dense_lattice"]]
    with engine.session("sg") as s:
        ids = []
        for names in order:
            ids += list(zip(s.admit_many([_rows(k) for k in names]), names))
            s.step()
        s.run()
        for i, k in ids:
            want = engine.sg(_rows(k), dedup="sort")
            got = s.result(i)
            assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows), k


def test_sg_set_outgrown(engine):
    """More pairs than the first set holds (512K), in one instance of a batch."""
    sets = [graphs.lattice3d(side=14, p=0.3, seed=5), graphs.lattice3d(side=9, p=0.3, seed=1)]
    for e, got in zip(sets, engine.run_batch("sg", sets)):
        want = engine.sg(e, dedup="bitmap")
        assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows)
    assert len(got.rows) < 2**19 < len(engine.sg(sets[0]).rows)


def _chains(count, length, leaves, first):
    """A root above `count` chains of `length` nodes, each with `leaves` leaves at its
    end: count * (count - 1) * leaves^2 pairs of leaves, all found in level `length`."""
    head = first + 1 + np.arange(count) * length
    node = (head[:, None] + np.arange(length)).ravel()
    out = [np.stack([np.full(count, first), head], 1),
           np.stack([node, node + 1], 1).reshape(count, length, 2)[:, :-1].reshape(-1, 2)]
    last, leaf = head + length - 1, first + 1 + count * length + np.arange(count * leaves)
    out.append(np.stack([np.repeat(last, leaves), leaf], 1))
    return np.concatenate(out), int(leaf[-1]) + 1


@pytest.mark.parametrize("first,second", [(0, 9), (6, 61), (6, 60), (7, 62), (14, 61)])
def test_sg_levels_repeated_near_the_counters_end(engine, first, second):
    """The set is outgrown in level `first` (past 512K pairs) and again in level
    `second` (past 2M): the levels after it are repeated, at (6, 61) with the last of
    the 64 levels' counters."""
    a, top = _chains(12, first, 64, 0) if first else _chains(1, 1, 1, 0)
    if not first:  # one node above 64 nodes of 64 leaves would come later: siblings past 512K in the base
        a = np.stack([np.repeat(np.arange(200), 60), 1000 + np.arange(12_000)], 1)
        top = 13_000
    b, _ = _chains(24, second, 64, top)
    e = np.concatenate([a, b]).astype(np.int32)
    want, got = engine.sg(e, dedup="bitmap"), engine.sg(e)
    assert got.deltas.tolist() == want.deltas.tolist() and got.join_rows.tolist() == want.join_rows.tolist()
    assert np.array_equal(got.rows, want.rows)
    res = engine.run_batch("sg", [e])[0]
    assert res.deltas.tolist() == want.deltas.tolist() and np.array_equal(res.rows, want.rows)


def _batch_against_sorted(eng, sets, on_runs):
    """The batch's results, and whether it ran on the sorted runs."""
    sets = [np.ascontiguousarray(e).astype(np.int32) for e in sets]
    want = [eng.sg(e, dedup="sort") for e in sets]
    eng.profile(False)
    res = eng.run_batch("sg", sets)
    assert (eng.profile_read()["join_emit"]["launches"] > 0) == on_runs
    for w, got in zip(want, res):
        assert got.deltas.tolist() == w.deltas.tolist() and np.array_equal(got.rows, w.rows)


def test_sg_session_search_is_bounded():
    """A search that would pass bitmap_max_gib hands its instances to the sorted runs, before it
    starts (0) or when its set is outgrown (33M pairs in 0.8 GB, the next size takes 3)."""
    from mnmgdatalog_b200 import Engine
    small, mesh = graphs.lattice3d(side=8, seed=1), graphs.lattice3d(side=22, p=0.29, seed=0)
    with Engine(0) as eng:
        _batch_against_sorted(eng, [small, mesh], False)
        assert len(eng.sg(mesh).rows) > 2**25
        eng.set_tuning(bitmap_max_gib=1)
        _batch_against_sorted(eng, [small, mesh], True)
        _batch_against_sorted(eng, [small], False)
        eng.set_tuning(bitmap_max_gib=0)
        _batch_against_sorted(eng, [small], True)


def test_sg_session_many_pairs_of_wide_sources(engine):
    """Both sides of the rule by sources' out-edges and pairs (pair_search_outrun)."""
    def rnd(n, d, seed):
        return np.random.default_rng(seed).integers(0, n, (int(n * d), 2))
    _batch_against_sorted(engine, [rnd(3000, 3, 1), rnd(3000, 3, 2)], True)
    _batch_against_sorted(engine, [rnd(3000, 1.8, 1), rnd(3000, 1.8, 2)], False)
    _batch_against_sorted(engine, [rnd(300, 3, k) for k in range(6)], False)
    _batch_against_sorted(engine, [_tree(1000, 3), _tree(1800, 3)], True)
    _batch_against_sorted(engine, [[[0, i + 1] for i in range(60)]] * 20, False)
    with engine.session("sg") as s:  # a session with both kinds
        e = [np.asarray(x, np.int32) for x in (rnd(5000, 3, 3), _tree(40, 3))]
        ids = s.admit_many(e[:1])
        s.step()
        ids += s.admit_many(e[1:])
        s.run()
        for i, x in zip(ids, e):
            want, got = engine.sg(x, dedup="sort"), s.result(i)
            assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows)


def _full_stats(got, want):
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    for f in ("join_rows_total", "join_rows_max", "iterations", "nodes", "output_tuples"):
        assert getattr(got, f) == getattr(want, f), f
    assert np.array_equal(got.rows, want.rows)


@pytest.mark.parametrize("stop", [0, 1, 3])
@pytest.mark.parametrize("name", ["lattice", "wide_ids", "random", "forest", "wide_tree", "loops", "most_64"])
def test_sg_past_the_matrix_reports_the_sorted_runs_joins(name, stop):
    """Graphs whose bit matrix passes bitmap_max_gib: rows and join sizes are those of the sorted
    runs, by the search (which counts them) or by the runs."""
    from mnmgdatalog_b200 import Engine
    n = 130_000
    rng = np.random.default_rng(1)
    e = {"lattice": lambda: graphs.lattice3d(side=52, p=0.16, seed=3),
         "wide_ids": lambda: graphs.lattice3d(side=50, p=0.15, seed=4) * 17_001 - 2 * 10**9,
         "random": lambda: rng.integers(0, n, (100_000, 2)),
         "forest": lambda: np.concatenate([np.asarray(_tree(13, 3)) + 40 * k for k in range(3300)]),
         # (twice 64 words a pair: more than the set has slots for the large levels, not for the last ones)
         "most_64": lambda: np.concatenate([graphs.lattice3d(side=50, p=0.17, seed=6), np.asarray(_hubs(64)) + n]),
         "wide_tree": lambda: np.stack([np.arange(n) // 10, np.arange(n) + 1], 1),
         "loops": lambda: np.concatenate([np.stack([np.arange(n), np.arange(n)], 1),
                                          np.stack([np.arange(n - 1), np.arange(1, n)], 1)])}[name]()
    e = np.ascontiguousarray(e).astype(np.int32)
    if name == "wide_tree" and stop != 1:
        pytest.skip("10^9 pairs")
    if name == "loops" and not stop:
        stop = 5
    with Engine(0) as eng:
        eng.set_tuning(bitmap_max_gib=1)
        assert len(np.unique(e)) > 93_000
        _full_stats(eng.sg(e, max_iterations=stop), eng.sg(e, dedup="sort", max_iterations=stop))


@pytest.mark.parametrize("children,nodes,stop,listed", [(3, 60_000, 3, True), (3, 60_000, 4, False), (2, 90_000, 5, True),
                                                        (2, 90_000, 6, True), (2, 90_000, 7, False), (6, 50_000, 1, True),
                                                        (11, 50_000, 1, True), (13, 50_000, 1, False)])
def test_sg_with_few_iterations_left(children, nodes, stop, listed):
    """Levels of more than a pair a node: the list goes on to the last iteration when that ends with
    128 pairs a node at most, and is handed over when not; rows and sizes are the matrix's."""
    from mnmgdatalog_b200 import Engine
    c = np.arange(1, nodes)
    e = np.stack([(c - 1) // children, c], 1).astype(np.int32)
    with Engine(0) as eng:
        want = eng.sg(e, dedup="bitmap", max_iterations=stop)
        eng.profile(False)
        got = eng.sg(e, max_iterations=stop)
        by_rows = eng.profile_read()["bitmap_extract"]["launches"]
    assert (by_rows == 0) == listed
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    assert np.array_equal(got.rows, want.rows)


def _random_above(n, m, seed):
    return np.concatenate([np.random.default_rng(seed).integers(0, n, (m, 2)), [[0, n - 1]]]).astype(np.int32)


@pytest.mark.parametrize("n,m,stop", [(60_000, 60_000, 0), (140_000, 140_000, 0), (140_000, 152_000, 30),
                                      (140_000, 175_000, 12), (100_000, 106_000, 25), (125_000, 119_000, 0)])
def test_sg_handed_over_to_other_forms(engine, n, m, stop):
    """Lists past 16 pairs a node with small levels, and large ones that go to the matrix or to bit rows."""
    import torch
    e = _random_above(n, m, 7)
    want = engine.sg(e, dedup="bitmap", output="device", max_iterations=stop)
    got = engine.sg(e, output="device", max_iterations=stop)
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    assert torch.equal(got.rows, want.rows)
