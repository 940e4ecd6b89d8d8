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


def _two_fans(heads, every):
    """`heads` sources of 4,200 targets each, or 2,000 for one in `every`: past a CTA's search, and within it."""
    x, root, small = np.arange(heads), heads, heads + 1
    t = heads + 2 + np.arange(4200)
    return np.concatenate([np.stack([x, np.where(x % every, root, small)], 1), np.stack([np.full(4200, root), t], 1),
                           np.stack([np.full(2000, small), t[:2000]], 1)])


# sources left over by most CTA searches (the later ones are then not begun), by half of them, by few
@pytest.mark.parametrize("heads,every", [(3000, 3000), (3000, 3), (3000, 2), (511, 8), (2400, 1)])
def test_tc_sources_that_cta_searches_leave_over(engine, heads, every, monkeypatch):
    name = f"two_fans_{heads}_{every}"
    monkeypatch.setitem(CASES, name, (_two_fans(heads, every), 0))
    test_tc_searches_equal_sorted_runs(engine, name)


def _chain(n):
    """0 -> 1 -> n leaves."""
    return np.concatenate([[[0, 1]], np.stack([np.full(n, 1), 2 + np.arange(n)], 1)])


def _hubs(hubs, each):
    """A source above `hubs` nodes of `each` out-edges, all to their own leaves."""
    leaves = hubs + 1 + np.arange(hubs * each)
    return np.concatenate([np.stack([np.zeros(hubs, int), 1 + np.arange(hubs)], 1),
                           np.stack([np.repeat(1 + np.arange(hubs), each), leaves], 1)])


def _two_groups(hubs, each, small):
    """The same with `small` further nodes of one out-edge each, which another warp takes."""
    e = _hubs(hubs, each)
    top = int(e.max()) + 1
    mid = top + np.arange(small)
    return np.concatenate([e, np.stack([np.zeros(small, int), mid], 1), np.stack([mid, mid + small], 1)])


# join words of one warp's rows on both sides of a CTA's 2^18 and of a warp's 2^14
WIDE = {f"chain_{n}": _chain(n) for n in (16383, 16384, 16385, 262143, 262144, 262145, 300_000)}
WIDE |= {"hubs_8191": _hubs(32, 8191), "hubs_8192": _hubs(32, 8192), "hubs_9000": _hubs(32, 9000),
         "two_groups": _two_groups(32, 9000, 40), "fan_262145": _fan(262_145, 3)}


def _check_wide(got, want, name):
    assert got.deltas.tolist() == want.deltas.tolist(), name
    assert got.output_tuples == want.output_tuples and np.array_equal(got.rows, want.rows), name


@pytest.mark.parametrize("name", sorted(WIDE))
def test_tc_rows_past_a_searchs_join_words(engine, name):
    e = np.ascontiguousarray(WIDE[name]).astype(np.int32)
    want, got = engine.tc(e, dedup="sort"), engine.tc(e)
    _check_wide(got, want, name)
    assert got.join_rows.tolist() == want.join_rows.tolist() and got.full_rows.tolist() == want.full_rows.tolist()


def test_tc_wide_rows_in_a_batch_and_a_session(engine):
    """Wide nodes and heavy sources side by side with small instances."""
    sets = {k: np.ascontiguousarray(v).astype(np.int32) for k, v in WIDE.items()}
    sets["both"] = np.concatenate([_chain(300_000), 400_000 + _cycle(4200)]).astype(np.int32)
    sets["path"] = _path(30).astype(np.int32)
    want = {k: engine.tc(v, dedup="sort") for k, v in sets.items()}
    for k, got in zip(sets, engine.run_batch("tc", list(sets.values()))):
        _check_wide(got, want[k], k)
    with engine.session("tc") as s:
        ids = [(i, k) for k, i in zip(sets, s.admit_many(list(sets.values())))]
        s.step()
        ids += [(s.admit(sets[k]), k) for k in ("chain_262145", "two_groups", "path")]
        s.run()
        for i, k in ids:
            _check_wide(s.result(i), want[k], k)


@pytest.mark.parametrize("algorithm", [0, 1])
def test_tc_result_order_under_both_sorts(algorithm):
    """The searched words are lined up by source and sorted by target only; as a plain run and
    in a batch, whose ranks start above those of earlier instances."""
    from mnmgdatalog_b200 import Engine
    sets = [np.ascontiguousarray(CASES[k][0]).astype(np.int32) for k in ("dag", "random_sparse_ids", "chung_lu")]
    with Engine(0) as eng:
        eng.set_tuning(sort_algorithm=algorithm)
        want = [eng.tc(e, dedup="sort") for e in sets]
        res = eng.run_batch("tc", sets)
        for w, b, e in zip(want, res, sets):
            got = eng.tc(e)
            assert np.array_equal(got.rows, w.rows) and np.array_equal(b.rows, w.rows)
            assert got.deltas.tolist() == w.deltas.tolist() == b.deltas.tolist()


def _tiny(seed, count=12_000):
    """Components around what one lane searches alone (paths of up to three targets, rows of up to
    four sinks): paths, stars, paths into stars and cycles, self loops, in shuffled id order."""
    rng = np.random.default_rng(seed)
    kinds = [_path(k) for k in (1, 2, 3, 4, 5)] + [_cycle(k) for k in (1, 2, 3, 4)]
    kinds += [np.stack([np.zeros(k, int), 1 + np.arange(k)], 1) for k in (2, 3, 4, 5)]
    kinds += [np.concatenate([_path(p), [[p, p + 1 + j] for j in range(k)]]) for p in (1, 2) for k in (2, 4)]
    kinds += [np.array(x) for x in ([[0, 1], [1, 1]], [[0, 1], [1, 2], [2, 1]], [[0, 1], [1, 2], [2, 2]],
                                    [[0, 1], [0, 2], [1, 2]], [[0, 0], [0, 1]], [[0, 1], [1, 2], [2, 0], [2, 3]],
                                    [[0, 1], [0, 2], [2, 3]])]
    out, top = [], 0
    for k in rng.integers(0, len(kinds), count):
        out.append(kinds[k] + top)
        top += int(kinds[k].max()) + 1
    ids = rng.permutation(top) if seed % 2 else np.arange(top)
    return ids[np.concatenate(out)].astype(np.int32)


@pytest.mark.parametrize("stop", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("seed", [0, 1])
def test_tc_tiny_searches(engine, seed, stop):
    e = _tiny(seed)
    want, got = engine.tc(e, dedup="sort", max_iterations=stop), engine.tc(e, max_iterations=stop)
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    assert np.array_equal(got.rows, want.rows)


def test_tc_tiny_searches_in_a_batch(engine):
    """Instances that begin and end inside a warp's 32 sources."""
    sets = [_tiny(k, c) for k, c in enumerate((5, 9000, 1, 1, 3, 2, 400, 1, 2000))] + [_path(1).astype(np.int32)] * 40
    for e, got in zip(sets, engine.run_batch("tc", sets)):
        want = engine.tc(e, dedup="sort")
        assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows)


def test_tc_many_tiny_searches(engine):
    """Millions of them beside searches of 400 targets."""
    k = np.arange(1_500_000, dtype=np.int32)
    hub = np.stack([np.repeat(np.arange(3_000_000, 3_000_200, dtype=np.int32), 200), np.arange(40_000, dtype=np.int32)], 1)
    e = np.concatenate([np.stack([k, k // 3 + 1_500_000], 1), hub])
    want, got = engine.tc(e, dedup="sort"), engine.tc(e)
    assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows)


def _layers(width, layers, degree, seed=1):
    """Each node of a layer has `degree` edges into the next one on average."""
    rng = np.random.default_rng(seed)
    return np.concatenate([np.stack([i * width + rng.integers(0, width, degree * width),
                                     (i + 1) * width + rng.integers(0, width, degree * width)], 1)
                           for i in range(layers)])


def _light_and_heavy(light, heavy, seed):
    """`light` sources above a hub of 20 targets, and `heavy` ones above it and 5000 leaves of their
    own, with ids in any order: a target's row has all of them."""
    hub, out = light + heavy, []
    out.append(np.stack([np.arange(light + heavy), np.full(light + heavy, hub)], 1))
    out.append(np.stack([np.full(20, hub), hub + 1 + np.arange(20)], 1))
    leaf = hub + 21 + np.arange(heavy * 5000)
    out.append(np.stack([light + np.repeat(np.arange(heavy), 5000), leaf], 1))
    e = np.concatenate(out)
    return np.random.default_rng(seed).permutation(int(e.max()) + 1)[e]


MERGED = {"layers": _layers(1000, 20, 2), "layers_thin": _layers(3000, 10, 1), "layers_wide": _layers(6000, 5, 5),
          "one_window": _light_and_heavy(31, 3, 1), "window_edge": _light_and_heavy(33, 5, 2),
          "one_heavy": _light_and_heavy(3000, 1, 3), "chunks": _light_and_heavy(4000, 40, 4),
          "past_16_bits": _light_and_heavy(70_000, 6, 5), "at_16_bits": _light_and_heavy(65_535, 2, 6)}


@pytest.mark.parametrize("name", sorted(MERGED))
def test_tc_rows_of_many_light_sources(engine, name):
    e = np.ascontiguousarray(MERGED[name]).astype(np.int32)
    want, got = engine.tc(e, dedup="sort"), engine.tc(e)
    assert got.deltas.tolist() == want.deltas.tolist()
    assert np.array_equal(got.rows, want.rows)


def _kary(n, k):
    a = np.arange(1, n)
    return np.stack([(a - 1) // k, a], 1)


THIN = {f"heads_{h}": _fan(4200, h) for h in (1, 1022, 1023, 1024, 2046, 2047, 2048)}
THIN |= {"tree_3": _kary(120_000, 3), "tree_10": _kary(200_000, 10), "tree_2": _kary(60_000, 2),
         "tree_and_back": np.concatenate([_kary(40_000, 4), [[39_000, 20_000], [38_000, 1], [30_000, 30_000]]]),
         "in_degrees": np.concatenate([_fan(4200, 40)] + [np.stack([3 + np.arange(d) + 40 * k, np.full(d, 9000 + k)], 1)
                                                          for k, d in enumerate((1, 7, 8, 9, 31, 32, 33, 64))])}


@pytest.mark.parametrize("stop", [0, 4])
@pytest.mark.parametrize("name", sorted(THIN))
def test_tc_few_heavy_sources(engine, name, stop):
    """Rows of one and two chunks, by eight lanes, and of three, by a warp."""
    e = np.ascontiguousarray(THIN[name]).astype(np.int32)
    want, got = engine.tc(e, dedup="sort", max_iterations=stop), engine.tc(e, max_iterations=stop)
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    assert np.array_equal(got.rows, want.rows)


def test_tc_searches_go_on_with_more_room(engine):
    """More than 2^27 words of eight-lane searches, the most that is reserved at first: sources from where
    the room was full, and those under way then, as a run and in a batch."""
    import torch
    e = graphs.sized("tc", 3_200_000)
    sets = [e, _tiny(3, 30_000), graphs.sized("tc", 200_000, seed=1)]
    want = [engine.tc(x, dedup="sort", output="device") for x in sets]
    assert want[0].output_tuples > 2**27
    engine.release_memory()  # (a cached buffer may be larger than what is asked for)
    got = engine.tc(e, output="device")
    assert torch.equal(got.rows, want[0].rows)
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want[0], f).tolist(), f
    del got
    for w, b in zip(want, engine.run_batch("tc", sets, output="device")):
        assert b.deltas.tolist() == w.deltas.tolist() and torch.equal(b.rows, w.rows)
