"""SG on bit rows (dl_sgrows.cu, what AUTO runs on well-connected graphs) against
the stepped bit matrix, exactly: rows, iterations and per-iteration sizes -- with
a warp, four and eight warps to a row, more than 32 chunks to an activity word,
more than 32 in-neighbours and more than 8 children of a node, and runs that
stop inside and at the end of a batch of levels."""
import numpy as np
import pytest

from mnmgdatalog_b200 import graphs

pytestmark = pytest.mark.gpu


def _random(n, m, seed=0):
    return np.random.default_rng(seed).integers(0, n, (m, 2))


def _fan(n):
    a = np.arange(n)
    return np.concatenate([np.stack([np.zeros(n), a + 1], 1), np.stack([a + 1, np.full(n, 2 * n)], 1),
                           np.stack([np.full(n, 2 * n), a + 3 * n], 1)])


CASES = [("mesh", graphs.lattice3d(side=14, p=0.3, seed=5), 0), ("mesh_stops", graphs.lattice3d(side=14, p=0.3, seed=5), 7),
         ("mesh_stops_8", graphs.lattice3d(side=20, p=0.3, seed=1), 8), ("one_chunk", _random(1000, 3000), 0),
         ("degrees", graphs.chung_lu(n=4000, m=12_000, seed=3), 0), ("fan", _fan(1500), 0),
         ("children_9", np.stack([np.repeat(np.arange(900), 9), (np.arange(8100) * 7) % 1000], 1), 0),
         ("chunks_33", _random(34_000, 76_000, 1), 3), ("four_warps", _random(60_000, 130_000, 2), 3),
         ("eight_warps", _random(135_000, 290_000, 3), 2), ("spread_ids", _random(3000, 9000, 4) * 700_001 - 2**31, 0)]


@pytest.mark.parametrize("name,edges,stop", CASES, ids=[c[0] for c in CASES])
def test_sg_rows_equal_matrix(engine, name, edges, stop):
    import torch
    e = np.ascontiguousarray(edges).astype(np.int32)
    want = engine.sg(e, dedup="bitmap", output="device", max_iterations=stop)
    got = engine.sg(torch.from_numpy(e).cuda(), output="device", max_iterations=stop)
    assert got.iterations == want.iterations and got.nodes == want.nodes
    for f in ("deltas", "join_rows", "full_rows"):
        assert getattr(got, f).tolist() == getattr(want, f).tolist(), f
    assert torch.equal(got.rows, want.rows)
    if want.output_tuples < 10**7:
        assert np.array_equal(engine.sg(e, max_iterations=stop).rows, want.rows.cpu().numpy())


@pytest.mark.parametrize("name,edges,stop", [
    ("one_in_60", graphs.lattice3d(side=14, p=0.3, seed=5), 5), ("one_in_19", graphs.lattice3d(side=14, p=0.3, seed=5), 10),
    ("one_in_119", _random(40_000, 80_000, 5), 3), ("one_in_31", _random(40_000, 80_000, 5), 4),
    ("ids_of_a_sort", _random(3000, 4500, 4) * 700_001 - 2**31, 3), ("eight_warps_sparse", _random(135_000, 290_000, 3), 3)])
def test_sg_rows_sparse_and_dense_results(engine, name, edges, stop):
    """Results on both sides of the density (a bit in 32) at which their writer changes."""
    test_sg_rows_equal_matrix(engine, name, edges, stop)


def _into_hubs(n, m, hubs, seed):
    """A random graph, a third of whose edges go into `hubs` nodes."""
    rng = np.random.default_rng(seed)
    b = rng.integers(0, n, m)
    b[: m // 3] = rng.integers(0, hubs, m // 3)
    return np.stack([rng.integers(0, n, m), b], 1)


def _in_degrees(*ds):
    """Nodes of d in-neighbours each, below a root and a second generation that mixes them."""
    out, o = [], 1
    for d in ds:
        hub = o + d
        out += [np.stack([np.zeros(d, int), o + np.arange(d)], 1), np.stack([o + np.arange(d), np.full(d, hub)], 1),
                [[hub, hub + 1], [hub, hub + 2], [hub + 1, 1], [hub + 2, 2]]]
        o = hub + 3
    return np.concatenate(out)


HUBS = [("edges_of_segments", _in_degrees(31, 32, 33, 63, 64, 65, 96, 97, 1000), 0),
        ("small", _into_hubs(900, 2500, 3, 1), 0), ("deep", _into_hubs(9000, 18_000, 4, 2), 0),
        ("deep_stops", _into_hubs(9000, 18_000, 4, 2), 8), ("three_pieces", _into_hubs(20_000, 40_000, 4, 3), 0),
        ("four_warps", _into_hubs(60_000, 130_000, 5, 4), 3), ("granules", _into_hubs(36_000, 80_000, 40, 5), 5)]


@pytest.mark.parametrize("name,edges,stop", HUBS, ids=[c[0] for c in HUBS])
def test_sg_rows_of_many_in_neighbours(engine, name, edges, stop):
    """Accumulated rows of nodes past 32 in-neighbours."""
    test_sg_rows_equal_matrix(engine, name, edges, stop)
