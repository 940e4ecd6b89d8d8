"""WCC's iterations launched in batches (dl_wcc.cu) against the iteration written
out in numpy, exactly: labels, |delta| and joined rows per iteration, both stop
rules and early stops -- with lists on both sides of the 128 edges a warp takes
at once, more iterations than one batch, and instances that stop at different
iterations of a batch."""
import numpy as np
import pytest

from mnmgdatalog_b200 import graphs

pytestmark = pytest.mark.gpu


def _star(d, base=0):
    return [[base + 1 + i, base + d + 1] for i in range(d)]  # the hub has the largest id


CASES = {
    "one": [[1, 2]], "loop": [[5, 5]], "path8": [[i, i + 1] for i in range(8)], "path9": [[i, i + 1] for i in range(9)],
    "path40": [[i, i + 1] for i in range(40)], "back_path": [[40 - i, 39 - i] for i in range(40)],
    "star_128": _star(128), "star_129": _star(129), "star_1025": _star(1025),
    # hubs whose labels fall late: their long lists are walked in iterations above 1
    "late_hubs": [[0, 1], [1, 2], [2, 3], [3, 100_001]] + [[100_001, 9000 + i] for i in range(5000)]
    + [[14_000 - 1, 200_000]] + [[200_000, 20_000 + i] for i in range(2048)],
    "random": np.random.default_rng(0).integers(0, 3000, (2500, 2)), "dag": graphs.dag(n=1500, extra=500, seed=2),
    "mesh": graphs.lattice3d(side=14, p=0.3, seed=5), "wide_ids": graphs.lattice3d(side=10, seed=4) * 1_000_003 - 10**9,
}


def _rows(name):
    return np.ascontiguousarray(CASES[name]).astype(np.int32)


def _wcc(e, rule, cap):
    ids, r = np.unique(e, return_inverse=True)
    r = r.reshape(-1, 2)
    s = np.unique(np.concatenate([r, r[:, ::-1]]), axis=0)
    label = np.arange(len(ids))
    changed = np.ones(len(ids), bool)
    deltas, joins, prev = [], [], len(ids)
    while True:
        m = changed[s[:, 0]]
        joins.append(int(m.sum()))
        new = label.copy()
        np.minimum.at(new, s[m, 1], label[s[m, 0]])
        changed = new < label
        label = new
        d = int(changed.sum())
        deltas.append(d)
        if (d == 0 if rule == "fixpoint" else d == prev) or (cap and len(deltas) >= cap):
            return ids, ids[label], deltas, joins
        prev = d


@pytest.mark.parametrize("cap", [0, 1, 8, 9])
@pytest.mark.parametrize("rule", ["reference", "fixpoint"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_wcc_levels(engine, name, rule, cap):
    e = _rows(name)
    ids, label, deltas, joins = _wcc(e, rule, cap)
    got = engine.wcc(e, wcc_stop=rule, max_iterations=cap, labels=True)
    assert got.deltas.tolist() == deltas and got.join_rows.tolist() == joins
    assert np.array_equal(got.node_ids, ids) and np.array_equal(got.labels, label)
    comp, size = np.unique(label, return_counts=True)
    assert got.largest_component == size.max() and np.array_equal(got.rows[:, 0], comp)


@pytest.mark.parametrize("cap", [0, 9])
@pytest.mark.parametrize("rule", ["reference", "fixpoint"])
def test_wcc_levels_batch(engine, rule, cap):
    names = sorted(CASES)
    sets = [_rows(k) for k in names] + [np.zeros((0, 2), np.int32)]
    res = engine.run_batch("wcc", sets, wcc_stop=rule, max_iterations=cap, labels=True)
    for e, got in zip(sets[:-1], res):
        ids, label, deltas, _ = _wcc(e, rule, cap)
        assert got.deltas.tolist() == deltas
        assert np.array_equal(got.node_ids, ids) and np.array_equal(got.labels, label)
        comp, size = np.unique(label, return_counts=True)
        assert got.largest_component == size.max() and np.array_equal(got.rows[:, 0], comp)
