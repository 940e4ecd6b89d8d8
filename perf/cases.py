"""The work that users of the engine have it do, as timed cases.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges,
`prepare(case, seed)` makes what a program holds before the call, and
`run(state)` is one pass through the public entry points. Every output is a
whole number (node ids, counts), so there is no 64-bit value to compare with:
`exact` is `None` throughout.

Sizes come from the repository's own workloads (mnmgdatalog_b200/graphs.py,
bench.py): the 5K-edge DAG, the 317K-node Chung-Lu graph, lattice meshes, the
1K-500K-edge requests of the served mix, the 1K-200K-edge instances of the
batched mix and the 10M-row self-join.
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from mnmgdatalog_b200 import Engine, graphs, serve

# A program keeps one engine; the states that are alive share it, and it goes
# with the last of them.
_engines = weakref.WeakValueDictionary()


def _engine() -> Engine:
    eng = _engines.get(0)
    if eng is None:
        eng = _engines[0] = Engine(0)
    return eng


def listed() -> list[dict]:
    return [
        # one small query, host rows in and out: some 80 iterations over a few
        # hundred tuples each, so launches and host waits count
        {"name": "tc_small", "kind": "program", "program": "tc", "graph": "dag", "edges": 5500, "on_device": False},
        # a large sparse closure (the served mix's largest TC request): many
        # iterations, 55 tuples a node
        {"name": "tc_dag", "kind": "program", "program": "tc", "graph": "dag", "edges": 500_000, "on_device": True},
        # TC at scale: 1.9e9 tuples of a power-law graph, rows left on the device
        {"name": "tc_chung_lu", "kind": "program", "program": "tc", "graph": "chung_lu", "edges": 1_050_000,
         "on_device": True},
        # one small SG query, host rows in and out
        {"name": "sg_small", "kind": "program", "program": "sg", "graph": "lattice", "edges": 5000,
         "on_device": False},
        # SG over a well-connected mesh: 10^8 tuples and more
        {"name": "sg_mesh", "kind": "program", "program": "sg", "graph": "mesh", "side": 28, "percent": 30,
         "on_device": True},
        # one small WCC query, host rows in, components and labels out
        {"name": "wcc_small", "kind": "program", "program": "wcc", "graph": "chung_lu", "edges": 20_000,
         "on_device": False, "wcc_stop": "reference"},
        # WCC of a graph of a million edges to its fixpoint
        {"name": "wcc_large", "kind": "program", "program": "wcc", "graph": "chung_lu", "edges": 1_050_000,
         "on_device": True, "wcc_stop": "fixpoint"},
        # the self-join of the strong-scaling input: 10M rows, 1.04e9 output rows
        {"name": "single_join", "kind": "program", "program": "single_join", "graph": "uniform",
         "edges": 10_000_000, "range": 90_000, "on_device": True},
        # batched form: many independent queries of uneven sizes in one call
        {"name": "batch_tc", "kind": "batch", "program": "tc", "count": 48, "low": 1000, "high": 200_000},
        {"name": "batch_wcc", "kind": "batch", "program": "wcc", "count": 48, "low": 1000, "high": 200_000},
        # served form: requests from host memory join a running session, and
        # each result leaves to host memory as it finishes
        {"name": "session_sg", "kind": "session", "program": "sg", "count": 32, "low": 1000, "high": 100_000},
        # one iteration of a caller's own loop over the relational operators
        {"name": "operators", "kind": "operators", "edges": 1_000_000, "range": 100_000, "full": 8_000_000},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["tc_dag", "tc_chung_lu", "sg", "mesh", "wcc", "single_join", "batch", "session", "operators"])
    if kind == "tc_dag":
        m = _log(rng, 1000, 500_000)
        return {"kind": "program", "program": "tc", "graph": "dag", "edges": m, "on_device": m > 20_000}
    if kind == "tc_chung_lu":
        return {"kind": "program", "program": "tc", "graph": "chung_lu", "edges": _log(rng, 5000, 1_050_000),
                "on_device": True}
    if kind == "sg":
        m = _log(rng, 1000, 500_000)
        return {"kind": "program", "program": "sg", "graph": "lattice", "edges": m, "on_device": m > 20_000}
    if kind == "mesh":
        return {"kind": "program", "program": "sg", "graph": "mesh", "side": rng.randint(10, 28),
                "percent": rng.randint(28, 30), "on_device": True}
    if kind == "wcc":
        m = _log(rng, 1000, 1_050_000)
        return {"kind": "program", "program": "wcc", "graph": "chung_lu", "edges": m, "on_device": m > 50_000,
                "wcc_stop": rng.choice(["reference", "fixpoint"])}
    if kind == "single_join":
        m = _log(rng, 10_000, 10_000_000)
        return {"kind": "program", "program": "single_join", "graph": "uniform", "edges": m,
                "range": max(64, int(m / rng.uniform(10, 111))), "on_device": True}
    if kind == "batch":
        return {"kind": "batch", "program": rng.choice(["tc", "sg", "wcc"]), "count": rng.randint(8, 48),
                "low": 1000, "high": _log(rng, 5000, 200_000)}
    if kind == "session":
        return {"kind": "session", "program": rng.choice(["tc", "sg", "wcc"]), "count": rng.randint(8, 32),
                "low": 1000, "high": _log(rng, 5000, 100_000)}
    m = _log(rng, 10_000, 1_000_000)
    return {"kind": "operators", "edges": m, "range": max(64, int(m / rng.uniform(4, 20))),
            "full": int(m * rng.uniform(1, 8))}


# The graph of a case is fixed by its sizes; the seed renames its nodes and
# shuffles its rows, so every seed is another input with another result of the
# same number of rows.
def _shifted(a: np.ndarray, rng) -> np.ndarray:
    """Node ids keep their order and their dense range."""
    return rng.permutation(a + np.int32(rng.integers(0, 1 << 20)))


def _spread(a: np.ndarray, rng) -> np.ndarray:
    """Node ids keep their order, with gaps between them."""
    ids = np.cumsum(rng.integers(1, 9, int(a.max()) + 1)).astype(np.int32)
    return rng.permutation(ids[a])


def _permuted(a: np.ndarray, rng) -> np.ndarray:
    """Node ids change places within their range."""
    ids = rng.permutation(int(a.max()) + 1).astype(np.int32)
    return rng.permutation(ids[a])


def _pairs(rows: int, top: int, which: int, seed: int):
    """Uniform pairs over 1..top, relation number `which`; the seed permutes the
    ids (alike in every relation) and the rows."""
    g = torch.Generator(device="cuda").manual_seed(which)
    a = torch.randint(0, top, (rows, 2), generator=g, device="cuda")
    g.manual_seed(1000 + seed)
    ids = (1 + torch.randperm(top, generator=g, device="cuda")).int()
    return ids[a[torch.randperm(rows, generator=g, device="cuda")]].contiguous()


def _edges(case: dict, seed: int):
    g, rng = case["graph"], np.random.default_rng(seed)
    if g == "uniform":
        return _pairs(case["edges"], case["range"], 0, seed)
    if g == "dag":
        a = _shifted(graphs.sized("tc", case["edges"]), rng)
    elif g == "lattice":
        a = _shifted(graphs.sized("sg", case["edges"]), rng)
    elif g == "mesh":
        a = _shifted(graphs.lattice3d(side=case["side"], p=case["percent"] / 100), rng)
    else:  # the node/edge ratio of the 317K-node graph; WCC's iterations depend on the order of the ids
        a = graphs.chung_lu(n=_chung_lu_nodes(case["edges"]), m=case["edges"])
        a = (_shifted if case["program"] == "wcc" else _permuted)(a, rng)
    return torch.from_numpy(a).cuda() if case["on_device"] else a


def _chung_lu_nodes(edges: int) -> int:
    return max(16, int(edges * 317 / 1050))


def _sizes(case: dict) -> list[int]:
    """Instance sizes spread evenly over their logarithm."""
    n, lo, hi = case["count"], case["low"], case["high"]
    return [int(lo * (hi / lo) ** ((i + 0.5) / n)) for i in range(n)]


def prepare(case: dict, seed: int) -> dict:
    st = {"case": case, "engine": _engine()}
    if case["kind"] == "program":
        st["edges"] = _edges(case, seed)
    elif case["kind"] in ("batch", "session"):
        rng = np.random.default_rng(seed)
        sets = [graphs.sized(case["program"], m, seed=i) for i, m in enumerate(_sizes(case))]
        if case["kind"] == "batch":
            st["sets"] = [torch.from_numpy(_shifted(a, rng)).cuda() for a in sets]
        else:  # requests arrive in no order of size, with ids of any kind
            order = np.random.default_rng(len(sets)).permutation(len(sets))
            if case["program"] == "wcc":
                st["sets"] = [_spread(sets[k], rng) for k in order]
            else:
                st["sets"] = [serve.relabel(sets[k], seed * 1009 + int(k)) for k in order]
    else:
        m, top = case["edges"], case["range"]
        st["edges"], st["delta"] = _pairs(m, top, 0, seed), _pairs(m, top, 1, seed)
        st["full"] = st["engine"].sort_unique(_pairs(case["full"], top, 2, seed)).clone()
    return st


def _result(r) -> list:
    out = [r.rows, r.deltas]
    if r.program == "wcc":
        out.append(r.largest_component)
    if r.labels is not None:
        out += [r.node_ids, r.labels]
    return out


def run(st: dict):
    case, eng = st["case"], st["engine"]
    if case["kind"] == "program":
        return _result(eng.run(case["program"], st["edges"], wcc_stop=case.get("wcc_stop", "reference"),
                               output="device" if case["on_device"] else "host", labels=case["program"] == "wcc"))
    if case["kind"] == "batch":
        wcc = case["program"] == "wcc"
        res = eng.run_batch(case["program"], st["sets"], output="device", labels=wcc)
        out = [[r.rows for r in res], np.concatenate([r.deltas for r in res])]
        if wcc:
            out += [np.array([r.largest_component for r in res]), np.concatenate([r.labels for r in res])]
        return out
    if case["kind"] == "session":
        res = {}

        def collect(s):
            for i in s.poll():
                res[i] = s.result(i)
                s.release(i)

        sets = st["sets"]
        half = len(sets) // 2
        with eng.session(case["program"]) as s:
            s.admit_many(sets[:half])
            for _ in range(3):
                s.step()
                collect(s)
            s.admit_many(sets[half:])
            while s.step():
                collect(s)
            collect(s)
        return [[res[i].rows for i in range(len(sets))], np.concatenate([res[i].deltas for i in range(len(sets))])]
    table = eng.get_hash_table(st["edges"])
    joined = eng.get_join(table, st["delta"])
    fresh = eng.sort_unique(joined)
    delta = eng.set_difference(fresh, st["full"])
    return [fresh, delta, eng.merge(st["full"], delta)]


def _out_rows(program: str, case: dict, edges: float) -> float:
    """Expected result rows, from the generators' measured closures."""
    if program == "tc":
        if case.get("graph") == "chung_lu":
            return 0.0187 * _chung_lu_nodes(int(edges)) ** 2
        return 55.0 * edges / 1.1
    if program == "sg":
        if case.get("graph") == "mesh":
            return 0.5 * case["side"] ** 6
        return 3.2 * edges
    if program == "wcc":
        return edges * 0.0006 + 1
    r2 = float(case["range"]) ** 2  # distinct pairs among edges^2 / range join rows
    return r2 * -math.expm1(-edges * edges / case["range"] / r2)


def work(case: dict) -> dict:
    """Each input row read once and each result row (or label) written once,
    8 bytes each; the engine does no floating-point work."""
    if case["kind"] == "program":
        m = float(case["edges"]) if "edges" in case else 6 * case["percent"] / 100 * case["side"] ** 3
        rows = m + _out_rows(case["program"], case, m)
        if case["program"] == "wcc":
            rows += _chung_lu_nodes(case["edges"])  # a node id and a label, 4 bytes each
    elif case["kind"] in ("batch", "session"):
        rows = sum(m + _out_rows(case["program"], {}, m) for m in _sizes(case))
        if case["program"] == "wcc":
            rows += sum(_sizes(case)) / 3.3 / 2  # a 4-byte label per node
    else:
        m, r2 = float(case["edges"]), float(case["range"]) ** 2
        joined = r2 * -math.expm1(-m * m / case["range"] / r2)
        rows = 2 * m + case["full"] + joined + joined + case["full"] + joined
    return {"bytes": 8.0 * rows, "flops": 0.0}


def exact(case: dict, seed: int):
    return None
