"""Buffers behind handles: hash tables and join outputs come from the context's
cache and go back to it, whatever the order in which they are given up."""
import ctypes as C

import numpy as np
import pytest

from mnmgdatalog_b200 import DatalogError, Engine, graphs

pytestmark = pytest.mark.gpu


def _pairs(n, m, seed):
    import torch
    return torch.from_numpy(np.random.default_rng(seed).integers(0, n, (m, 2)).astype(np.int32)).cuda()


def test_hash_table_outlives_its_context():
    with Engine(0) as eng:
        ht = eng.get_hash_table(_pairs(50, 400, 1))
    ht.close()  # the context is gone: the memory is freed


def test_reused_buffers_hold_no_old_rows():
    from oracle import ops
    with Engine(0) as eng:
        for seed, (n, m) in enumerate([(500, 4000), (20, 300), (500, 4000), (3000, 9000), (20, 300)]):
            rel, probe = _pairs(n, m, seed), _pairs(n, m // 2, 100 + seed)
            ht = eng.get_hash_table(rel)
            got = eng.get_join(ht, probe).cpu().numpy()
            want = ops.join(rel.cpu().numpy(), probe.cpu().numpy())
            order = lambda a: a[np.lexsort((a[:, 1], a[:, 0]))]  # noqa: E731
            assert np.array_equal(order(got), order(np.asarray(want)))
            ht.close()


def test_join_outputs_are_separate_and_freed_once():
    from mnmgdatalog_b200.capi import check, lib
    with Engine(0) as eng:
        ht = eng.get_hash_table(_pairs(100, 2000, 1))
        probe = _pairs(100, 500, 2)
        ptrs = []
        for _ in range(3):
            out, n = C.c_void_p(), C.c_int64()
            check(lib().dl_join(eng.ctx, ht.handle, C.c_void_p(probe.data_ptr()), len(probe), C.byref(out), C.byref(n)))
            ptrs.append(out.value)
        assert len(set(ptrs)) == 3
        for p in ptrs:
            check(lib().dl_free(eng.ctx, C.c_void_p(p)))
        ht.close()


@pytest.mark.parametrize("prog", ["tc", "sg", "wcc"])
def test_results_in_one_call(engine, prog):
    sets = [graphs.dag(n=300, extra=90, seed=1), np.zeros((0, 2), np.int32), graphs.dag(n=80, extra=10, seed=2)]
    with engine.session(prog) as s:
        ids = s.admit_many(sets)
        s.run()
        for out in ("host", "device", "none"):
            for i, r in zip(reversed(ids), s.results(reversed(ids), output=out, labels=True)):
                w = s.result(i, output=out, labels=True)
                if out != "none":
                    assert np.array_equal(np.asarray(r.rows.cpu() if out == "device" else r.rows),
                                          np.asarray(w.rows.cpu() if out == "device" else w.rows))
                if prog == "wcc":
                    assert np.array_equal(r.labels, w.labels) and np.array_equal(r.node_ids, w.node_ids)
        assert s.results([]) == []
        with pytest.raises(DatalogError):
            s.results([99])


def test_bit_rows_take_at_most_half_of_the_free_memory():
    """SG's three bit-row matrices (0.8 GB) while 1.2 GB are free and 1.9 cached in buffers that
    none of them fits into: those are freed first, or another form runs."""
    import torch
    rng = np.random.default_rng(3)
    e = np.concatenate([rng.integers(0, 46_000, (70_000, 2)), [[0, 45_999]]]).astype(np.int32)
    with Engine(0) as eng:
        want = eng.sg(e, max_iterations=1)
    with Engine(0) as eng:
        eng.sg(e[:3000], max_iterations=1)  # the workspace's small buffers
        rel = torch.stack([torch.randperm(4_000_000, device="cuda", dtype=torch.int32)] * 2, 1).contiguous()
        tables = [eng.get_hash_table(rel) for _ in range(12)]  # 0.14 GB each
        del rel
        torch.cuda.empty_cache()
        for t in tables:
            t.close()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 1200 * 2**20, dtype=torch.uint8, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        got = eng.sg(e, max_iterations=1)
        after = torch.cuda.mem_get_info()[0]
        del fill
        torch.cuda.empty_cache()
        assert before < 1300 * 2**20 and after >= before // 2
        assert got.deltas.tolist() == want.deltas.tolist() and np.array_equal(got.rows, want.rows)


def _held(eng, prog, e, **kw):
    """Device bytes that a run took from a fresh context, and those that its result keeps
    when the context's workspace and cache are freed."""
    import torch
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    seen = []

    def at_output(rows):
        seen.append(before - torch.cuda.mem_get_info()[0])
        eng.release_memory()
        seen.append(before - torch.cuda.mem_get_info()[0])
        return torch.empty((rows, 2), dtype=torch.int32, device="cuda")

    got = eng.run(prog, e, output="device", out=at_output, **kw)
    return got, seen


def test_searches_take_room_by_the_result_not_by_the_nodes():
    """8M edges to 8M sinks: 64 MB of rows (12 GB were reserved before anything was found)."""
    import torch
    k = torch.arange(8_000_000, dtype=torch.int32, device="cuda")
    e = torch.stack([k, k + 8_000_000], 1).contiguous()
    with Engine(0) as eng:
        got, (taken, kept) = _held(eng, "tc", e)
        assert got.output_tuples == len(e) and taken < 4 * 2**30 and kept < 2**29
        assert torch.equal(got.rows, e)


@pytest.mark.parametrize("prog,edges", [("tc", 300_000), ("tc", 3_000_000), ("sg", 60_000), ("sg", 1_000_000)])
def test_results_do_not_hold_the_searchs_room(prog, edges):
    """A few words a node: the run keeps at most 64 MiB beside four times its words and its ids."""
    k = np.arange(edges, dtype=np.int32)
    e = np.stack([k // 2 if prog == "sg" else k, k + edges], 1)
    with Engine(0) as eng:
        got, (_, kept) = _held(eng, prog, e)
        assert kept < 4 * 8 * got.output_tuples + 2 * 4 * 2 * edges + (72 << 20)
        want = eng.run(prog, e, dedup="sort")
        assert np.array_equal(got.rows.cpu().numpy(), want.rows) and got.deltas.tolist() == want.deltas.tolist()


def test_tc_without_room_for_bit_rows():
    """Heavy sources whose rows pass bitmap_max_gib (2.1 GB at 1 GiB): the bit matrix (0.3 GB) runs."""
    e = np.random.default_rng(2).integers(0, 76_000, (220_000, 2)).astype(np.int32)
    with Engine(0) as eng:
        want = eng.tc(e, output="none", max_iterations=9)
        eng.set_tuning(bitmap_max_gib=1)
        got = eng.tc(e, output="none", max_iterations=9)
        assert got.deltas.tolist() == want.deltas.tolist() and got.output_tuples == want.output_tuples


def _permutation(n):
    import torch
    return torch.stack([torch.randperm(n, device="cuda", dtype=torch.int32)] * 2, 1).contiguous()


def test_large_join_output_while_the_cache_holds_the_memory():
    """1.7 GB of closed hash tables are cached, 0.7 GB are free: an output of 1.2 GB takes the cache's."""
    import torch
    with Engine(0) as eng:
        rel = _permutation(4_000_000)
        tables = [eng.get_hash_table(rel) for _ in range(12)]
        one = torch.zeros((12_000, 2), dtype=torch.int32, device="cuda")
        ht = eng.get_hash_table(one)  # 12,000 rows of one key
        probe = one[:12_500]
        del rel
        torch.cuda.empty_cache()
        for t in tables:
            t.close()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 700 * 2**20, dtype=torch.uint8, device="cuda")
        out, n = C.c_void_p(), C.c_int64()
        from mnmgdatalog_b200.capi import check, lib
        check(lib().dl_join(eng.ctx, ht.handle, C.c_void_p(probe.data_ptr()), len(probe), C.byref(out), C.byref(n)))
        assert n.value == 12_000 * len(probe)
        check(lib().dl_free(eng.ctx, out))
        ht.close()
        del fill
        torch.cuda.empty_cache()


def test_a_cache_of_zero_keeps_no_handles_buffers():
    import torch
    rel = _permutation(1_000_000)
    with Engine(0) as eng:
        eng.get_hash_table(rel).close()  # the workspace
        eng.set_tuning(cache_max_gib=0)
        free = torch.cuda.mem_get_info()[0]
        tables = [eng.get_hash_table(rel) for _ in range(4)]
        for t in tables:
            t.close()
        assert torch.cuda.mem_get_info()[0] >= free
        eng.set_tuning(cache_max_gib=96)
        for t in [eng.get_hash_table(rel) for _ in range(4)]:
            t.close()
        assert torch.cuda.mem_get_info()[0] < free
        eng.set_tuning(cache_max_gib=0)  # what is cached goes too
        assert torch.cuda.mem_get_info()[0] >= free


def test_join_output_freed_twice_is_refused():
    """A freed output is the cache's: freeing it again must not take it from there."""
    from mnmgdatalog_b200.capi import check, lib
    from oracle import ops
    with Engine(0) as eng:
        rel, probe = _pairs(200, 3000, 5), _pairs(200, 800, 6)
        ht = eng.get_hash_table(rel)
        out, n = C.c_void_p(), C.c_int64()
        check(lib().dl_join(eng.ctx, ht.handle, C.c_void_p(probe.data_ptr()), len(probe), C.byref(out), C.byref(n)))
        assert lib().dl_free(eng.ctx, out) == 0
        assert lib().dl_free(eng.ctx, out) != 0
        got = np.sort(eng.get_join(ht, probe).cpu().numpy().view(np.int64).ravel())  # reuses the buffer
        want = np.ascontiguousarray(ops.join(rel.cpu().numpy(), probe.cpu().numpy()), dtype=np.int32)
        assert np.array_equal(got, np.sort(want.view(np.int64).ravel()))
        ht.close()


def test_the_cache_makes_room_for_bit_rows():
    """0.5 GB free, 4.3 GB cached in buffers too small for SG's matrices (0.8 GB): the run takes the
    form that it takes when the memory is free."""
    import torch
    rng = np.random.default_rng(3)
    e = np.concatenate([rng.integers(0, 46_000, (70_000, 2)), [[0, 45_999]]]).astype(np.int32)

    def launches(eng):
        eng.profile(False)
        got = eng.sg(e, max_iterations=3)
        return got, eng.profile_read()["bitmap_expand"]["launches"]

    with Engine(0) as eng:
        want, of_rows = launches(eng)
    with Engine(0) as eng:
        rel = _permutation(4_000_000)
        tables = [eng.get_hash_table(rel) for _ in range(30)]
        del rel
        torch.cuda.empty_cache()
        for t in tables:
            t.close()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 500 * 2**20, dtype=torch.uint8, device="cuda")
        got, n = launches(eng)
        del fill
        torch.cuda.empty_cache()
    assert n == of_rows and np.array_equal(got.rows, want.rows)


def test_the_workspace_of_other_forms_makes_room_for_the_matrix():
    """After TC on bit rows (8 GB, two thirds of it workspace) 1 GB is free: SG that goes to the bit
    matrix (2 GB) still does, and not to the sorted runs, whose join sizes are others."""
    import torch
    rng = np.random.default_rng(5)
    tc = rng.integers(0, 150_000, (430_000, 2)).astype(np.int32)
    sg = np.concatenate([rng.integers(0, 125_000, (132_000, 2)), [[0, 124_999]]]).astype(np.int32)
    with Engine(0) as eng:
        want = eng.sg(sg, max_iterations=25)
    with Engine(0) as eng:
        eng.tc(tc, output="none")
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 2**30, dtype=torch.uint8, device="cuda")
        got = eng.sg(sg, max_iterations=25)
        del fill
        torch.cuda.empty_cache()
    assert got.join_rows.tolist() == want.join_rows.tolist() and np.array_equal(got.rows, want.rows)
    assert got.nodes == want.nodes


def test_an_empty_batch_takes_any_output():
    with Engine(0) as eng:
        assert eng.run_batch("tc", [], output="nowhere") == []
        with pytest.raises(DatalogError):
            eng.run_batch("tc", [np.array([[1, 2]], np.int32)], output="nowhere")
