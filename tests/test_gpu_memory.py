"""GPU tests of what a context does when device memory runs out, by injected
allocation failures: a form that needs more memory than another gives way to
it, and the results stay bit-exact."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import chunks_of, random_codes
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def test_a_union_without_room_for_the_hash_set_goes_by_sorts():
    codes = random_codes(9, 120_000, 51)
    chunks, sub = chunks_of(codes, 9, 1)
    with D.Context(0) as c:
        dags = [c.create_dag(x, sub) for x in chunks]
        c.free_all()  # the union's scratch has to be allocated
        before = c.dedup_fallbacks()
        c.set_option(D.OPT_TEST_FAIL_ALLOCS, 2)  # the hash-set form's scratch and its retry fail
        body, roots = c.union_dags(dags)
        assert c.dedup_fallbacks() == before + 1
        assert_dag_equal(c.lift_dag(body, roots).to_host(), O.create_dag(codes, 9))
        assert_dag_equal(c.merge_dags(dags).to_host(), O.create_dag(codes, 9))  # by hash set again
        assert c.dedup_fallbacks() == before + 1


def test_a_union_without_room_for_the_table_goes_by_sorts():
    parts = [random_codes(10, 60_000, 60 + i) for i in range(4)]
    with D.Context(0) as c, D.Context(0) as other:
        dags = [other.create_dag(p, 10) for p in parts]
        ref = other.union_dags(dags)[0].to_host()
        # A context with a large arena and a small table: many fragments of few bricks, through the radix sort.
        c.set_option(D.OPT_GROUP, 0)
        c.create_dag(random_codes(4, 20_000_000, 64), 4).free()
        before, fell = c.memory_events(), c.dedup_fallbacks()
        c.set_option(D.OPT_TEST_FAIL_ALLOCS, 2)  # the table's allocation and its retry
        got = c.union_dags(dags)[0].to_host()
        assert c.memory_events()["alloc_failures"] == before["alloc_failures"] + 2
        assert c.dedup_fallbacks() == fell + 1
        assert_dag_equal(got, ref)


def has_brick_table(c):
    return "brick table" in c.memory_report()


def test_idle_brick_tables_are_given_back_to_any_allocation():
    """The voxelizer's scratch in one context takes the idle tables of both; each is taken again and exact."""
    codes = random_codes(10, 30_000, 71)
    ref = O.final_dag(O.create_dag(codes, 10))
    tri = np.random.default_rng(72).uniform(0, 64, (5_000, 9))
    with D.Context(0) as a, D.Context(0) as b:
        for c in (a, b):
            assert np.array_equal(c.compress(codes, 10).to_numpy(), ref)
            assert has_brick_table(c)
        before = a.memory_events()
        a.set_option(D.OPT_TEST_FAIL_ALLOCS, 1)
        a.voxelize(tri, (0, 0, 0, 64, 64, 64), 6)
        after = a.memory_events()
        assert (after["alloc_failures"], after["retries_ok"]) == (before["alloc_failures"] + 1, before["retries_ok"] + 1)
        assert not has_brick_table(a) and not has_brick_table(b)
        for c in (a, b):
            for _ in range(3):
                assert np.array_equal(c.compress(codes, 10).to_numpy(), ref)
            assert has_brick_table(c)


@pytest.mark.parametrize("graphs", [0, 1])
def test_a_call_without_room_for_the_brick_table(graphs):
    """Only the table's allocation fails: the call does without it, the next one takes it."""
    import torch
    big = random_codes(9, 1_500_000, 81)
    codes = torch.from_numpy(random_codes(10, 20_000, 82).view(np.int64)).cuda()
    ref = O.final_dag(O.create_dag(codes.cpu().numpy().view(np.uint64), 10))
    with D.Context(0) as c:
        c.set_option(D.OPT_GRAPHS, graphs)
        c.set_option(D.OPT_GROUP, 2)
        c.compress(big, 9).free()  # scratch and tables larger than the next call's, but for the brick table
        c.set_option(D.OPT_GROUP, 1)
        for turn in range(2):
            before = c.memory_events()
            c.set_option(D.OPT_TEST_FAIL_ALLOCS, 1)
            assert np.array_equal(c.compress(codes, 10).to_numpy(), ref)
            after = c.memory_events()
            assert (after["alloc_failures"], after["retries_ok"]) == (before["alloc_failures"] + 1, before["retries_ok"])
            assert not has_brick_table(c)
            for _ in range(3):
                assert np.array_equal(c.compress(codes, 10).to_numpy(), ref)
            assert has_brick_table(c)
            if turn == 0:
                c.voxelize(np.zeros((1, 9)), (0, 0, 0, 1, 1, 1), 1)
                c.set_option(D.OPT_TEST_FAIL_ALLOCS, 1)  # takes the table back for the second turn
                c.voxelize(np.zeros((90_000, 9)), (0, 0, 0, 1, 1, 1), 1)
                c.set_option(D.OPT_TEST_FAIL_ALLOCS, 0)


def test_a_server_jobs_staging_buffer():
    small, many = random_codes(9, 300_000, 91), random_codes(5, 2_000_000, 92)
    ref = O.final_dag(O.create_dag(many, 5))
    srv = D.Server(0, slots=1, hbm_budget_bytes=64 << 30)
    try:
        srv.wait(srv.submit(small, 9))
        srv.set_option(D.OPT_TEST_FAIL_ALLOCS, 2)  # of the next job only its staging buffer has to grow
        with pytest.raises(D.DagcError) as e:
            srv.wait(srv.submit(many, 5))
        assert e.value.status == D.ERR_OUT_OF_MEMORY
        srv.set_option(D.OPT_TEST_FAIL_ALLOCS, 1)
        assert np.array_equal(srv.wait(srv.submit(many, 5))[0], ref)
    finally:
        srv.close()


def test_grouping_scratch_only_for_calls_that_group():
    """Marked straight into the brick table, or chunk by chunk: no grouping scratch; deeper volumes take it."""
    with D.Context(0) as c:
        codes = random_codes(9, 20_000, 101)
        assert np.array_equal(c.compress(codes, 9).to_numpy(), O.final_dag(O.create_dag(codes, 9)))
        chunks, sub = chunks_of(codes, 9, 1)
        batched = c.create_dag_batched(np.concatenate(chunks), [x.size for x in chunks], list(range(8)), sub, 1)
        assert_dag_equal(batched.to_host(), O.create_dag(codes, 9))
        assert "grouping table" not in c.memory_report()
        deep = random_codes(12, 20_000, 102, cluster=True)
        assert np.array_equal(c.compress(deep, 12).to_numpy(), O.final_dag(O.create_dag(deep, 12)))
        assert "grouping table" in c.memory_report()


def test_the_depth_11_table_only_once_fragments_are_grouped():
    """1 GB, and of use only to grouped fragments: not for sorted ones, and from the second grouped call on (launched,
    recorded, replayed)."""
    sparse = random_codes(11, 2**21, 111)
    rng = np.random.default_rng(112)
    bricks = rng.integers(0, 8**9, 30_000, dtype=np.uint64)
    crowded = (bricks[rng.integers(0, bricks.size, 2**21 + 77)] << np.uint64(6)) | rng.integers(0, 64, 2**21 + 77, dtype=np.uint64)
    refs = [O.final_dag(O.create_dag(x, 11, threads=8)) for x in (sparse, crowded)]
    with D.Context(0) as c:
        import torch
        sparse, crowded = (torch.from_numpy(x.view(np.int64)).cuda() for x in (sparse, crowded))
        for _ in range(3):
            assert np.array_equal(c.compress(sparse, 11).to_numpy(), refs[0])
        assert np.array_equal(c.compress(crowded, 11).to_numpy(), refs[1])
        assert not has_brick_table(c)
        for _ in range(4):
            assert np.array_equal(c.compress(crowded, 11).to_numpy(), refs[1])
            assert has_brick_table(c)
        assert np.array_equal(c.compress(sparse, 11).to_numpy(), refs[0])
        c.free_all()
        assert np.array_equal(c.compress(crowded, 11).to_numpy(), refs[1])


def test_brick_table_option_gives_it_back():
    codes = random_codes(10, 40_000, 121)
    ref = O.final_dag(O.create_dag(codes, 10))
    with D.Context(0) as c:
        for on in (1, 0, 1):
            c.set_option(D.OPT_BRICK_TABLE, on)
            assert not has_brick_table(c) or on
            for _ in range(3):
                assert np.array_equal(c.compress(codes, 10).to_numpy(), ref)
            assert has_brick_table(c) == bool(on)


@pytest.mark.parametrize("room", ["tight", "roomy"])
def test_server_budget_holds_the_brick_tables(room):
    """Tight: as many jobs side by side as their scratch allows, without tables, inside the budget. Roomy: tables, and
    they count."""
    jobs = [random_codes(10, 2_000 + i, 130 + i) for i in range(12)]
    table = 8 * 8**8
    need = max(D.create_footprint(x.size, 10) + 24 * x.size for x in jobs)
    assert need < table
    budget = 4 * need if room == "tight" else 16 << 30
    srv = D.Server(0, slots=4, hbm_budget_bytes=budget)
    try:
        for _ in range(2):
            tickets = [srv.submit(x, 10) for x in jobs]
            for x, t in zip(jobs, tickets):
                assert np.array_equal(srv.wait(t)[0], O.final_dag(O.create_dag(x, 10)))
        s = srv.stats()
        assert s["max_concurrent"] >= 2
        assert s["peak_footprint"] <= budget
        if room == "roomy":
            assert s["peak_footprint"] > table
    finally:
        srv.close()
