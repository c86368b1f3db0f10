"""GPU tests of MergeDAGs by hash set (all levels at once) against the form by
one sort per level and the oracle: few and many inputs, empty ones, equal ones,
merges of merges, deep DAGs, and uploads with a hash or a leaf of zero."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import chunks_of, random_codes
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def both_forms(build):
    """build(ctx) in the hash-set form and in the sort form; the two are equal."""
    out = []
    for form in (1, 0):
        with D.Context(0) as c:
            c.set_option(D.OPT_DEDUP, form)
            out.append(build(c).to_host())
    assert_dag_equal(out[0], out[1])
    return out[0]


@pytest.mark.parametrize("depth,levels_up,n,cluster", [(3, 1, 300, False), (5, 2, 4000, True), (9, 1, 300_000, False),
                                                       (11, 1, 400_000, True), (7, 3, 60_000, True)])
def test_merge_forms_equal_the_whole_volume(depth, levels_up, n, cluster):
    codes = random_codes(depth, n, depth * 31 + n, cluster=cluster)
    chunks, sub = chunks_of(codes, depth, levels_up)
    got = both_forms(lambda c: c.merge_dags([c.create_dag(x, sub) for x in chunks]))
    assert_dag_equal(got, O.create_dag(codes, depth))


def test_merge_of_equal_inputs_and_of_merges():
    codes = random_codes(6, 5000, 3)

    def build(c):
        once = [c.merge_dags([c.create_dag(codes if i % 3 else np.zeros(0, np.uint64), 6) for i in range(8)]) for _ in range(8)]
        return c.merge_dags(once)

    got = both_forms(build)
    assert got.level_sizes()[0] == 1 and got.level_sizes()[1] == 1


def test_union_of_three():
    parts = [random_codes(8, 20_000, s, cluster=bool(s & 1)) for s in (1, 2, 3)]
    got = both_forms(lambda c: c.union_dags([c.create_dag(p, 8) for p in parts])[0])
    assert got.level_sizes()[0] == 3


def test_merge_deeper_than_the_deepest_volume():
    """19 levels, then 20 and 21 (past the hash-set form's levels)."""
    def build(c):
        def one(seed):
            return c.create_dag(random_codes(21, 3, seed) >> np.uint64(1), 21)
        return c.merge_dags([c.merge_dags([one(8 * j + i) for i in range(8)]) for j in range(8)])

    assert both_forms(build).num_levels == 21


@pytest.mark.parametrize("zero", ["hash", "leaf"])
def test_uploaded_zero_takes_the_sort_form(zero):
    """0 marks an empty slot of the hash set: such inputs are merged by sorts."""
    empty = D.HostDag(masks=[np.zeros(0, np.uint8)], children=[np.zeros((0, 8), np.uint32)], hashes=[np.zeros(0, np.uint64)],
                      leaves=np.zeros(0, np.uint64))
    one = D.HostDag(masks=[np.array([1], np.uint8)], children=[np.array([[0] + [0xFFFFFFFF] * 7], np.uint32)],
                    hashes=[np.array([0 if zero == "hash" else 5], np.uint64)],
                    leaves=np.array([0 if zero == "leaf" else 9], np.uint64))
    other = D.HostDag(masks=[np.array([2], np.uint8)], children=[np.array([[0xFFFFFFFF, 0] + [0xFFFFFFFF] * 6], np.uint32)],
                      hashes=[np.array([77], np.uint64)], leaves=np.array([3], np.uint64))
    got = both_forms(lambda c: c.union_dags([c.upload_dag(x) for x in (one, other, empty)])[0])
    assert got.level_sizes() == [2] and got.leaves.size == 2
