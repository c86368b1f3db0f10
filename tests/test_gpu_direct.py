"""GPU tests of the leaves by a direct-mapped brick table: the default path up
to depth 10, and at depth 11 from 2^21 fragments on. Bit-exact against the
oracle at the edges of its blocks (64 bricks), of its two compaction forms
(depth 8 / 9) and of its fragment limit."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import random_codes
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def blocks_edges(depth):
    """Fragments in the first, last and block-boundary bricks of the volume."""
    bricks = 8 ** (depth - 2)
    b = np.array([x for x in (0, 1, 31, 32, 63, 64, 65, 511, 512, 4095, 4096, bricks // 2, bricks - 65, bricks - 64, bricks - 1)
                  if 0 <= x < bricks], np.uint64)
    return np.concatenate([(b << np.uint64(6)) | np.uint64(v) for v in (0, 31, 32, 63)])


def dense(depth):
    """Every brick, one voxel each."""
    b = np.arange(8 ** (depth - 2), dtype=np.uint64)
    return np.random.default_rng(depth).permutation((b << np.uint64(6)) | (b * np.uint64(7) & np.uint64(63)))


CASES = {
    "edges_d2": lambda: (blocks_edges(2), 2), "edges_d5": lambda: (blocks_edges(5), 5),
    "edges_d6": lambda: (blocks_edges(6), 6), "edges_d8": lambda: (blocks_edges(8), 8),
    "edges_d9": lambda: (blocks_edges(9), 9),
    "edges_d10": lambda: (blocks_edges(10), 10), "edges_d11": lambda: (blocks_edges(11), 11),
    "dense_d5": lambda: (dense(5), 5), "dense_d7": lambda: (dense(7), 7),
    "one_code": lambda: (np.full(70_001, (1 << 30) - 1, np.uint64), 10),
    "few_bricks": lambda: (np.random.default_rng(1).integers(0, 256, 300_001, dtype=np.uint64), 9),
    "ragged_d9": lambda: (random_codes(9, 65_537, 2), 9),
    "below_limit_d11": lambda: (random_codes(11, 2**21 - 1, 3), 11),
    "at_limit_d11": lambda: (random_codes(11, 2**21, 4), 11),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_direct_table_bit_exact(case):
    codes, depth = CASES[case]()
    ref = O.create_dag(codes, depth, threads=8)
    with D.Context(0) as c:
        for _ in range(3):  # direct launches, recording, replay: the table is empty again after each
            assert_dag_equal(c.create_dag(codes, depth).to_host(), ref)
        assert np.array_equal(c.compress(codes, depth).to_numpy(), O.final_dag(ref))
        assert c.dedup_fallbacks() == 0


def test_grouped_bricks_ordered_by_the_table():
    """Depth 11, many fragments per brick: grouped by hash, the bricks put in
    order by the table; equal to the brick sort (grouping forced)."""
    rng = np.random.default_rng(7)
    bricks = rng.choice(8**9, 40_000, replace=False).astype(np.uint64)
    bricks[:2] = 0, 8**9 - 1
    codes = (bricks[rng.integers(0, bricks.size, 2**21 + 5)] << np.uint64(6)) | rng.integers(0, 64, 2**21 + 5, dtype=np.uint64)
    ref = O.create_dag(codes, 11, threads=8)
    for mode in (1, 2):
        with D.Context(0) as c:
            c.set_option(D.OPT_GROUP, mode)
            for _ in range(3):
                assert_dag_equal(c.create_dag(codes, 11).to_host(), ref)
            assert c.dedup_fallbacks() == 0


def test_direct_table_is_clean_after_bad_input_and_across_depths():
    a, b = random_codes(10, 50_000, 5), random_codes(7, 50_000, 6)
    bad = a.copy()
    bad[777] = np.uint64(1 << 30)
    with D.Context(0) as c:
        for _ in range(2):
            assert_dag_equal(c.create_dag(b, 7).to_host(), O.create_dag(b, 7))  # the table grows after this
            with pytest.raises(D.DagcError) as e:
                c.create_dag(bad, 10)
            assert e.value.status == D.ERR_BAD_INPUT
            assert_dag_equal(c.create_dag(a, 10).to_host(), O.create_dag(a, 10))
        c.free_all()
        assert_dag_equal(c.create_dag(b, 7).to_host(), O.create_dag(b, 7))
