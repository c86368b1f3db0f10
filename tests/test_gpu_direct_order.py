"""GPU tests of fragments in order through the direct-mapped brick table, whose
marking merges a row's runs of equal bricks and consecutive rows of one brick:
runs at and around its limits (rows of 32, eight runs, eight rows, a CTA's 2048
fragments), sorted and repeated lists, out-of-range codes inside a run."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def runs(lengths, n, depth, seed):
    """n fragments in runs of one brick each, the run lengths in turn; the bricks differ from run to run."""
    rng = np.random.default_rng(seed)
    reps = np.resize(np.asarray(lengths), n)
    reps = reps[: int(np.searchsorted(np.cumsum(reps), n)) + 1]
    brick = rng.integers(0, 8 ** (depth - 2), reps.size, dtype=np.uint64)
    brick[1:] ^= (brick[1:] == brick[:-1]).astype(np.uint64)
    b = np.repeat(brick, reps)[:n]
    return (b << np.uint64(6)) | rng.integers(0, 64, n, dtype=np.uint64)


LENGTHS = {"rows": [32], "off_by_one": [31, 33], "eight_runs": [4], "nine_runs": [4, 4, 4, 4, 4, 4, 4, 3, 1],
           "seven_and_one": [5, 5, 5, 5, 5, 6, 1], "whole_then_split": [64, 16, 16, 96, 1, 31], "eight_rows": [256],
           "past_eight_rows": [257], "cta": [2048], "past_cta": [2049], "mixed": [1, 1, 1, 300, 2, 7, 500, 1]}


@pytest.mark.parametrize("depth", [3, 5, 10])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_runs_bit_exact(name, depth):
    with D.Context(0) as c:
        for n in (1, 31, 33, 255, 2048, 2049, 70_001):
            codes = runs(LENGTHS[name], n, depth, n + depth)
            assert_dag_equal(c.create_dag(codes, depth).to_host(), O.create_dag(codes, depth))


@pytest.mark.parametrize("depth,n", [(2, 40_000), (5, 400_000), (8, 400_000), (10, 300_000)])
def test_sorted_and_repeated_bit_exact(depth, n):
    rng = np.random.default_rng(depth)
    lists = [np.sort(rng.integers(0, 8**depth, n, dtype=np.uint64)), np.repeat(rng.integers(0, 8**depth, n // 50, dtype=np.uint64), 50),
             np.sort(rng.integers(0, min(8**depth, n // 20), n, dtype=np.uint64)), np.zeros(n, np.uint64),
             np.full(n, 8**depth - 1, np.uint64)]
    with D.Context(0) as c:
        for codes in lists:
            assert_dag_equal(c.create_dag(codes, depth).to_host(), O.create_dag(codes, depth))


@pytest.mark.parametrize("at", [0, 1, 31, 32, 2047, 4999])
def test_a_code_out_of_range_inside_a_run(at):
    codes = np.full(5000, 77, np.uint64)
    bad = codes.copy()
    bad[at] = np.uint64(8**6)
    huge = codes.copy()
    huge[at] = np.uint64(0xFFFFFFFFFFFFFFFF)
    with D.Context(0) as c:
        for x in (bad, huge):
            with pytest.raises(D.DagcError) as e:
                c.create_dag(x, 6)
            assert e.value.status == D.ERR_BAD_INPUT
            assert_dag_equal(c.create_dag(codes, 6).to_host(), O.create_dag(codes, 6))
