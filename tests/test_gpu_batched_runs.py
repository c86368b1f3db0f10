"""GPU test of the batched form's runs of tiles (two to four 8192-fragment tiles
per work item from ~10M fragments on) and of its groups of bins: chunks that end
at, before and after a tile and a run, against the oracle's whole volume."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.test_gpu_batched import global_codes
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk_depth,sizes", [
    (10, (8191, 0, 8192, 8193, 16_384, 16_385, 32_768, 1, 25_600_000)),       # ragged ends, runs of four tiles
    (7, (11_000_001, 40_000, 65_536)),                                         # four bins per chunk, runs of two
    (8, (700, 90_000, 8192, 0, 41)),                                           # one bin per item
])
def test_batched_runs_and_groups(chunk_depth, sizes):
    rng = np.random.default_rng(chunk_depth)
    bricks = rng.choice(8 ** (chunk_depth - 2), min(30_000, 8 ** (chunk_depth - 2) // 2), replace=False).astype(np.uint64)
    bricks[:2] = 0, 8 ** (chunk_depth - 2) - 1
    # Repeated voxels: few codes, so that the oracle's tree stays small.
    pool = (bricks[rng.integers(0, bricks.size, 200_000)] << np.uint64(6)) | rng.integers(0, 64, 200_000, dtype=np.uint64)
    chunks = [pool[rng.integers(0, pool.size, n)] for n in sizes]
    morton = np.sort(rng.choice(64, len(sizes), replace=False)).astype(np.uint64)
    counts = np.array(sizes, np.uint64)
    whole = O.create_dag(np.unique(global_codes(chunks, morton, chunk_depth)), chunk_depth + 2, threads=8)
    frag = np.concatenate(chunks)
    with D.Context(0) as c:
        for _ in range(3):  # direct launches, recording, replay
            assert_dag_equal(c.create_dag_batched(frag, counts, morton, chunk_depth, 2).to_host(), whole)
        assert c.dedup_fallbacks() == 0
