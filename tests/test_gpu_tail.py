"""GPU tests of the one-CTA tail at the edges of its range: levels of up to 4096
children (where it starts depends on the counts), of up to 32 (one warp), every
level of the deepest DAG, many equal nodes."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def scattered(depth, bricks, seed, distinct=True):
    """Fragments in `bricks` bricks spread over the volume; their masks all
    different, or all one mask (so that nodes repeat)."""
    rng = np.random.default_rng(seed)
    space = 8 ** (depth - 2)
    if bricks * 4 > space:
        b = rng.choice(space, bricks, replace=False).astype(np.uint64)
    else:
        b = np.unique(rng.integers(0, space, 2 * bricks, dtype=np.uint64))
        b = rng.choice(b, bricks, replace=False)
    if not distinct:
        return rng.permutation((b << np.uint64(6)) | np.uint64(21))
    k = np.arange(bricks, dtype=np.uint64)
    return rng.permutation(np.concatenate([(b << np.uint64(6)) | (k & np.uint64(63)), (b << np.uint64(6)) | (k >> np.uint64(6)) % np.uint64(64)]))


@pytest.mark.parametrize("depth,bricks", [(3, 1), (3, 8), (4, 64), (6, 31), (9, 32), (9, 33), (8, 4095), (8, 4096), (8, 4097),
                                          (12, 4096), (12, 4097), (11, 20_000), (21, 1), (21, 32), (21, 33), (21, 4096)])
@pytest.mark.parametrize("distinct", [True, False])
def test_tail_start_bit_exact(depth, bricks, distinct):
    codes = scattered(depth, bricks, depth * 10007 + bricks, distinct)
    ref = O.create_dag(codes, depth)
    with D.Context(0) as c:
        for _ in range(3):  # direct launches, recording, replay
            assert_dag_equal(c.create_dag(codes, depth).to_host(), ref)
        assert np.array_equal(c.compress(codes, depth).to_numpy(), O.final_dag(ref))
        assert c.dedup_fallbacks() == 0
        c.set_option(D.OPT_DEDUP, 0)  # the radix form: the tail starts where the bounds say
        assert_dag_equal(c.create_dag(codes, depth).to_host(), ref)
