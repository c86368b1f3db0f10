"""GPU tests of the final layout whose positions are made with the call: one
node a level, sparse volumes with as many nodes on every level as fragments,
a full tree, positions over one tile and over many."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,n", [(2, 5), (3, 1), (3, 512), (5, 4000), (8, 300_000), (12, 3000), (16, 60_000), (21, 1), (21, 341)])
def test_words_equal_general_form(depth, n):
    codes = np.random.default_rng(depth * 7 + n).integers(0, 8 ** depth, n, dtype=np.uint64)
    words = O.final_dag(O.create_dag(codes, depth))
    with D.Context(0) as c:
        for _ in range(3):  # direct launches, recording, replay
            assert np.array_equal(c.compress(codes, depth).to_numpy(), words)
            dag = c.create_dag(codes, depth)  # the same call without the positions
            assert np.array_equal(c.create_final_dag(dag).to_numpy(), words)
        c.set_option(D.OPT_DEDUP, 0)
        assert np.array_equal(c.compress(codes, depth).to_numpy(), words)
