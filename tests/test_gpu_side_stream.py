"""GPU tests of the node extraction that runs beside a call's stream: a call
that fails while it is queued waits for it, directly launched or while its
shape is recorded, and the calls after it (which write the same scratch) are
bit-exact."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import random_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("depth,n", [(6, 3_000), (12, 300_000)])
def test_a_call_that_fails_beside_its_stream(depth, n, graphs):
    import torch
    codes = torch.from_numpy(random_codes(depth, n, 21).view(np.int64)).cuda()
    other = random_codes(depth, n - 7, 22)
    ref = O.final_dag(O.create_dag(codes.cpu().numpy().view(np.uint64), depth))
    ref_other = O.final_dag(O.create_dag(other, depth))
    with D.Context(0) as c:
        c.set_option(D.OPT_GRAPHS, graphs)
        for _ in range(3):  # a direct launch, then (with graphs) the call that would record the shape
            c.set_option(D.OPT_TEST_FAIL_BESIDE, 1)
            with pytest.raises(D.DagcError) as e:
                c.compress(codes, depth)
            assert e.value.status == D.ERR_CUDA
            c.set_option(D.OPT_TEST_FAIL_BESIDE, 0)
            assert np.array_equal(c.compress(other, depth).to_numpy(), ref_other)
        for _ in range(3):
            assert np.array_equal(c.compress(codes, depth).to_numpy(), ref)
