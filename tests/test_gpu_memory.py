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
