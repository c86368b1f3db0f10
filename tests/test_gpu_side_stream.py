"""GPU tests of the node extraction that runs beside a call's stream: a call
that fails while it is queued waits for it, directly launched or while its
shape is recorded, and the calls after it (which write the same scratch) are
bit-exact."""
import ctypes

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


def _cudart():
    for name in ("libcudart.so.13", "libcudart.so", "/usr/local/cuda/lib64/libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            continue
    pytest.skip("no CUDA runtime library to record a stream with")


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("used", [False, True])
def test_a_call_on_a_recording_stream_is_refused_alone(graphs, used):
    """A call cannot be recorded by its caller; while the recording is open, the context's calls on other streams go
    through, and afterwards all do (a first call refused so leaves no table uncleared)."""
    import torch
    rt = _cudart()
    a, b = random_codes(9, 200_000, 31), random_codes(9, 150_000, 32)
    ref_a, ref_b = O.final_dag(O.create_dag(a, 9)), O.final_dag(O.create_dag(b, 9))
    a, b = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with D.Context(0) as c:
        c.set_option(D.OPT_GRAPHS, graphs)
        if used:
            for _ in range(2):
                assert np.array_equal(c.compress(a, 9).to_numpy(), ref_a)
        torch.cuda.synchronize()
        assert rt.cudaStreamBeginCapture(ctypes.c_void_p(s.cuda_stream), 2) == 0  # relaxed
        try:
            with pytest.raises(D.DagcError):
                c.compress(a, 9, stream=s)
            w = c.compress(b, 9, stream=other)
        finally:
            graph = ctypes.c_void_p()
            rt.cudaStreamEndCapture(ctypes.c_void_p(s.cuda_stream), ctypes.byref(graph))
            rt.cudaGetLastError()
        assert np.array_equal(w.to_numpy(), ref_b)
        for _ in range(3):
            assert np.array_equal(c.compress(a, 9).to_numpy(), ref_a)
            assert np.array_equal(c.compress(b, 9, stream=s).to_numpy(), ref_b)
