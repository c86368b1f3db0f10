"""GPU tests of the voxelizer's runs of triangles per warp, at the counts where
the runs grow (608 or 1216 tiles of four runs): a call equals the calls on
pieces small enough for one triangle a warp, one after another. Every seventh
triangle is long, so that some warps keep all their hits and some do not."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.test_gpu_voxelize_tiles import sat_reference, soup

pytestmark = pytest.mark.gpu
STEP = {D.VOXELIZE_GL: 608 * 4, D.VOXELIZE_SAT: 1216 * 4}


@pytest.mark.parametrize("mode", sorted(STEP))
@pytest.mark.parametrize("runs,more", [(2, -1), (2, 0), (4, -1), (4, 1), (8, 0), (16, -1), (16, 0), (16, 3), (37, 1)])
def test_runs_equal_pieces(ctx, mode, runs, more):
    n, depth = runs * STEP[mode] + more, 9
    tris = soup(n, depth, 2, runs + more)
    long = n // 97 * 7 if runs < 16 else 700
    tris[:long:7] = soup(len(tris[:long:7]), depth, 30, 1)
    box = (0, 0, 0) + (1 << depth,) * 3
    got = ctx.voxelize(tris, box, depth, mode).cpu().numpy().view(np.uint64)
    parts = [ctx.voxelize(tris[i:i + 2400], box, depth, mode).cpu().numpy().view(np.uint64) for i in range(0, n, 2400)]
    assert np.array_equal(got, np.concatenate(parts))
    last = tris[-40:]
    ref = O.voxelize_gl(last, box, depth) if mode == D.VOXELIZE_GL else sat_reference(last, box, depth)
    assert np.array_equal(got[-len(ref):], ref)
