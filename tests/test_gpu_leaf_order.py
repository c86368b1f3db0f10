"""GPU tests of the distinct leaf masks' order at the edges of its forms: up to
8192 masks ranked at once, buckets between samples of them above (counted whole
up to 96 masks, in sub-buckets beyond), more samples and buckets above 2^18."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def codes_with_masks(masks, depth, seed):
    """Fragments whose bricks carry exactly these masks (shuffled)."""
    rng = np.random.default_rng(seed)
    bricks = rng.choice(8 ** (depth - 2), size=masks.size, replace=False).astype(np.uint64)
    codes = [(bricks[sel] << np.uint64(6)) | np.uint64(k)
             for k in range(64) for sel in [(masks >> np.uint64(k)) & np.uint64(1) == 1]]
    return rng.permutation(np.concatenate(codes))


def sparse_masks(count, seed):
    """Distinct masks of up to five bits anywhere."""
    rng = np.random.default_rng(seed)
    m = np.zeros(2 * count + 64, np.uint64)
    for _ in range(5):
        m |= np.uint64(1) << rng.integers(0, 64, m.size).astype(np.uint64)
    m = np.unique(m)
    assert m.size >= count
    return rng.choice(m, count, replace=False)


@pytest.mark.parametrize("kind,count", [("sparse", 2), ("sparse", 8191), ("sparse", 8192), ("sparse", 8193),
                                        ("skewed", 30_001), ("sparse", 2**18), ("sparse", 2**18 + 1),
                                        ("skewed", 300_007)])
def test_leaf_order_bit_exact(kind, count):
    if kind == "sparse":
        masks = sparse_masks(count, count)
    else:  # half of the masks within 2^18 of the lowest, the rest up to the highest value
        masks = np.concatenate([np.arange(1, count // 2 + 1, dtype=np.uint64),
                                np.uint64(2**64 - 1) - np.arange(count - count // 2, dtype=np.uint64) * np.uint64(2**41 + 1)])
    masks = np.concatenate([masks, masks[:777]])  # some bricks share a mask
    codes = codes_with_masks(masks, 9, count)
    ref = O.create_dag(codes, 9, threads=8)
    assert ref.leaves.size == count
    with D.Context(0) as c:
        for _ in range(3):  # direct launches, recording, replay
            assert_dag_equal(c.create_dag(codes, 9).to_host(), ref)
        assert c.dedup_fallbacks() == 0
