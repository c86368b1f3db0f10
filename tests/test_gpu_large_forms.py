"""GPU tests of the routes that only large inputs take: crowded volumes past the
fragment limit of the direct marking (grouped or sorted, with the brick table's
compaction waiting for the device's choice), merges whose levels fall into two
groups, and levels with more distinct nodes than the hash set holds."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import random_codes
from tests.test_gpu_parity import assert_dag_equal

pytestmark = pytest.mark.gpu


def crowded(depth, n, seed):
    """n fragments of 3000 voxels on the device, each voxel present; and the voxels."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    voxels = np.unique(random_codes(depth, 3000, seed))
    v = torch.from_numpy(voxels.view(np.int64)).cuda()
    codes = v[torch.randint(0, v.numel(), (n,), device="cuda", generator=gen)]
    codes[torch.randperm(n, device="cuda", generator=gen)[: v.numel()]] = v
    return codes, voxels


@pytest.mark.parametrize("n", [2**25, 2**25 + 1])
@pytest.mark.parametrize("depth", [5, 8, 9])
def test_crowded_volumes_at_the_marking_limit(depth, n):
    """Marked straight into the table / grouped into it: one compaction form up to depth 8, the other beyond."""
    codes, voxels = crowded(depth, n, depth)
    ref = O.final_dag(O.create_dag(voxels, depth))
    small = random_codes(depth, 5000, 77)
    small_ref = O.final_dag(O.create_dag(small, depth))
    with D.Context(0) as c:
        for _ in range(3):  # launched, recorded, replayed
            assert np.array_equal(c.compress(codes, depth).to_numpy(), ref)
        keep = codes[n - 1].item()
        codes[n - 1] = 8**depth  # out of range
        with pytest.raises(D.DagcError) as e:
            c.compress(codes, depth)
        assert e.value.status == D.ERR_BAD_INPUT
        assert np.array_equal(c.compress(small, depth).to_numpy(), small_ref)  # the table is clean
        codes[n - 1] = keep
        assert np.array_equal(c.compress(codes, depth).to_numpy(), ref)
        assert c.dedup_fallbacks() == 0


def test_a_full_volume_past_the_limit_is_sorted():
    """1024^3 with four fragments in every brick: too many bricks to group, so the compaction returns at once."""
    import torch
    n = 4 * 8**8 + 1
    gen = torch.Generator(device="cuda").manual_seed(3)
    codes = (torch.arange(n, device="cuda") % 8**8) << 6 | torch.randint(0, 2, (n,), device="cuda", generator=gen)
    codes = codes[torch.randperm(n, device="cuda", generator=gen)]
    words = []
    for mode in (1, 0):
        with D.Context(0) as c:
            c.set_option(D.OPT_GROUP, mode)
            for _ in range(3 if mode else 1):
                words.append(c.compress(codes, 10).to_numpy())
            assert c.dedup_fallbacks() == 0
    for w in words[1:]:
        assert np.array_equal(words[0], w)


def test_a_merge_in_two_groups_of_levels():
    """8 inputs of 2M nodes in their last level: above the nodes of one group."""
    rng = np.random.default_rng(5)
    cells = rng.permutation(8**7)[:2_050_000].astype(np.uint64)
    codes = np.concatenate([(cells << np.uint64(9)) | rng.integers(0, 512, cells.size, dtype=np.uint64) for _ in range(4)])
    out = []
    for form in (1, 0):
        with D.Context(0) as c:
            c.set_option(D.OPT_DEDUP, form)
            dags = [c.create_dag(codes[i * 1000:], 10) for i in range(8)]
            sizes = [d.level_sizes() for d in dags]
            assert sum(s[-1] for s in sizes) < 2**24 < sum(sum(s) for s in sizes)
            out.append(c.merge_dags(dags).to_host())
            assert c.dedup_fallbacks() == 0
    assert_dag_equal(out[0], out[1])


def test_more_distinct_nodes_than_the_hash_set_holds():
    """Rerun by sorts, again and again in the same scratch."""
    codes = random_codes(17, 6_000_000, 6)
    with D.Context(0) as c:
        c.set_option(D.OPT_DEDUP, 0)
        ref = c.compress(codes, 17).to_numpy()
        c.set_option(D.OPT_DEDUP, 1)
        for k in range(3):
            assert np.array_equal(c.compress(codes, 17).to_numpy(), ref)
            assert c.dedup_fallbacks() == k + 1
