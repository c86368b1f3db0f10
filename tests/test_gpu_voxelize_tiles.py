"""GPU tests of the voxelizer's tiles, kept hits and float32 filter at their
edges: the separating-axis rule against a float64 numpy restatement (same
operations, same order), the reference (GL) rule against its oracle."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import morton

pytestmark = pytest.mark.gpu


def sat_reference(tris, box, depth):
    """Codes of every voxel each triangle touches, triangles in order, each
    one's voxels with z fastest."""
    G = 1 << depth
    box = np.asarray(box, np.float64)
    out = []
    for t in np.asarray(tris, np.float64).reshape(-1, 3, 3):
        v = (t - box[:3]) * (G / (box[3:] - box[:3]))
        lo = np.floor(np.clip(v.min(0), -1, G)).astype(int).clip(0)
        hi = np.minimum(np.floor(np.clip(v.max(0), -1, G)).astype(int), G - 1)
        if (hi < lo).any():
            continue
        x, y, z = (a.ravel() for a in np.meshgrid(*[np.arange(l, h + 1) for l, h in zip(lo, hi)], indexing="ij"))
        c = np.stack([x, y, z], 1) + 0.5
        w = [v[k] - c for k in range(3)]
        e = [w[1] - w[0], w[2] - w[1], w[0] - w[2]]
        hit = np.ones(x.size, bool)
        for i in range(3):
            a, b = (i + 1) % 3, (i + 2) % 3
            for j in range(3):
                p = [(-e[j][:, b]) * w[k][:, a] + e[j][:, a] * w[k][:, b] if i != 1 else
                     e[j][:, a] * w[k][:, b] + (-e[j][:, b]) * w[k][:, a] for k in range(3)]
                mn, mx = np.minimum(p[0], np.minimum(p[1], p[2])), np.maximum(p[0], np.maximum(p[1], p[2]))
                r = 0.5 * (np.abs(e[j][:, a]) + np.abs(e[j][:, b]))
                hit &= ~((mn > r) | (mx < -r))
        n = np.stack([e[0][:, 1] * e[1][:, 2] - e[0][:, 2] * e[1][:, 1], e[0][:, 2] * e[1][:, 0] - e[0][:, 0] * e[1][:, 2],
                      e[0][:, 0] * e[1][:, 1] - e[0][:, 1] * e[1][:, 0]], 1)
        dist = n[:, 0] * w[0][:, 0] + n[:, 1] * w[0][:, 1] + n[:, 2] * w[0][:, 2]
        hit &= np.abs(dist) <= 0.5 * (np.abs(n[:, 0]) + np.abs(n[:, 1]) + np.abs(n[:, 2]))
        out.append(morton(x[hit].astype(np.uint64), y[hit].astype(np.uint64), z[hit].astype(np.uint64)))
    return np.concatenate(out) if out else np.zeros(0, np.uint64)


def soup(n, depth, size, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 1 << depth, (n, 1, 3))
    return np.concatenate([a, a + rng.normal(0, size, (n, 2, 3))], 1)


def lattice(n, depth, seed):
    """Vertices on whole and half coordinates: triangles that just touch voxels."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 2 << depth, (n, 1, 3)) / 2
    t = a + np.concatenate([np.zeros((n, 1, 3)), rng.integers(-6, 7, (n, 2, 3)) / 2], 1)
    t[::3, :, 1] = np.floor(t[::3, :1, 1])  # a third in planes between voxels
    t[::10, 2] = t[::10, 1]                 # some of no area
    return t


CASES = {
    "one": lambda: (soup(1, 6, 3, 1), 6), "tile_less": lambda: (soup(63, 6, 3, 2), 6), "tile": lambda: (soup(64, 6, 3, 3), 6),
    "tile_more": lambda: (soup(65, 6, 3, 4), 6), "small": lambda: (soup(1500, 9, 0.3, 5), 9),
    "more_than_kept": lambda: (soup(40, 7, 25, 6), 7),  # a triangle's hits pass its warp's list
    "lattice": lambda: (lattice(1500, 6, 7), 6),
    "long": lambda: (np.array([[[3.2, 5, 5], [1900.7, 5.9, 6.1], [900.5, 6.5, 5.2]]]), 11),  # extents above 1024
    "outside": lambda: (soup(200, 6, 40, 8) * 1.6 - 20, 6),
    "far_outside": lambda: (np.array([[[1, 1, 1], [3e5, 2, 2], [5, 30, 3]], [[4, 4, 4], [5, 5, 6], [6, 4, 4]]]), 5),
    "cross_box": lambda: (np.array([[[-1e9, 3, 3], [1e9, 4, 4], [0, 20, 5]]]), 5),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_sat_rule_in_order(ctx, case):
    tris, depth = CASES[case]()
    box = (0, 0, 0) + (1 << depth,) * 3
    got = ctx.voxelize(tris, box, depth, D.VOXELIZE_SAT).cpu().numpy().view(np.uint64)
    assert np.array_equal(got, sat_reference(tris, box, depth))


@pytest.mark.parametrize("case", ["one", "tile_less", "tile_more", "more_than_kept", "outside", "long"])
def test_gl_rule_in_order(ctx, case):
    tris, depth = CASES[case]()
    box = (0, 0, 0) + (1 << depth,) * 3
    got = ctx.voxelize(tris, box, depth, D.VOXELIZE_GL).cpu().numpy().view(np.uint64)
    assert np.array_equal(got, O.voxelize_gl(tris, box, depth))


def test_sat_rule_scene_units_and_not_a_number(ctx):
    box = (-1.5, 0.25, 3.0, 2.5, 4.75, 7.0)
    rng = np.random.default_rng(9)
    tris = np.array(box[:3]) + rng.uniform(0, 4, (300, 1, 3)) + rng.normal(0, 0.1, (300, 3, 3))
    ref = sat_reference(tris, box, 8)
    bad = np.concatenate([tris[:100], np.full((2, 3, 3), np.nan), tris[100:]])
    assert np.array_equal(ctx.voxelize(tris, box, 8, D.VOXELIZE_SAT).cpu().numpy().view(np.uint64), ref)
    assert np.array_equal(ctx.voxelize(bad, box, 8, D.VOXELIZE_SAT).cpu().numpy().view(np.uint64), ref)


@pytest.mark.parametrize("mode", [D.VOXELIZE_GL, D.VOXELIZE_SAT])
def test_room_for_some_of_the_codes(ctx, mode):
    """Too little room: the count is whole, the room holds the first codes."""
    import ctypes

    import torch
    tris = soup(500, 7, 3, 10)
    box = np.array((0, 0, 0) + (128,) * 3, np.float64)
    full = ctx.voxelize(tris, box, 7, mode)
    v = torch.from_numpy(tris).cuda().contiguous()
    for room in (1, 77, full.numel() - 1):
        out = torch.zeros(full.numel() + 8, dtype=torch.int64, device="cuda")
        n = ctypes.c_uint64(0)
        st = D.lib().dagc_voxelize(ctx.handle, v.data_ptr(), 500, box.ctypes.data, 7, mode, out.data_ptr(), room,
                                   ctypes.byref(n), torch.cuda.current_stream().cuda_stream)
        assert st == D.ERR_TOO_LARGE and n.value == full.numel()
        assert torch.equal(out[:room], full[:room]) and not out[room:].any()
