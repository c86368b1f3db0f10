"""Performance cases of the compression framework: what its users have it do, over the range of sizes they do it at.

A case is a dict of plain values; `path` says which public entry points a pass goes through:

  compress    Context.compress: fragments on the device to the final words, in one call
  create      Context.create_dag, then create_final_dag (the reference's own two calls)
  merge       create_dag per subvolume, merge_dags over the 8, create_final_dag (the reference's subvolume loop)
  batched     create_dag_batched over many uneven chunks, then create_final_dag
  serve       Server: host fragments of several jobs in, each job's words out
  voxelize    Context.voxelize: triangles on the device to Morton fragments
  trace       dagc_trace: a frame of primary rays through a final DAG, into device buffers

Scenes are the repository's own workloads, drawn on the device from a seed: a sphere shell, fBm terrain (three voxels
per kept column) and a triangle soup (edges of 1 to 16 voxels, voxelized by the separating-axis rule), each as shuffled
Morton codes with duplicates, as the voxelization passes leave them.
"""
import math

import numpy as np
import torch

import dag_compression_fast_gb300 as D

DEVICE = "cuda"

# One context for the process, as a program keeps it: its scratch grows to the largest call.
_context = None


def context():
    global _context
    if _context is None:
        _context = D.Context(0)
    return _context


# ------------------------------------------------------------------------------------------------------------ cases --
def listed():
    return [
        # The smallest call: a shell of a few thousand fragments in a 32^3 grid (launches and latency alone).
        {"name": "shell_d5", "path": "compress", "scene": "sphere", "depth": 5},
        # The smallest benchmark configuration, through the reference's two calls: a shell in a 128^3 grid, ~100k fragments.
        {"name": "shell_d7", "path": "create", "scene": "sphere", "depth": 7},
        # A subvolume of ordinary size, a ragged share of the columns of a 512^2 terrain: ~0.7M fragments.
        {"name": "terrain_d9", "path": "compress", "scene": "terrain", "depth": 9, "fraction": 0.371},
        # A subvolume of scattered triangles, few fragments per brick: ~2.3M fragments.
        {"name": "soup_d10", "path": "compress", "scene": "soup", "depth": 10, "triangles": 70001},
        # The benchmark's second workload: terrain in a 2048^3 grid, 31.5M fragments.
        {"name": "terrain_d11", "path": "compress", "scene": "terrain", "depth": 11, "fraction": 1.0},
        # The benchmark's headline workload: 2M triangles in an 8192^3 grid, 65M fragments.
        {"name": "soup_d13", "path": "compress", "scene": "soup", "depth": 13, "triangles": 2000000},
        # The reference's subvolume loop: 8 subvolumes of 512^3, each compressed, then merged.
        {"name": "merge_8xd9", "path": "merge", "scene": "terrain", "depth": 9, "fraction": 0.5},
        # The batched workload: 256 uneven chunks of 1024^3 over one terrain, ~270M fragments.
        {"name": "batched_256xd10", "path": "batched", "depth": 10, "top": 4, "chunks": 256, "least": 10000, "most": 8000000},
        # A burst of requests on a running server: nine jobs of the three scenes on four slots, host to host.
        {"name": "serve_9", "path": "serve", "jobs": 9, "depth": 8, "least": 20000, "most": 1000000},
        # The reference's voxelization rule at the size of a loaded scene.
        {"name": "voxelize_gl", "path": "voxelize", "mode": "gl", "depth": 12, "triangles": 500000},
        # The separating-axis rule that feeds the soups.
        {"name": "voxelize_sat", "path": "voxelize", "mode": "sat", "depth": 11, "triangles": 60000},
        # A full-HD frame of the 2048^3 terrain: colours and hit voxels.
        {"name": "trace_1080p", "path": "trace", "scene": "terrain", "depth": 11, "fraction": 1.0, "width": 1920, "height": 1080},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["compress", "compress", "compress", "create", "merge", "batched", "serve", "voxelize", "trace"])
    if path == "batched":
        depth = rng.choice([6, 7, 8, 9, 10])
        most = _log(rng, 2000, min(3 * 4 ** depth, 4000000))
        return {"path": path, "depth": depth, "top": 4, "chunks": rng.randint(3, 200), "least": max(100, most // rng.randint(5, 500)),
                "most": most}
    if path == "serve":
        most = _log(rng, 100000, 2000000)
        return {"path": path, "jobs": rng.randint(2, 12), "depth": rng.choice([8, 9, 10]), "least": max(5000, most // 40), "most": most}
    if path == "voxelize":
        mode = rng.choice(["gl", "sat"])
        return {"path": path, "mode": mode, "depth": rng.randint(8, 13), "triangles": _log(rng, 1001, 800000 if mode == "gl" else 80000)}
    scene = rng.choice(["terrain", "soup"]) if path in ("merge", "trace") else rng.choice(["sphere", "terrain", "soup"])
    c = {"path": path, "scene": scene}
    if scene == "sphere":
        c["depth"] = rng.randint(5, 9)
        c["radius"] = round(rng.uniform(0.2, 0.44), 4)
    elif scene == "terrain":
        c["depth"] = rng.randint(7, 9) if path == "merge" else rng.randint(8, 11)
        c["fraction"] = round(math.exp(rng.uniform(math.log(0.05), 0.0)), 4)
    else:
        c["depth"] = rng.randint(8, 10) if path == "merge" else rng.randint(9, 14)
        c["triangles"] = _log(rng, 501, 100000 if path in ("merge", "trace") else 1900000)
    if path == "trace":
        c["width"], c["height"] = rng.randint(300, 2560), rng.randint(200, 1440)
    return c


# ----------------------------------------------------------------------------------------------------------- scenes --
def _spread(x):
    """Every bit of x (below 2^21) moved to three times its place."""
    x = x & 0x1FFFFF
    x = (x | x << 32) & 0x1F00000000FFFF
    x = (x | x << 16) & 0x1F0000FF0000FF
    x = (x | x << 8) & 0x100F00F00F00F00F
    x = (x | x << 4) & 0x10C30C30C30C30C3
    return (x | x << 2) & 0x1249249249249249


def _morton(x, y, z):
    return _spread(x) << 2 | _spread(y) << 1 | _spread(z)


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _shuffled(codes, g):
    return codes[torch.randperm(codes.numel(), device=DEVICE, generator=g)]


def _repeated(codes, g):
    """Each voxel once to four times, in random order."""
    times = torch.randint(1, 5, (codes.numel(),), device=DEVICE, generator=g)
    return _shuffled(torch.repeat_interleave(codes, times), g)


def _lattice(g):
    """Four octaves of random values for fBm over the unit square, base period a quarter."""
    return [torch.rand((4 * 2 ** o + 2, 4 * 2 ** o + 2), device=DEVICE, generator=g) for o in range(4)]


def _heights(lattice, u, v):
    """fBm in [0, 1) at the columns u by v (each in [0, 1))."""
    total, norm = 0.0, 0.0
    for o, table in enumerate(lattice):
        f = 4.0 * 2 ** o
        i, j = (u * f).long(), (v * f).long()
        s, t = u * f - i, v * f - j
        s, t = (s * s * (3 - 2 * s))[:, None], (t * t * (3 - 2 * t))[None, :]
        low, high = table[i], table[i + 1]
        row0, row1 = low[:, j], low[:, j + 1]
        row2, row3 = high[:, j], high[:, j + 1]
        total = total + (row0 * (1 - s) * (1 - t) + row1 * (1 - s) * t + row2 * s * (1 - t) + row3 * s * t) * 0.5 ** o
        norm += 0.5 ** o
    return total / norm


def _columns(heights, side, fraction, g):
    """The three voxels of a random share of the columns of a height field, y in [side / 4, 3 side / 4)."""
    n = heights.shape[0]
    kept = torch.rand(heights.shape, device=DEVICE, generator=g) < fraction
    x, z = kept.nonzero(as_tuple=True)
    y = (side // 4 + heights[x, z] * (side // 2)).long()
    return torch.cat([_morton(x % n, y - k, z % n) for k in range(3)])


def _terrain(depth, fraction, seed, lattice=None, at=(0, 0), of=1):
    """Terrain of a 2^depth grid: tile `at` of an `of` by `of` array of such grids over one height field."""
    g = _generator(seed)
    side = 1 << depth
    lattice = lattice or _lattice(g)
    steps = torch.arange(side, device=DEVICE, dtype=torch.float32) / side
    heights = _heights(lattice, (at[0] + steps) / of, (at[1] + steps) / of)
    return _repeated(_columns(heights, side, fraction, g), g)


def _sphere(depth, radius, seed):
    g = _generator(seed)
    side = 1 << depth
    centre = (side / 2 + torch.rand(3, device=DEVICE, generator=g) * 2 - 1).tolist()
    axis = torch.arange(side, device=DEVICE, dtype=torch.float32) + 0.5
    d2 = [(axis - c) ** 2 for c in centre]
    away = (d2[0][:, None, None] + d2[1][None, :, None] + d2[2][None, None, :]).sqrt_()
    x, y, z = ((away - radius * side).abs_() <= 0.5).nonzero(as_tuple=True)
    return _repeated(_morton(x, y, z), g)


def _triangles(depth, count, seed):
    """v0 uniform in the grid, two edges of log-uniform length in [1, 16] voxels and uniform direction; count x 9."""
    g = _generator(seed)
    v0 = torch.rand((count, 1, 3), device=DEVICE, generator=g, dtype=torch.float64) * (1 << depth)
    way = torch.randn((count, 2, 3), device=DEVICE, generator=g, dtype=torch.float64)
    length = 16.0 ** torch.rand((count, 2, 1), device=DEVICE, generator=g, dtype=torch.float64)
    edges = way / way.norm(dim=2, keepdim=True) * length
    return torch.cat([v0, v0 + edges], dim=1).reshape(count, 9).contiguous()


def _soup(depth, count, seed):
    box = (0, 0, 0) + (1 << depth,) * 3
    codes = context().voxelize(_triangles(depth, count, seed), box, depth, D.VOXELIZE_SAT, capacity=64 * count + 4096)
    return _shuffled(codes, _generator(seed + 1))


def _scene(case, seed):
    if case["scene"] == "sphere":
        return _sphere(case["depth"], case.get("radius", 0.4375), seed)
    if case["scene"] == "terrain":
        return _terrain(case["depth"], case["fraction"], seed)
    return _soup(case["depth"], case["triangles"], seed)


def _chunks(case, seed):
    """(codes, counts, Morton indices) of chunks with log-uniform fragment targets on a 16 by 16 footprint of one
    terrain, in ascending Morton order of the chunks; every eighth chunk keeps twice its target."""
    rng = np.random.default_rng(seed)
    lattice = _lattice(_generator(seed))
    cells = rng.permutation(256)[: case["chunks"]]
    x, z = torch.from_numpy(cells // 16), torch.from_numpy(cells % 16)
    morton, order = torch.sort(_morton(x, torch.full_like(x, 7), z))
    side = 1 << case["depth"]
    codes = []
    for i in order.tolist():
        target = math.exp(rng.uniform(math.log(case["least"]), math.log(case["most"])))
        fraction = min(1.0, target * (2.0 if i % 8 == 0 else 1.0) / (7.5 * side * side))
        codes.append(_terrain(case["depth"], fraction, int(rng.integers(1 << 40)), lattice, (int(x[i]), int(z[i])), 16))
    return torch.cat(codes), [c.numel() for c in codes], morton.numpy().astype(np.uint64)


def _jobs(case, seed):
    """(host fragments, depth) of a burst: the three scenes in turn, log-uniform sizes."""
    rng = np.random.default_rng(seed)
    jobs = []
    for k in range(case["jobs"]):
        target = math.exp(rng.uniform(math.log(case["least"]), math.log(case["most"])))
        s, side = int(rng.integers(1 << 40)), 1 << case["depth"]
        if k % 3 == 0:
            codes = _terrain(case["depth"], min(1.0, target / (7.5 * side * side)), s)
        elif k % 3 == 1:
            codes = _soup(case["depth"] + 2, max(1, int(target / 32)), s)
        else:
            codes = _sphere(case["depth"], min(0.44, math.sqrt(target / (2.5 * 4 * math.pi * 1.1)) / side), s)
        jobs.append((codes.cpu().pin_memory(), case["depth"] + (2 if k % 3 == 1 else 0)))
    return jobs


def _camera(depth, width, height):
    """From outside one corner of the unit box, looking across the volume."""
    position, target, up = np.array([0.1, 0.85, -0.4]), np.array([0.6, 0.4, 0.7]), np.array([0.0, 1.0, 0.0])
    forward = (target - position) / np.linalg.norm(target - position)
    right = np.cross(up, forward)
    right /= np.linalg.norm(right)
    return D.trace_camera(position, right, np.cross(forward, right), forward, 60.0, width, height, (0, 0, 0), (1, 1, 1), depth)


# ------------------------------------------------------------------------------------------------------------ a pass --
class _Device:
    """A word array of the library as torch sees it."""

    def __init__(self, words):
        self.words = words
        self.__cuda_array_interface__ = {"shape": (words.n,), "typestr": "<i4", "data": (words.ptr, False), "version": 3}


def _room(case):
    """Words (or codes) that a program holding this case's results keeps room for: above what any seed gives."""
    side = 1 << case["depth"]
    if case["path"] == "voxelize":
        return 64 * case["triangles"] + 65536
    if case["path"] == "batched":
        mean = (case["most"] - case["least"]) / math.log(case["most"] / case["least"])
        return int(min(3 * mean * case["chunks"], case["chunks"] * side * side)) + 65536
    if case["scene"] == "soup":
        return (8 if case["path"] == "merge" else 1) * 32 * case["triangles"] + 65536
    if case["scene"] == "sphere":
        return 8 * side * side + 65536
    return (8 if case["path"] == "merge" else 1) * int(4 * case["fraction"] * side * side) + 65536


def _keep(state, words):
    """The words into the program's own array (its end stays zero); their room goes back to the context."""
    state["out"][: words.n].copy_(torch.as_tensor(_Device(words), device=DEVICE))
    words.free()
    return state["out"]


def prepare(case, seed):
    ctx, path, depth = context(), case["path"], case["depth"]
    state = {"case": case}
    if path in ("compress", "create"):
        state["fragments"] = _scene(case, seed)
    elif path == "merge":
        state["fragments"] = [_scene(case, 8 * seed + k) for k in range(8)]
    elif path == "batched":
        state["fragments"], state["counts"], state["morton"] = _chunks(case, seed)
    elif path == "serve":
        state["server"] = D.Server(0, slots=4)
        state["jobs"] = _jobs(case, seed)
        state["out"] = [torch.zeros(4 * case["most"] + 65536, dtype=torch.int32, pin_memory=True) for _ in state["jobs"]]
    elif path == "voxelize":
        state["triangles"] = _triangles(depth, case["triangles"], seed)
        state["box"] = (0, 0, 0) + (1 << depth,) * 3
        state["out"] = torch.zeros(_room(case), dtype=torch.int64, device=DEVICE)
    else:
        state["words"] = ctx.compress(_scene(case, seed), depth)
        state["camera"] = _camera(depth, case["width"], case["height"])
        pixels = case["width"] * case["height"]
        state["colors"] = torch.zeros(pixels, dtype=torch.int32, device=DEVICE)
        state["hits"] = torch.zeros(pixels, dtype=torch.int64, device=DEVICE)
    if path in ("compress", "create", "merge", "batched"):
        state["out"] = torch.zeros(_room(case), dtype=torch.int32, device=DEVICE)
    return state


def run(state):
    ctx, case = context(), state["case"]
    path, depth = case["path"], case["depth"]
    if path == "compress":
        return _keep(state, ctx.compress(state["fragments"], depth))
    if path == "create":
        return _keep(state, ctx.create_final_dag(ctx.create_dag(state["fragments"], depth)))
    if path == "merge":
        dags = [ctx.create_dag(f, depth) for f in state["fragments"]]
        return _keep(state, ctx.create_final_dag(ctx.merge_dags(dags)))
    if path == "batched":
        dag = ctx.create_dag_batched(state["fragments"], state["counts"], state["morton"], depth, case["top"])
        return _keep(state, ctx.create_final_dag(dag))
    if path == "serve":
        server = state["server"]
        tickets = [server.submit_into(codes.numpy(), d, out.numpy().view(np.uint32))
                   for (codes, d), out in zip(state["jobs"], state["out"])]
        for t in tickets:
            server.wait(t)
        return state["out"]
    if path == "voxelize":
        mode = D.VOXELIZE_GL if case["mode"] == "gl" else D.VOXELIZE_SAT
        codes = ctx.voxelize(state["triangles"], state["box"], depth, mode)
        state["out"][: codes.numel()].copy_(codes)
        return state["out"]
    status = D.lib().dagc_trace(ctx.handle, state["words"].ptr, state["words"].n, depth, D.ctypes.byref(state["camera"]),
                                state["colors"].data_ptr(), state["hits"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if status:
        raise D.DagcError(status, "trace failed")
    return state["colors"], state["hits"]


def _bytes(v):
    return sum(_bytes(x) for x in v) if isinstance(v, (list, tuple)) else v.numel() * v.element_size()


def _used(v):
    """Bytes of an output up to its last nonzero value: the program's array is longer than the result."""
    if isinstance(v, (list, tuple)):
        return sum(_used(x) for x in v)
    return (int(v.nonzero()[-1]) + 1) * v.element_size()


def work(case):
    """Each input once and each output once, counted on one draw of the case's inputs."""
    state = prepare(case, 1)
    path = case["path"]
    if path == "voxelize":
        read = _bytes(state["triangles"])
    elif path == "trace":
        return {"bytes": 4 * state["words"].n + _bytes(run(state)), "flops": 0}
    elif path == "serve":
        read = _bytes([codes for codes, _ in state["jobs"]])
    else:
        read = _bytes(state["fragments"])
    return {"bytes": read + _used(run(state)), "flops": 0}


def exact(case, seed):
    """Every output is words, codes or colours: whole numbers, held equal as they are."""
    return None
