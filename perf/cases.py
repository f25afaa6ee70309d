"""Workloads of the DAG build as its users call it, for timing and for comparing two versions.

listed() gives the fixed cases, draw() more of the same ranges, prepare() what a caller
holds before the call (device inputs, descriptors, pools), run() one pass through the
public entry points and its whole outputs, work() the bytes a pass cannot do without and
exact() the floating outputs (the boxes of the RT prims) in 64 bits from plain torch.

Contents: terrain (a heightfield, the shape of generated chunks), thresholded value noise
(~30 % solid, materials in 8^3 blocks), Bernoulli cells (no structural sharing) and thin
skins (one surface layer). PyrVoxel lists are in raster order, as a generator or a dense
grid gives them, unless a case says that they are shuffled.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from pyrit_b200 import gpu_build, native
from pyrit_b200 import workloads as wl

NONE = 0xFFFFFFFF
EXACT_MOST = 400_000_000  # entries that exact() still orders in the time it has


def listed():
    return [
        # a 64^3 terrain chunk rebuilt inside a frame loop that cannot allocate: the smallest call
        {"name": "frame_terrain_64", "kind": "volume", "form": "noalloc", "fill": "terrain", "log2": 6, "edits": 0,
         "rt": 4, "shuffled": False},
        # pyr_geometry_build of a 128^3 scene of ~310 k voxels from host memory, upload included
        {"name": "host_scene_128", "kind": "volume", "form": "host", "fill": "skin", "log2": 7, "edits": 0, "rt": 5,
         "shuffled": False},
        # plain build of a 256^3 noise volume with a 0.5 % set/remove overlay: the headline
        {"name": "noise_256", "kind": "volume", "form": "build", "fill": "noise", "log2": 8, "edits": 83886, "rt": 7,
         "shuffled": False},
        # worst case for deduplication: 1024^3, i.i.d. 15 % cells, a million edits
        {"name": "bernoulli_1024", "kind": "volume", "form": "build", "fill": "bernoulli", "log2": 10,
         "edits": 1000000, "rt": 7, "shuffled": False, "p": 0.15},
        # a scanned landscape: one surface layer in a 4096^3 volume (64-bit sort keys)
        {"name": "surface_4096", "kind": "surface", "log2": 12, "nx": 3001, "nz": 2477, "rt": 7},
        # pyr_geometry_edit: 90 000 entries over the sorted voxels of a 256^3 geometry
        {"name": "edit_90k_256", "kind": "rebuild", "log2": 8, "edits": 90000, "rt": 7},
        # world streaming: 1063 chunks of 32^3, skins only, with the edit overlay merged
        {"name": "world_1063", "kind": "world", "log2": 5, "chunks": 1063, "capacity": 4096, "edits": 9, "rt": 5},
        # batched build of 1024 chunks of edges 32..256 (p .4/.3/.2/.1): the batched form
        {"name": "batch_1024", "kind": "batch", "chunks": 1024, "first": 0, "edits": 0, "rt": 5},
        # one batch of the served loop: a few requests on a resident pool with player edits
        {"name": "served_5", "kind": "batch", "chunks": 5, "first": 11, "edits": 40, "rt": 5},
        # LOD: a 256^3 geometry to 128^3
        {"name": "lod_256", "kind": "downsample", "log2": 8, "shift": 1, "rt": 6},
        # chunk install after a batched build: palettes found and attributes packed
        {"name": "install_256", "kind": "install", "chunks": 256, "first": 0},
        # player edits on installed chunks without a rebuild
        {"name": "path_edit_256", "kind": "path_edit", "chunks": 256, "first": 0, "edits": 32, "rt": 5},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["volume", "volume", "volume", "surface", "rebuild", "world", "batch", "batch", "downsample",
                       "install", "path_edit"])
    if kind == "volume":
        form = rng.choice(["build", "build", "host", "noalloc"])
        fill = rng.choice(["terrain", "noise", "bernoulli", "skin"])
        log2 = {"build": rng.randint(5, 9), "host": rng.randint(4, 8), "noalloc": rng.randint(4, 6)}[form]
        case = {"kind": kind, "form": form, "fill": fill, "log2": log2, "rt": rng.randint(3, log2),
                "edits": rng.choice([0, logint(1, max(2, 1 << (3 * log2 - 6)))]), "shuffled": rng.random() < 0.25}
        if fill == "bernoulli":
            case["p"] = round(math.exp(rng.uniform(math.log(0.01), math.log(0.5))), 4)
        return case
    if kind == "surface":
        log2 = rng.randint(11, 13)
        return {"kind": kind, "log2": log2, "nx": logint(100, 3000), "nz": logint(100, 3000),
                "rt": rng.randint(4, 8)}
    if kind == "rebuild":
        log2 = rng.randint(5, 9)
        return {"kind": kind, "log2": log2, "edits": logint(1, 200000), "rt": rng.randint(3, log2)}
    if kind == "world":
        log2 = rng.randint(4, 6)
        return {"kind": kind, "log2": log2, "chunks": logint(3, 3000 >> (log2 - 4)),
                "capacity": rng.randint(3, 5) << (2 * log2), "edits": rng.choice([0, logint(1, 64)]),
                "rt": rng.randint(3, log2)}
    if kind == "batch":
        return {"kind": kind, "chunks": logint(1, 600), "first": rng.randint(0, 400),
                "edits": rng.choice([0, logint(1, 64)]), "rt": rng.randint(3, 5)}
    if kind == "downsample":
        log2 = rng.randint(6, 9)
        return {"kind": kind, "log2": log2, "shift": rng.randint(1, 3), "rt": rng.randint(3, 7)}
    if kind == "install":
        return {"kind": kind, "chunks": logint(2, 400), "first": rng.randint(0, 400)}
    return {"kind": kind, "chunks": logint(1, 300), "first": rng.randint(0, 400), "edits": logint(1, 200),
            "rt": rng.randint(3, 5)}


# ---------------------------------------------------------------------------
# inputs
#
# A case's geometry is fixed up to a mirroring or swap of its axes (chunk batches: up to
# the order of the chunks), which the seed picks with the materials: the positions, keys,
# node order and attributes change with the seed, the sizes of the outputs do not.
# ---------------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _mirror(seed, axes="xyz"):
    """(flip x, flip y, flip z, swap x and z) of a seed."""
    bits = np.random.default_rng([int(seed), 11]).integers(0, 2, 4)
    return tuple(bool(bits[k]) and name in axes for k, name in enumerate("xyz")) + (bool(bits[3]) and "s" in axes,)


def _mirror_points(pts, mirror, n):
    """Coordinates of pts[:, :3] inside an n^3 cube, mirrored in place."""
    if mirror[3]:
        pts[:, [0, 2]] = pts[:, [2, 0]]
    for k in range(3):
        if mirror[k]:
            pts[:, k] = n - 1 - pts[:, k]
    return pts


def _mirror_cells(cells, mirror):
    """The same for cells[..., z, y, x]."""
    if mirror[3]:
        cells = cells.transpose(-1, -3)
    dims = [d for d, on in ((-1, mirror[0]), (-2, mirror[1]), (-3, mirror[2])) if on]
    return cells.flip(dims) if dims else cells


def _fbm(shape, period, octaves, g):
    """Multi-octave value noise in [0, 1) on the device (gain 0.5, lacunarity 2)."""
    mode = "bilinear" if len(shape) == 2 else "trilinear"
    total, weight, amp = torch.zeros(shape, device="cuda"), 0.0, 1.0
    for k in range(octaves):
        cells = [max(2, int(n * (1 << k) / period) + 2) for n in shape]
        lattice = torch.rand(cells, generator=g, device="cuda")
        total += amp * F.interpolate(lattice[None, None], size=tuple(shape), mode=mode, align_corners=True)[0, 0]
        weight += amp
        amp *= 0.5
    return total / weight


def _points(mask, attr, z0=0):
    """PyrVoxel list (int32 [n, 4]) of the set cells of mask[z, y, x], in raster order."""
    idx = mask.reshape(-1).nonzero().reshape(-1)
    ny, nx = mask.shape[1], mask.shape[2]
    out = torch.empty((idx.numel(), 4), dtype=torch.int32, device="cuda")
    out[:, 0] = idx % nx
    out[:, 1] = (idx // nx) % ny
    out[:, 2] = idx // (nx * ny) + z0
    out[:, 3] = attr(idx)
    return out


def _heights(n, m, g, edge):
    """Terrain height of every column [z, x]: half the edge, 0.19 edge of relief."""
    return edge / 2 + 0.38 * edge * (_fbm((m, n), max(edge / 2, 4), 4, g) - 0.5)


def _volume(fill, log2, seed, p=0.15):
    n = 1 << log2
    if fill == "bernoulli":
        mirror, step = _mirror(seed), max(1, (1 << 27) // (n * n))
        parts, slabs = [], list(range(0, n, step))
        for k, z0 in enumerate(slabs):
            at = slabs[-1 - k] if mirror[2] else z0      # the slab that ends up at z0
            mask = torch.rand((min(step, n), n, n), generator=_gen(at, 17 * log2), device="cuda") < p
            parts.append(_points(_mirror_cells(mask, mirror),
                                 lambda i, z0=z0: torch.randint(1, 256, (len(i),), generator=_gen(seed, z0),
                                                                device="cuda", dtype=torch.int32), z0))
        return torch.cat(parts)
    g = _gen(1, 17 * log2)
    if fill == "noise":
        mirror = _mirror(seed, "xyzs")
        field = _fbm((n, n, n), min(64, n), 3, g)
        sample = field.reshape(-1)[:: max(1, (n * n * n) // (1 << 20))]
        mask = field > sample.kthvalue(max(1, int(0.7 * sample.numel()))).values
        b = max(n // 8, 1)
        block = torch.randint(1, 9, (b * b * b,), generator=_gen(seed, 23), device="cuda", dtype=torch.int32)
        return _points(_mirror_cells(mask, mirror).contiguous(),
                       lambda i: block[(i // (n * n) * b // n * b + i // n % n * b // n) * b + i % n * b // n])
    mirror = _mirror(seed, "xzs")
    h = _heights(n, n, g, n).floor().clamp(1, n).to(torch.int64)
    depth = h[:, None, :] - torch.arange(n, device="cuda")[None, :, None]      # 1: the top layer
    depth = _mirror_cells(depth, mirror).contiguous()
    mask = depth >= 1
    if fill == "skin":
        mask = mask & (depth <= max(n // 7, 1))     # a scene of shells: what a mesh voxeliser gives
    depth = depth.reshape(-1)
    base = 1 + int(seed) % 5
    return _points(mask, lambda i: (base + (depth[i] > 1).int() + (depth[i] > 4).int()).to(torch.int32))


def _edits(log2, count, seed, mirror):
    """Random set/remove entries (half and half, materials 1..8) in any order."""
    g = _gen(2, 91 + log2)
    e = torch.randint(0, 1 << log2, (count, 4), generator=g, device="cuda", dtype=torch.int32)
    remove = torch.rand(count, generator=g, device="cuda") < 0.5
    m = torch.randint(1, 9, (count,), generator=_gen(seed, 91), device="cuda", dtype=torch.int32)
    e[:, 3] = torch.where(remove, 0, m)
    return _mirror_points(e, mirror, 1 << log2)


def _surface(case, seed):
    """One layer of terrain over nx x nz columns of a 2^log2 volume."""
    nx, nz, n = case["nx"], case["nz"], 1 << case["log2"]
    mirror = _mirror(seed, "xz")
    h = _heights(nx, nz, _gen(3, 5), 1 << 10).floor().to(torch.int32)
    h = h.flip([d for d, on in ((1, mirror[0]), (0, mirror[2])) if on]).reshape(-1)
    i = torch.arange(nx * nz, device="cuda", dtype=torch.int32)
    out = torch.empty((nx * nz, 4), dtype=torch.int32, device="cuda")
    out[:, 0] = i % nx + (n - nx if mirror[0] else 0)
    out[:, 1] = h
    out[:, 2] = i // nx + (n - nz if mirror[2] else 0)
    out[:, 3] = 1 + ((h + int(seed)) & 7)
    return out


def _axes(fill):
    return {"bernoulli": "xyz", "noise": "xyzs"}.get(fill, "xzs")


def _input(case, seed):
    """The PyrVoxel list of a volume or surface case."""
    if case["kind"] == "surface":
        return _surface(case, seed)
    v = _volume(case["fill"], case["log2"], seed, case.get("p", 0.15))
    if case["edits"]:
        v = torch.cat([v, _edits(case["log2"], case["edits"], seed, _mirror(seed, _axes(case["fill"])))])
    if case["shuffled"]:
        # the edits stay behind the voxels they change
        order = torch.randperm(len(v) - case["edits"], generator=_gen(seed, 3), device="cuda")
        v[:len(order)] = v[order]
    return v.contiguous()


def _spread3(v):
    for shift, mask in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F),
                        (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        v = (v | (v << shift)) & mask
    return v


def _morton(x, y, z):
    return _spread3(x) | (_spread3(y) << 1) | (_spread3(z) << 2)


def _sorted_voxels(log2, seed):
    """Sorted unique keys (brick Morton << 6 | cell in the brick) and attributes of a noise
    volume: what an editable geometry keeps of its last build; and its voxels."""
    v = _volume("noise", log2, seed)
    x, y, z = (v[:, k].long() for k in range(3))
    keys = (_morton(x >> 2, y >> 2, z >> 2) << 6) | (x & 3) | ((y & 3) << 2) | ((z & 3) << 4)
    keys, order = keys.sort()
    return keys, v[order, 3].contiguous(), v


def _roll(seed, count):
    """Order of the chunks of a batch: the seed's rotation."""
    return np.roll(np.arange(count), int(np.random.default_rng([int(seed), 13]).integers(0, count)))


def _world(case, seed):
    """Generated skins of neighbouring chunks: the voxels within one of a terrain surface
    that runs through the chunks, `capacity` slots per chunk, and each chunk's edits."""
    n, K, cap = 1 << case["log2"], case["chunks"], case["capacity"]
    mirror, g = _mirror(seed, "xyzs"), _gen(4, 7)
    h = torch.rand((K, 1, 5, 5), generator=g, device="cuda") * n
    h = F.interpolate(h, size=(n, n), mode="bilinear", align_corners=True)[:, 0].floor()      # [K, z, x]
    y = torch.arange(n, device="cuda")[None, None, :, None]
    mask = (y - h[:, :, None, :]).abs() <= 1                                                   # [K, z, y, x]
    roll = torch.from_numpy(_roll(seed, K)).cuda()
    mask = _mirror_cells(mask, mirror).reshape(K, -1)[roll]
    counts = mask.sum(1)
    rank = mask.cumsum(1) - 1
    c, i = mask.nonzero(as_tuple=True)
    vox = torch.zeros((K, cap, 4), dtype=torch.int32, device="cuda")
    pts = torch.stack([i % n, (i // n) % n, i // (n * n), 1 + ((i // n) + int(seed)) % 5], 1).to(torch.int32)
    vox[c, rank[mask]] = pts
    e_max = case["edits"]
    per = torch.randint(0, e_max + 1, (K,), generator=g, device="cuda") if e_max else counts * 0
    every = _edits(case["log2"], max(K * e_max, 1), seed, mirror)[:K * e_max].reshape(K, e_max, 4)
    held = torch.arange(e_max, device="cuda")[None, :] < per[:, None]
    eofs = F.pad(per[roll].cumsum(0), (1, 0)).to(torch.int32)
    edits = every[roll][held[roll]].contiguous()
    return vox, counts.to(torch.int32), edits, eofs, len(edits)


def _edges(case):
    return np.ascontiguousarray(wl.chunk_mix(case["first"] + case["chunks"], 0)[case["first"]:])


def _mix(case, seed):
    """Chunks of the mix (terrain tiled per chunk, spherical caves carved) in a resident
    pool on the device: (order of the chunks in the batch, their edges, pool, first voxel
    and size of each)."""
    log2s = _edges(case)
    vox, offs = wl.mix_chunks_device(log2s, case["first"], 0)
    vox[:, 3] += int(seed) % 7
    order = _roll(seed, len(log2s))
    return order, np.ascontiguousarray(log2s[order]), vox, offs[:-1][order], np.diff(offs)[order]


def _mix_edits(case, order, log2s, seed, exactly=False):
    """Up to (or exactly) `edits` player edits per chunk: (edits uint32 [n, 4], offsets
    int64 [K + 1]), chunk order[k] holding the k-th run."""
    per, pts = [], []
    material = np.random.default_rng([int(seed), 29])
    for c, l in zip(order, log2s):
        rng = np.random.default_rng([int(c), 31])
        n = case["edits"] if exactly or not case["edits"] else int(rng.integers(0, case["edits"] + 1))
        e = np.empty((n, 4), np.uint32)
        e[:, :3] = rng.integers(0, 1 << int(l), (n, 3))
        e[:, 3] = np.where(rng.random(n) < 0.5, 0, material.integers(1, 9, n))
        per.append(n)
        pts.append(e)
    return np.concatenate(pts), np.concatenate([[0], np.cumsum(per)]).astype(np.int64)


# ---------------------------------------------------------------------------
# outputs
# ---------------------------------------------------------------------------
class _Buffer:
    """Device memory of a finished build as torch sees it; keeps the build alive."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}


def _tensor(owner, ptr, shape, kind, dtype):
    if shape[0] == 0:
        return torch.empty(shape, dtype=dtype, device="cuda")
    return torch.as_tensor(_Buffer(owner, ptr, shape, kind), device="cuda")


def _outputs(b):
    """Everything a build returns."""
    out = {"nodes": _tensor(b, b.nodes, (b.node_words,), "<i4", torch.int32),
           "leaves": _tensor(b, b.leaves, (b.leaf_count,), "<i8", torch.int64),
           "keys": _tensor(b, b.keys, (b.voxel_count,), "<i8", torch.int64),
           "attrs": _tensor(b, b.attrs, (b.voxel_count,), "<i4", torch.int32),
           "prims": _tensor(b, b.prims, (b.prim_count, 4), "<i4", torch.int32),
           "aabbs": _tensor(b, b.aabbs, (b.prim_count, 6), "<f4", torch.float32),
           "root": int(b.root)}
    if b.roots is not None:
        out.update(roots=b.roots, first_voxel=b.first_voxel, first_prim=b.first_prim)
    return out


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _noalloc_state(case, v):
    """Output buffers at the upper bounds the fixed-array build asks for."""
    log2, n = case["log2"], max(len(v), 1)
    bricks = max(min(n, 8 ** (log2 - 2)), 1)
    words, prev, parents = 2, bricks, {}
    for lv in range(2, log2):
        prev = parents[lv] = max(min(prev, 8 ** (log2 - lv - 1)), 1)
        words += 10 * prev
    prims = max(parents[min(max(case["rt"], 3), log2) - 1], 1)
    new = lambda shape, dtype: torch.empty(shape, dtype=dtype, device="cuda")  # noqa: E731
    return {"voxels": v, "nodes": new(words, torch.int32), "leaves": new(bricks, torch.int64),
            "keys": new(n, torch.int64), "attrs": new(n, torch.int32), "prims": new((prims, 4), torch.int32),
            "aabbs": new((prims, 6), torch.float32)}


def _batch_state(case, seed):
    """A batch over chunks of a resident pool: descriptor, device offsets, host results."""
    order, log2s, vox, starts, sizes = _mix(case, seed)
    edits, eoffs = _mix_edits(case, order, log2s, seed)
    K, n_edits = len(log2s), int(eoffs[-1])
    offs = np.concatenate([[0], np.cumsum(sizes)])
    dev = {"log2": torch.from_numpy(log2s.view(np.int32)).cuda(),
           "offs": torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda(),
           "starts": torch.from_numpy(np.ascontiguousarray(starts, dtype=np.int64)).cuda(),
           "edits": torch.from_numpy(edits.view(np.int32)).cuda(),
           "eoffs": torch.from_numpy(eoffs.astype(np.uint32).view(np.int32)).cuda()}
    desc = native.Batch(count=K, log2_host=log2s.ctypes.data, log2=dev["log2"].data_ptr(),
                        voxels=vox.data_ptr() if int(offs[-1]) else 0, voxel_offsets=dev["offs"].data_ptr(),
                        edits=dev["edits"].data_ptr() if n_edits else 0,
                        edit_offsets=dev["eoffs"].data_ptr() if n_edits else 0, voxel_total=int(offs[-1]),
                        edit_total=n_edits, voxel_starts=dev["starts"].data_ptr())
    return {"desc": desc, "order": order, "log2s": log2s, "voxels": vox, "dev": dev, "K": K}


def _run_batch(s, rt):
    roots, first, prim = (np.empty(s["K"], np.uint32) for _ in range(3))
    ex, out = native.Exec(), native.BuiltC()
    ex.stream = ctypes.c_void_p(_stream())
    native.check(native.lib().pyrb_build_batch(ctypes.byref(ex), ctypes.byref(s["desc"]), rt, roots.ctypes.data,
                                               first.ctypes.data, prim.ctypes.data, ctypes.byref(out)))
    b = gpu_build.Built(out, _stream())
    b.roots, b.first_voxel, b.first_prim = roots, first, prim
    return b


def _install_state(case, seed):
    """Attributes of a finished batch and its chunks' first voxels. Every fifth chunk gets
    more materials than a palette holds, so that both installed formats occur."""
    s = _batch_state(dict(case, edits=0), seed)
    b = _run_batch(s, 3)
    o = _outputs(b)
    held = o["roots"] != NONE
    bounds = np.concatenate([o["first_voxel"][held], [b.voxel_count]]).astype(np.uint32)
    attrs = o["attrs"].clone()
    for k in np.nonzero(s["order"][held] % 5 == 0)[0]:
        part = attrs[int(bounds[k]):int(bounds[k + 1])]
        part += torch.arange(len(part), device="cuda", dtype=torch.int32) // 64 % 40 * 16
    words = int((16 + np.diff(bounds.astype(np.int64))).sum())
    return {"attrs": attrs, "first": bounds, "pool": torch.zeros(words, dtype=torch.int32, device="cuda")}


def _path_edit_state(case, seed):
    """Pools of a finished batch with an arena and attribute targets above it, one job per
    chunk, its prims and boxes (restored before every pass: a pass starts from the build)."""
    s = _batch_state(dict(case, edits=0), seed)
    b = _run_batch(s, case["rt"])
    o = _outputs(b)
    nz = np.nonzero(o["roots"] != NONE)[0]
    per, log2s = case["edits"], s["log2s"].astype(np.int64)[nz]
    first, fprim = o["first_voxel"][nz].astype(np.int64), o["first_prim"][nz].astype(np.int64)
    counts = np.diff(np.concatenate([first, [b.voxel_count]]))
    pcounts = np.diff(np.concatenate([fprim, [b.prim_count]]))
    caps = per * ((log2s - 2) * 10 + 4) + 8
    npos = b.node_words + np.concatenate([[0], np.cumsum(caps)])
    apos = b.voxel_count + np.concatenate([[0], np.cumsum(counts + per)])
    zeros = lambda n, dtype: torch.zeros(int(n), dtype=dtype, device="cuda")  # noqa: E731
    st = {"nodes": torch.cat([o["nodes"], zeros(caps.sum(), torch.int32)]),
          "leaves": torch.cat([o["leaves"], zeros(per * len(nz), torch.int64)]),
          "attrs": torch.cat([o["attrs"], zeros((counts + per).sum(), torch.int32)]),
          "prims0": o["prims"].clone(), "aabbs0": o["aabbs"].clone(), "out": int(b.voxel_count)}
    st["prims"], st["aabbs"] = st["prims0"].clone(), st["aabbs0"].clone()
    st["edits"], _ = _mix_edits(case, s["order"][nz], s["log2s"][nz], seed, exactly=True)
    jobs = (native.PathEditJob * len(nz))()
    for k in range(len(nz)):
        jobs[k] = native.PathEditJob(
            root=int(o["roots"][nz[k]]), log2_size=int(log2s[k]), attr_src=int(first[k]), attr_count=int(counts[k]),
            attr_a=int(apos[k]), attr_cap=int(counts[k]) + per, node_arena=int(npos[k]), node_cap=int(caps[k]),
            leaf_arena=int(b.leaf_count) + per * k, leaf_cap=per, edit_first=per * k, edit_count=per,
            rt_log2=int(b.rt_log2), prims=st["prims"].data_ptr() + 16 * int(fprim[k]), prim_count=int(pcounts[k]),
            aabbs=st["aabbs"].data_ptr() + 24 * int(fprim[k]), aabbs_keep=0)
    st["jobs"] = jobs
    return st


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("volume", "surface"):
        v = _input(case, seed)
        form = case.get("form", "build")
        if form == "host":
            state["voxels"] = v.cpu().numpy().view(np.uint32)
        elif form == "noalloc":
            state.update(_noalloc_state(case, v))
        else:
            state["voxels"] = v
    elif kind == "rebuild":
        state["keys"], state["vals"], _ = _sorted_voxels(case["log2"], seed)
        state["edits"] = _edits(case["log2"], case["edits"], seed, _mirror(seed, "xyzs"))
    elif kind == "downsample":
        state["keys"], state["vals"], _ = _sorted_voxels(case["log2"], seed)
    elif kind == "world":
        state["world"] = _world(case, seed)
    elif kind == "batch":
        state.update(_batch_state(case, seed))
    elif kind == "install":
        state.update(_install_state(case, seed))
    else:
        state.update(_path_edit_state(case, seed))
    return state


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def _run_noalloc(s):
    case, v, out = s["case"], s["voxels"], native.BuiltC()
    native.check(native.lib().pyrb_build_noalloc(
        ctypes.c_void_p(_stream()), case["log2"], case["rt"], v.data_ptr(), len(v), s["nodes"].data_ptr(),
        len(s["nodes"]), s["leaves"].data_ptr(), len(s["leaves"]), s["keys"].data_ptr(), s["attrs"].data_ptr(),
        len(s["keys"]), s["prims"].data_ptr(), s["aabbs"].data_ptr(), len(s["prims"]), ctypes.byref(out)))
    return {"nodes": s["nodes"][:out.node_words], "leaves": s["leaves"][:out.leaf_count],
            "keys": s["keys"][:out.voxel_count], "attrs": s["attrs"][:out.voxel_count],
            "prims": s["prims"][:out.prim_count], "aabbs": s["aabbs"][:out.prim_count], "root": int(out.root)}


def _run_install(s):
    pal, counts = gpu_build.palette_scan(s["attrs"], s["first"])
    dst, words = gpu_build.palette_layout(s["first"], counts)
    gpu_build.palette_pack(s["attrs"], s["first"], pal, counts, dst, s["pool"])
    known = torch.from_numpy((counts != gpu_build.PALETTE_OVERFLOW).astype(np.int32)).cuda()
    return {"palettes": pal * known[:, None], "counts": counts.view(np.int32), "pool": s["pool"][:words]}


def _run_path_edit(s):
    s["prims"].copy_(s["prims0"])
    s["aabbs"].copy_(s["aabbs0"])
    ex = native.Exec()
    ex.stream = ctypes.c_void_p(_stream())
    native.check(native.lib().pyrb_path_edit(
        ctypes.byref(ex), s["nodes"].data_ptr(), s["leaves"].data_ptr(), s["attrs"].data_ptr(), s["jobs"],
        len(s["jobs"]), s["edits"].ctypes.data, len(s["edits"])))
    words = np.frombuffer(s["jobs"], np.int32).reshape(len(s["jobs"]), -1)
    at = native.PathEditJob.out_root.offset // 4
    return {"nodes": s["nodes"], "leaves": s["leaves"], "attrs": s["attrs"][s["out"]:], "prims": s["prims"],
            "aabbs": s["aabbs"], "jobs": words[:, at:at + 4].copy()}


def run(state):
    case = state["case"]
    kind, form = case["kind"], case.get("form", "build")
    if kind in ("volume", "surface"):
        if form == "noalloc":
            return _run_noalloc(state)
        if form == "host":
            return _outputs(gpu_build.geometry_build(case["log2"], case["rt"], state["voxels"]))
        return _outputs(gpu_build.build(case["log2"], case["rt"], state["voxels"]))
    if kind == "rebuild":
        return _outputs(gpu_build.build(case["log2"], case["rt"], state["edits"], old_keys=state["keys"],
                                        old_vals=state["vals"]))
    if kind == "downsample":
        return _outputs(gpu_build.downsample(case["log2"], case["rt"], state["keys"], state["vals"],
                                             len(state["keys"]), case["shift"]))
    if kind == "world":
        vox, counts, edits, eofs, total = state["world"]
        return _outputs(gpu_build.build_chunks_edits(case["log2"], case["rt"], case["chunks"], case["capacity"], vox,
                                                     counts, edits if total else None, eofs, total))
    if kind == "batch":
        return _outputs(_run_batch(state, case["rt"]))
    if kind == "install":
        return _run_install(state)
    return _run_path_edit(state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _voxels(case):
    """About how many voxels a case holds."""
    kind = case["kind"]
    if kind == "surface":
        return case["nx"] * case["nz"]
    if kind == "world":
        return case["chunks"] * min(case["capacity"], 3 << (2 * case["log2"]))
    if kind in ("batch", "install", "path_edit"):
        return int((8 ** _edges(case).astype(np.int64)).sum() // 2)
    part = {"terrain": 0.5, "noise": 0.3, "skin": 1 / 7, "bernoulli": case.get("p", 0.15)}[case.get("fill", "noise")]
    return int(part * 8 ** case["log2"])


def work(case):
    kind, n = case["kind"], _voxels(case)
    out = 12 * n                                  # keys and attributes of the result
    if kind in ("volume", "surface"):
        read = 16 * (n + case.get("edits", 0))
    elif kind == "rebuild":
        read = 12 * n + 16 * case["edits"]
    elif kind == "downsample":
        read, out = 12 * n, 12 * n // 8 ** case["shift"]
    elif kind in ("world", "batch"):
        read = 16 * n + 8 * case["edits"] * case["chunks"]
    elif kind == "install":                       # attributes in, a fifth of them out whole, the rest as nibbles
        read, out = 4 * n, int(n * (0.2 * 4 + 0.8 * 0.5))
    else:                                         # attributes copied to their new place
        read, out = 4 * n + 16 * case["edits"] * case["chunks"], 4 * n
    return {"bytes": read + out, "flops": 0}


# ---------------------------------------------------------------------------
# exact
# ---------------------------------------------------------------------------
def _boxes(chunk, pts, log2c, rt):
    """Boxes of the occupied cells of edge 2^rt (chunk after chunk, in Morton order) of a
    list of entries, the last of equal positions deciding and attribute 0 removing."""
    x, y, z = (pts[:, k].long() for k in range(3))
    n = 1 << log2c
    fits = (pts[:, :3] >= 0).all(1) & (x < n) & (y < n) & (z < n)
    chunk, x, y, z, a = chunk[fits], x[fits], y[fits], z[fits], pts[fits, 3]
    span = int(n.max()) if torch.is_tensor(n) else n
    order = (((chunk * span + z) * span + y) * span + x).sort(stable=True)
    last = torch.ones_like(order.values, dtype=torch.bool)
    last[:-1] = order.values[1:] != order.values[:-1]
    keep = order.indices[last]
    keep = keep[a[keep] != 0]
    chunk, x, y, z = chunk[keep], x[keep], y[keep], z[keep]
    cell = chunk * 8 ** max(span.bit_length() - 1 - rt, 0) + _morton(x >> rt, y >> rt, z >> rt)
    cells, at = cell.unique(return_inverse=True)
    out = torch.empty((len(cells), 6), dtype=torch.float64, device="cuda")
    for k, v in enumerate((x, y, z)):
        big = torch.full((len(cells),), 1 << 40, dtype=torch.int64, device="cuda")
        out[:, k] = big.scatter_reduce(0, at, v, "amin").double() - 1 / 256
        out[:, 3 + k] = (big * 0).scatter_reduce(0, at, v, "amax").double() + 1 + 1 / 256
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("install", "path_edit") or _voxels(case) > EXACT_MOST:
        return None
    if kind in ("volume", "surface"):
        v, log2c = _input(case, seed), case["log2"]
        chunk = torch.zeros(len(v), dtype=torch.int64, device="cuda")
    elif kind in ("rebuild", "downsample"):
        _, _, v = _sorted_voxels(case["log2"], seed)
        log2c = case["log2"]
        if kind == "rebuild":
            v = torch.cat([v, _edits(case["log2"], case["edits"], seed, _mirror(seed, "xyzs"))])
        else:
            v[:, :3] >>= case["shift"]
            log2c -= case["shift"]
        chunk = torch.zeros(len(v), dtype=torch.int64, device="cuda")
    elif kind == "world":
        vox, counts, edits, eofs, total = _world(case, seed)
        K, cap, log2c = case["chunks"], case["capacity"], case["log2"]
        ids = torch.arange(K, device="cuda")
        held = torch.arange(cap, device="cuda")[None, :] < counts[:, None]
        chunk = torch.cat([ids[:, None].expand(K, cap)[held], ids.repeat_interleave(eofs.diff().long())])
        v = torch.cat([vox[held], edits])
    else:
        order, log2s, vox, starts, sizes = _mix(case, seed)
        edits, eoffs = _mix_edits(case, order, log2s, seed)
        at = np.concatenate([np.arange(f, f + n) for f, n in zip(starts, sizes)])
        ids = np.arange(len(log2s))
        chunk = torch.from_numpy(np.concatenate([np.repeat(ids, sizes), np.repeat(ids, np.diff(eoffs))])).cuda()
        v = torch.cat([vox[torch.from_numpy(at).cuda()], torch.from_numpy(edits.view(np.int32)).cuda()])
        log2c = torch.from_numpy(log2s.astype(np.int64)).cuda()[chunk]
    least = int(_edges(case).min()) if kind == "batch" else log2c
    boxes = _boxes(chunk, v, log2c, min(max(case["rt"], 3), least))
    values = {name: None for name in ("nodes", "leaves", "keys", "attrs", "prims", "root")}
    if kind in ("world", "batch"):
        values.update(roots=None, first_voxel=None, first_prim=None)
    return dict(values, aabbs=boxes)
