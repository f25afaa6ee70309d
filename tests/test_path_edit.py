"""Path edits (src/device/pathedit.zig): voxels of a finished geometry changed without a
rebuild. CPU: the oracle's edited DAG decodes to the edited voxel set, its attributes
and RT prims equal those of a rebuild. GPU: the CUDA path edit equals the oracle byte
for byte on the pools, prims, boxes and job results (plain and palette attributes,
many jobs at once, a job that empties its geometry, a job whose arena overflows)."""
import numpy as np
import pytest

from oracle import oracle as orc
from pyrit_b200 import workloads as wl

EMPTY, OVERFLOW, REBUILD = 0x2, 0x4, 0x1


def _geometry(log2, rt, seed):
    vox = wl.mix_chunk(seed, log2, 0)
    return vox, orc.gb_build(log2, rt, vox)


def _edits(rng, log2, vox, n, remove_frac=0.4):
    """Random sets, inserts and removes (also of existing voxels), some repeated."""
    e = np.empty((n, 4), np.uint32)
    edge = 1 << log2
    for i in range(n):
        if rng.random() < 0.5 and len(vox):
            x, y, z = vox[rng.integers(len(vox))][:3]
        else:
            x, y, z = rng.integers(0, edge, 3)
        a = 0 if rng.random() < remove_frac else int(rng.integers(1, 9))
        e[i] = (x, y, z, a)
    if n > 4:
        e[n - 1] = e[0]
        e[n - 1, 3] = 7
    return e


def _job(g, log2, rt, n_edits, first=0, nodes_base=None, leaves_base=None, attrs_len=None, node_cap=None,
         attr_a=None):
    levels = max(log2 - 2, 0)
    return dict(node_offset=0, leaf_offset=0, root=g.root, log2_size=log2, attr_src=0, attr_count=g.voxel_count,
                attr_a=attr_a if attr_a is not None else len(g.attrs), attr_b=0, attr_cap=g.voxel_count + n_edits,
                palette=0, pal_src=0, pal_dst=0,
                node_arena=nodes_base if nodes_base is not None else len(g.nodes),
                node_cap=node_cap if node_cap is not None else n_edits * (levels * 10 + 4) + 8,
                leaf_arena=leaves_base if leaves_base is not None else len(g.leaves), leaf_cap=n_edits,
                edit_first=first, edit_count=n_edits, rt_log2=rt, prim_count=g.prim_count, aabbs_keep=0)


def _final_voxels(vox, edits):
    order = sorted(range(len(edits)), key=lambda i: (int(edits[i][2]) >> 2, int(edits[i][1]) >> 2,
                                                      int(edits[i][0]) >> 2))   # stable, as the host orders them
    cur = {(int(x), int(y), int(z)): int(a) for x, y, z, a in vox}
    for i in order:
        x, y, z, a = (int(v) for v in edits[i])
        if a:
            cur[(x, y, z)] = a
        else:
            cur.pop((x, y, z), None)
    return cur


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_oracle_path_edit_equals_rebuild(seed):
    log2, rt = 5, 4
    rng = np.random.default_rng(seed)
    vox, g = _geometry(log2, rt, seed)
    ed = _edits(rng, log2, vox, 60)
    job = _job(g, log2, rt, len(ed))
    nodes = np.concatenate([g.nodes, np.zeros(job["node_cap"], np.uint32)])
    leaves = np.concatenate([g.leaves, np.zeros(job["leaf_cap"], np.uint64)])
    attrs = np.concatenate([g.attrs, np.zeros(job["attr_cap"], np.uint32)])
    n2, l2, a2, p2, b2, out = orc.path_edit(nodes, leaves, attrs, [job], ed, g.prims, g.aabbs)
    o = out[0]
    final = _final_voxels(vox, ed)
    assert o["out_count"] == len(final)
    assert not (o["out_flags"] & (EMPTY | OVERFLOW))
    edge = 1 << log2
    idx = np.arange(edge ** 3, dtype=np.uint64)
    pts = np.stack([idx % edge, (idx // edge) % edge, idx // (edge * edge)], axis=1).astype(np.uint32)
    got = orc.lookup_many(log2, n2, l2, a2[o["attr_a"]:o["attr_a"] + o["out_count"]], o["out_root"], pts)
    want = np.array([final.get((int(x), int(y), int(z)), 0) for x, y, z in pts], np.uint32)
    assert np.array_equal(got, want)
    # attributes, prims and boxes equal a rebuild of the edited voxels
    fv = np.array([[x, y, z, a] for (x, y, z), a in final.items()], np.uint32)
    r = orc.gb_build(log2, rt, fv)
    assert np.array_equal(a2[o["attr_a"]:o["attr_a"] + o["out_count"]], r.attrs)
    if not (o["out_flags"] & REBUILD) and len(r.prims) // 16 == g.prim_count:
        gp, rp = p2.reshape(-1, 16), r.prims.reshape(-1, 16)
        assert np.array_equal(gp[:, 4:16], rp[:, 4:16])          # attribute rank and cell
        assert np.array_equal(b2.reshape(-1).view(np.uint32), r.aabbs.view(np.uint32))


def test_oracle_path_edit_empties_and_overflows():
    log2, rt = 5, 4
    vox, g = _geometry(log2, rt, 4)
    small = vox[:40]
    g = orc.gb_build(log2, rt, small)
    ed = small.copy()
    ed[:, 3] = 0                                               # remove everything
    job = _job(g, log2, rt, len(ed))
    nodes = np.concatenate([g.nodes, np.zeros(job["node_cap"], np.uint32)])
    leaves = np.concatenate([g.leaves, np.zeros(job["leaf_cap"], np.uint64)])
    attrs = np.concatenate([g.attrs, np.zeros(job["attr_cap"], np.uint32)])
    *_, out = orc.path_edit(nodes, leaves, attrs, [job], ed, g.prims, g.aabbs)
    assert out[0]["out_flags"] & EMPTY
    job = _job(g, log2, rt, 5, node_cap=6)
    *_, out = orc.path_edit(nodes, leaves, attrs, [job], _edits(np.random.default_rng(0), log2, small, 5, 0.0),
                            g.prims, g.aabbs)
    assert out[0]["out_flags"] & OVERFLOW


def _batch_jobs(rng, palette):
    """Jobs over the chunks of a batch built on the GPU: host pools with arenas and
    attribute targets, random edits per chunk, one chunk emptied, one with an arena
    too small. Returns (pools dict, jobs, edits, prim/box host arrays)."""
    from pyrit_b200 import gpu_build
    log2s = np.array([5, 6, 5, 5, 6, 5, 5, 6], np.uint32)
    chunks = [wl.mix_chunk(40 + c, int(l), 0) for c, l in enumerate(log2s)]
    chunks[3] = chunks[3][:30]
    offs = np.concatenate([[0], np.cumsum([len(c) for c in chunks])]).astype(np.uint32)
    b = gpu_build.build_batch(log2s, 4, np.concatenate(chunks), offs)
    h = b.download()
    roots, fv, fp = b.roots.copy(), b.first_voxel.copy(), b.first_prim.copy()
    b.free()
    nz = [c for c in range(len(log2s)) if roots[c] != 0xFFFFFFFF]
    nodes, leaves, attrs = list(h.nodes), list(h.leaves), list(h.attrs)
    prims, aabbs = h.prims.copy(), h.aabbs.copy()
    n_nodes, n_leaves = len(nodes), len(leaves)
    attr_pool = np.array(attrs, np.uint32)
    counts = first = None
    if palette:
        first = np.array([fv[c] for c in nz] + [h.voxel_count], np.uint32)
        pal, counts = orc.palette_scan(attr_pool, first)
        dst, total = orc.palette_layout(first, counts)
        attr_pool = orc.palette_pack(attr_pool, first, pal, counts, dst, total)
    jobs, edits, node_pos, leaf_pos = [], [], n_nodes, n_leaves
    attr_tail = len(attr_pool)
    extra_attrs = []
    for k, c in enumerate(nz):
        lc = int(log2s[c])
        vox_c = chunks[c]
        n_e = 0 if k == 5 else int(rng.integers(5, 60))
        if c == 3:   # the 30-voxel chunk: remove all of it
            e = vox_c.copy()
            e[:, 3] = 0
            n_e = len(e)
        else:
            e = _edits(rng, lc, vox_c, n_e)
        count = int(h.nodes[roots[c] + 1])
        nxt = [fp[d] for d in nz if d > c]
        pc = (nxt[0] if nxt else len(prims) // 16) - fp[c]
        levels = lc - 2
        node_cap = 4 if k == 4 else n_e * (levels * 10 + 4) + 8
        j = dict(node_offset=0, leaf_offset=0, root=int(roots[c]), log2_size=lc, attr_src=int(fv[c]),
                 attr_count=count, attr_b=0, palette=0, pal_src=0, pal_dst=0, node_arena=node_pos, node_cap=node_cap,
                 leaf_arena=leaf_pos, leaf_cap=n_e, edit_first=len(edits), edit_count=n_e, rt_log2=4,
                 prim_count=int(pc), prim_first=int(fp[c]), aabbs_keep=int(k % 2))
        if palette and counts[k] != 0xFFFFFFFF:
            words = 16 + (count + n_e + 7) // 8
            j.update(palette=1, pal_src=int(dst[k]), attr_src=int(dst[k]) + 16, pal_dst=attr_tail,
                     attr_a=attr_tail + 16, attr_cap=(words - 16) * 8)
        else:
            if palette:
                j["attr_src"] = int(dst[k])
            words = count + n_e
            j.update(attr_a=attr_tail, attr_cap=words)
        attr_tail += words
        node_pos += node_cap
        leaf_pos += n_e
        edits.extend(e.tolist())
        jobs.append(j)
    pools = dict(nodes=np.concatenate([np.array(nodes, np.uint32), np.zeros(node_pos - n_nodes, np.uint32)]),
                 leaves=np.concatenate([np.array(leaves, np.uint64), np.zeros(leaf_pos - n_leaves, np.uint64)]),
                 attrs=np.concatenate([attr_pool, np.zeros(attr_tail - len(attr_pool), np.uint32)]))
    return pools, jobs, np.array(edits, np.uint32).reshape(-1, 4), prims, aabbs


@pytest.mark.gpu
@pytest.mark.parametrize("palette", [False, True])
def test_cuda_path_edit_matches_oracle(palette):
    import ctypes
    import torch
    from pyrit_b200 import gpu_build, native
    from gpu_helpers import dev
    rng = np.random.default_rng(7 if palette else 8)
    pools, jobs, edits, prims, aabbs = _batch_jobs(rng, palette)
    n2, l2, a2, p2, b2, want = orc.path_edit(pools["nodes"], pools["leaves"], pools["attrs"], jobs, edits,
                                             prims, aabbs)
    dn, dl, da = dev(pools["nodes"]), dev(pools["leaves"]), dev(pools["attrs"])
    dp = torch.from_numpy(prims.copy()).cuda()
    db = torch.from_numpy(aabbs.copy()).cuda()
    cj = []
    for jd in jobs:
        j = native.PathEditJob()
        for k, v in jd.items():
            if k != "prim_first":
                setattr(j, k, v)
        j.prims = dp.data_ptr() + 16 * jd["prim_first"] if jd["prim_count"] else 0
        j.aabbs = db.data_ptr() + 24 * jd["prim_first"] if jd["prim_count"] else 0
        cj.append(j)
    gpu_build.path_edit(dn, dl, da, cj, edits)
    for w, g in zip(want, cj):
        assert (g.out_root, g.out_count, g.out_flags) == (w["out_root"], w["out_count"], w["out_flags"])
    flags = [w["out_flags"] for w in want]
    assert any(f & EMPTY for f in flags) and any(f & OVERFLOW for f in flags)
    assert np.array_equal(dn.cpu().numpy().view(np.uint32), n2)
    assert np.array_equal(dl.cpu().numpy().view(np.uint64), l2)
    assert np.array_equal(da.cpu().numpy().view(np.uint32), a2)
    assert np.array_equal(dp.cpu().numpy().reshape(-1, 16), p2)
    assert np.array_equal(db.cpu().numpy().reshape(-1).view(np.uint32), b2.reshape(-1).view(np.uint32))


def _decode(keys):
    """Coordinates of sorted voxel keys (brick Morton << 6 | x&3 + 4(y&3) + 16(z&3))."""
    k = keys.astype(np.uint64)
    out = np.empty((len(k), 3), np.uint32)
    for a in range(3):
        v = (k >> np.uint64(2 * a)) & np.uint64(3)
        for b in range(18):
            v |= ((k >> np.uint64(6 + 3 * b + a)) & np.uint64(1)) << np.uint64(2 + b)
        out[:, a] = v
    return out


# The attribute rewrite takes steps of 4096 attributes in tiles of 16384 and traces every
# operation once:
# operations at the steps' first and last places, voxels set, removed and set again in one
# job, the most edits a job takes, more prims than the walk keeps in shared memory, and
# one prim over the whole volume.
@pytest.mark.gpu
@pytest.mark.parametrize("log2,rt,n_edits,kind", [(6, 6, 96, "edges"), (6, 3, 300, "edges"), (5, 5, 4096, "repeats"),
                                                  (7, 3, 400, "random")])
def test_cuda_path_edit_tiles_and_repeats(log2, rt, n_edits, kind):
    import torch
    from pyrit_b200 import gpu_build, native
    from gpu_helpers import dev
    rng = np.random.default_rng(log2 * 100 + rt)
    vox, g = _geometry(log2, rt, 60 + log2)
    ed = _edits(rng, log2, vox, n_edits)
    if kind == "edges":
        ranks = np.concatenate([np.arange(t - 2, t + 3) for t in range(4096, g.voxel_count, 4096)] +
                               [np.array([0, 1, g.voxel_count - 1])])
        pos = _decode(g.keys[ranks[ranks < g.voxel_count]])
        at = rng.permutation(n_edits)[:min(len(pos), n_edits)]
        ed[at, :3] = pos[:len(at)]
        ed[at, 3] = np.where(rng.random(len(at)) < 0.6, 0, 9)
    elif kind == "repeats":
        ed[:, :3] = ed[rng.integers(0, 200, n_edits), :3]
    job = _job(g, log2, rt, n_edits)
    nodes = np.concatenate([g.nodes, np.zeros(job["node_cap"], np.uint32)])
    leaves = np.concatenate([g.leaves, np.zeros(job["leaf_cap"], np.uint64)])
    attrs = np.concatenate([g.attrs, np.zeros(job["attr_cap"], np.uint32)])
    n2, l2, a2, p2, b2, want = orc.path_edit(nodes, leaves, attrs, [job], ed, g.prims, g.aabbs)
    dn, dl, da = dev(nodes), dev(leaves), dev(attrs)
    dp, db = torch.from_numpy(g.prims.copy()).cuda(), torch.from_numpy(g.aabbs.copy()).cuda()
    j = native.PathEditJob(**job)
    j.prims, j.aabbs = dp.data_ptr(), db.data_ptr()
    out = [j]
    gpu_build.path_edit(dn, dl, da, out, ed)
    assert (out[0].out_root, out[0].out_count, out[0].out_flags) == tuple(
        want[0][k] for k in ("out_root", "out_count", "out_flags"))
    assert np.array_equal(dn.cpu().numpy().view(np.uint32), n2)
    assert np.array_equal(dl.cpu().numpy().view(np.uint64), l2)
    assert np.array_equal(da.cpu().numpy().view(np.uint32), a2)
    assert np.array_equal(dp.cpu().numpy().reshape(-1), p2.reshape(-1))
    assert np.array_equal(db.cpu().numpy().reshape(-1).view(np.uint32), b2.reshape(-1).view(np.uint32))


# A job whose arena has no room for the path of a brick that loses all its voxels: its count
# stays, its operations are there, and the last places of its target would come from behind
# its attributes. Here nothing of the caller's lies there: the source ends the pool, and
# words of a later owner follow it.
@pytest.mark.gpu
@pytest.mark.parametrize("palette", [False, True])
@pytest.mark.parametrize("room", [4, 12])
def test_cuda_path_edit_overflow_reads_its_own_attributes_only(palette, room):
    from pyrit_b200 import gpu_build, native
    from gpu_helpers import dev
    log2, rt = 5, 4
    brick = np.array([[x, y, z, 1 + (x + y + z) % 5] for z in range(4) for y in range(4) for x in range(4)], np.uint32)
    vox = np.concatenate([brick, brick + np.array([8, 8, 8, 0], np.uint32)])
    g = orc.gb_build(log2, rt, vox)
    ed = brick + np.array([8, 8, 8, 0], np.uint32)
    ed[:, 3] = 0
    if room > 4:  # room for the path of an earlier brick
        ed = np.concatenate([np.array([[4, 0, 0, 3]], np.uint32), ed])
    job = _job(g, log2, rt, len(ed), node_cap=room)
    cap = job["attr_cap"]
    src, first = g.attrs, np.array([0, g.voxel_count], np.uint32)
    job.update(attr_a=0, attr_src=cap)
    if palette:
        pal, counts = orc.palette_scan(g.attrs, first)
        dst, total = orc.palette_layout(first, counts)
        src = orc.palette_pack(g.attrs, first, pal, counts, dst, total)
        job.update(palette=1, pal_src=cap + 16, attr_src=cap + 32, pal_dst=0, attr_a=16, attr_cap=cap - 16)
        src = np.concatenate([np.zeros(16, np.uint32), src])
    pool = np.concatenate([np.zeros(cap, np.uint32), src])
    behind = np.full(128, 0x77777777, np.uint32)
    nodes = np.concatenate([g.nodes, np.zeros(room, np.uint32)])
    leaves = np.concatenate([g.leaves, np.zeros(job["leaf_cap"], np.uint64)])
    n2, l2, a2, p2, b2, want = orc.path_edit(nodes, leaves, np.concatenate([pool, 0 * behind]), [job], ed, g.prims, g.aabbs)
    assert want[0]["out_flags"] & OVERFLOW and want[0]["out_count"] == g.voxel_count + (room > 4)
    dn, dl, da = dev(nodes), dev(leaves), dev(np.concatenate([pool, behind]))
    dp, db = dev(g.prims), dev(g.aabbs.view(np.uint32))
    j = native.PathEditJob(**job)
    j.prims, j.aabbs = dp.data_ptr(), db.data_ptr()
    out = [j]
    gpu_build.path_edit(dn, dl, da, out, ed)
    assert (out[0].out_root, out[0].out_count, out[0].out_flags) == tuple(
        want[0][k] for k in ("out_root", "out_count", "out_flags"))
    assert np.array_equal(dn.cpu().numpy().view(np.uint32), n2)
    got = da.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[:len(pool)], a2[:len(pool)]) and np.array_equal(got[len(pool):], behind)


def _edited_by_both(job, nodes, leaves, attrs, ed, prims, aabbs):
    """The CUDA path edit against the oracle's, byte for byte; returns the oracle's boxes."""
    from pyrit_b200 import gpu_build, native
    from gpu_helpers import dev
    nodes = np.concatenate([nodes, np.zeros(job["node_cap"], np.uint32)])
    leaves = np.concatenate([leaves, np.zeros(job["leaf_cap"], np.uint64)])
    attrs = np.concatenate([attrs, np.zeros(job["attr_cap"], np.uint32)])
    n2, l2, a2, p2, b2, want = orc.path_edit(nodes, leaves, attrs, [job], ed, prims, aabbs)
    dn, dl, da, dp, db = dev(nodes), dev(leaves), dev(attrs), dev(prims), dev(aabbs.view(np.uint32))
    j = native.PathEditJob(**job)
    j.prims, j.aabbs = dp.data_ptr(), db.data_ptr()
    out = [j]
    gpu_build.path_edit(dn, dl, da, out, ed)
    assert (out[0].out_root, out[0].out_count, out[0].out_flags) == tuple(
        want[0][k] for k in ("out_root", "out_count", "out_flags"))
    assert np.array_equal(dn.cpu().numpy().view(np.uint32), n2)
    assert np.array_equal(dl.cpu().numpy().view(np.uint64), l2)
    assert np.array_equal(da.cpu().numpy().view(np.uint32), a2)
    assert np.array_equal(dp.cpu().numpy().reshape(-1), p2.reshape(-1))
    assert np.array_equal(db.cpu().numpy().reshape(-1).view(np.uint32), b2.reshape(-1).view(np.uint32))
    return b2


# Boxes of subtrees up to 2^10, by a warp with a stack in shared memory, and beyond, by one
# lane: the edges around the limit, few voxels in each prim and many.
@pytest.mark.gpu
@pytest.mark.parametrize("n", [30, 20000])
@pytest.mark.parametrize("log2,rt", [(7, 7), (9, 8), (10, 9), (10, 10), (11, 10), (11, 11), (12, 11)])
def test_cuda_path_edit_boxes_of_large_subtrees(log2, rt, n):
    rng = np.random.default_rng(log2 * 100 + rt + n)
    vox = np.concatenate([rng.integers(0, 1 << log2, (n, 3)), rng.integers(1, 9, (n, 1))], 1).astype(np.uint32)
    g = orc.gb_build(log2, rt, vox)
    ed = _edits(rng, log2, vox, 40)
    _edited_by_both(_job(g, log2, rt, len(ed)), g.nodes, g.leaves, g.attrs, ed, g.prims, g.aabbs)


# Full and nearly full trees of a 2^10 prim (8^8 bricks on a handful of shared nodes): the
# stack of the warp's walk at its deepest.
@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["full", "shared"])
def test_cuda_path_edit_box_of_a_full_subtree(kind):
    rng = np.random.default_rng(5)
    log2 = rt = 10
    leaf = np.array([1 << 21, 1 << 42, (1 << 21) | (1 << 22)], np.uint64)  # inner cells of a brick only
    count = [1, 1, 2]
    below = [(k, count[k]) for k in range(1 if kind == "full" else 3)]     # (reference, voxels) one level down
    nodes = []
    for s in range(2, log2):
        here = []
        for _ in range(1 if kind == "full" or s == log2 - 1 else 3):
            # (the first and last child stay: the whole cube is to be looked at)
            mask = 0xFF if kind == "full" or s == log2 - 1 else 0x81 | int(rng.integers(0, 256)) | 0x18
            kids = [below[int(rng.integers(len(below)))] for k in range(8) if mask >> k & 1]
            here.append((len(nodes), sum(c for _, c in kids)))
            nodes += [mask, sum(c for _, c in kids)] + [r for r, _ in kids]
        below = here
    root, voxels = below[0]
    attrs = (1 + np.arange(voxels) % 200).astype(np.uint32)
    ed = np.array([[1, 1, 1, 9], [2, 1, 1, 9], [1021, 1020, 1022, 9]], np.uint32)
    job = dict(node_offset=0, leaf_offset=0, root=root, log2_size=log2, attr_src=0, attr_count=voxels, attr_a=voxels,
               attr_b=0, attr_cap=voxels + 3, palette=0, pal_src=0, pal_dst=0, node_arena=len(nodes), node_cap=400,
               leaf_arena=len(leaf), leaf_cap=3, edit_first=0, edit_count=3, rt_log2=rt, prim_count=1, aabbs_keep=0)
    prim = np.zeros(16, np.uint8)
    prim[:4] = np.frombuffer(np.uint32(root).tobytes(), np.uint8)
    box = _edited_by_both(job, np.array(nodes, np.uint32), leaf, attrs, ed, prim, np.zeros(6, np.float32))
    assert (box.reshape(-1)[3:] - box.reshape(-1)[:3] > 1000).all()
