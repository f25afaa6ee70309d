"""Leaf and node levels at the sizes where their work changes hands: the leaves and first
levels of up to 4096 bricks in the one-block tail or in kernels of their own, tail levels
of up to 1024 parents in shared memory or through global memory, dedup tables whose
bounds (from the input size) are far above the real counts, and old voxels that come
twice or out of order. Byte for byte against the
oracle restatement of the reference GPU algorithm."""
import numpy as np
import pytest

from oracle import oracle as orc

from gpu_helpers import assert_same_build, dev

pytestmark = pytest.mark.gpu


def _bricks(rng, log2, n, per_parent):
    """n voxels in n different bricks, per_parent of them in every occupied 8^3 cell."""
    edge = 1 << (log2 - 3)
    parents = rng.choice(edge ** 3, (n + per_parent - 1) // per_parent, replace=False)
    cell = np.repeat(parents, per_parent)[:n]
    child = np.tile(np.arange(per_parent), len(parents))[:n]
    low = rng.integers(0, 4, (n, 3))
    pts = np.empty((n, 4), np.uint32)
    for a in range(3):
        pts[:, a] = (cell // edge ** a % edge) * 8 + ((child >> a) & 1) * 4 + low[:, a]
    pts[:, 3] = 1 + rng.integers(0, 200, n)
    return pts[rng.permutation(n)]


@pytest.mark.parametrize("n,per_parent", [(1, 1), (1023, 1), (1024, 1), (1025, 1), (4095, 1), (4096, 1), (4097, 1),
                                          (4096, 4), (4096, 8), (4097, 4), (3000, 3)])
@pytest.mark.parametrize("log2,rt", [(8, 5), (9, 9)])
def test_tail_limits(log2, rt, n, per_parent):
    from pyrit_b200 import gpu_build
    pts = _bricks(np.random.default_rng(n * 8 + per_parent), log2, n, per_parent)
    g = gpu_build.build(log2, rt, dev(pts)).download()
    assert_same_build(g, orc.gb_build(log2, rt, pts), label=f"{n} {per_parent}")


@pytest.mark.parametrize("edge", [3, 40, 300])
def test_tables_far_above_the_real_counts(edge):
    """2.2 M entries of a 2^11 volume inside a cube of `edge` bricks: bounds of millions of
    bricks (a leaf table of regions), a few, some ten thousand or as many real ones."""
    from pyrit_b200 import gpu_build
    rng = np.random.default_rng(edge)
    n = 2_200_000
    pts = np.empty((n, 4), np.uint32)
    pts[:, :3] = 512 + rng.integers(0, 4 * edge, (n, 3))
    pts[:, 3] = 1 + rng.integers(0, 200, n)
    g = gpu_build.build(11, 6, dev(pts)).download()
    assert_same_build(g, orc.gb_build(11, 6, pts), label=f"{edge}")


@pytest.mark.parametrize("path", [1, 2])
def test_one_large_chunk(path):
    """A batch of one chunk whose leaf table is filled region by region: its first voxel,
    first prim and root, which chunk batches of many chunks take from other kernels."""
    from pyrit_b200 import gpu_build
    rng = np.random.default_rng(path)
    log2, n = 9, 2_200_000
    pts = np.concatenate([rng.integers(0, 1 << log2, (n, 3)), rng.integers(1, 9, (n, 1))], 1).astype(np.uint32)
    offs = np.array([0, n], np.uint32)
    gpu_build.set_tuning(0, 0, 50, path)
    try:
        g = gpu_build.build_chunks(log2, 6, 1, n, dev(pts), dev(offs), n).download()
    finally:
        gpu_build.set_tuning(0, 0, 50, 0)
    assert_same_build(g, orc.gb_build_chunks(log2, 6, n, pts, offs), chunks=True, label=f"path {path}")


@pytest.mark.parametrize("order", ["sorted", "twice", "rotated", "shuffled"])
@pytest.mark.parametrize("n_new", [0, 1, 5000])
def test_order_of_the_old_voxels(order, n_new):
    """The last of equal keys counts, wherever it stands, and every edit after it."""
    from pyrit_b200 import gpu_build
    rng = np.random.default_rng(n_new)
    log2, n = 6, 60_000
    keys = np.sort(rng.choice(1 << 3 * log2, n, replace=False)).astype(np.uint64)
    if order != "sorted":
        keys = np.sort(keys[rng.integers(0, n, n)])
    if order == "rotated":
        keys = np.concatenate([keys[n // 3:], keys[: n // 2], np.array([1 << 3 * log2], np.uint64)])
    if order == "shuffled":
        keys = rng.permutation(keys)
    vals = rng.integers(0, 200, len(keys)).astype(np.uint32)
    ed = np.concatenate([rng.integers(0, 1 << log2, (n_new, 3)), rng.integers(0, 9, (n_new, 1))], 1).astype(np.uint32)
    gpu_build.set_tuning(0, 0, 50, 2)
    try:
        g = gpu_build.build(log2, 4, dev(ed) if n_new else None, old_keys=dev(keys), old_vals=dev(vals),
                            n_old=len(keys)).download()
    finally:
        gpu_build.set_tuning(0, 0, 50, 0)
    assert_same_build(g, orc.gb_build(log2, 4, ed, old_keys=keys, old_vals=vals), label=order)


@pytest.mark.parametrize("load", [25, 50, 90])
@pytest.mark.parametrize("n", [4096 * 4, 8192, 8193, 14745, 14747])
def test_table_sizes(n, load):
    """Bricks and parents at the counts where their tables stop taking four times the slots
    that the load factor asks for (2^14 slots), one voxel each and all of them different."""
    from pyrit_b200 import gpu_build
    rng = np.random.default_rng(n)
    pts = _bricks(rng, 9, n, 1)
    gpu_build.set_tuning(0, 0, load, 0)
    try:
        g = gpu_build.build(9, 5, dev(pts)).download()
    finally:
        gpu_build.set_tuning(0, 0, 50, 0)
    assert_same_build(g, orc.gb_build(9, 5, pts), label=f"{n} {load}")
