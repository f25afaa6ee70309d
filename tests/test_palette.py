"""Chunk attribute palettes (src/device/palette.zig): the oracle against hand-worked
cases of the reference's rules (CPU), and the CUDA scan/pack against the oracle byte
for byte on random chunks with colliding home slots and on a built chunk batch (GPU)."""
import numpy as np
import pytest

from oracle import oracle as orc

OVER = 0xFFFFFFFF


def _hash(v):
    h = (v * 0x9E3779B1) & 0xFFFFFFFF
    return h ^ (h >> 15)


def test_oracle_palette_rules():
    attrs = np.array([5, 5, 7] + list(range(1, 18)) + [9], np.uint32)
    first = np.array([0, 3, 20, 21, 21], np.uint32)   # last chunk empty
    pal, cnt = orc.palette_scan(attrs, first)
    assert list(cnt) == [2, OVER, 1, 0]
    order = sorted([5, 7], key=lambda v: _hash(v) & 63)
    assert list(pal[0]) == order + [order[0]] * 14          # slot order, padded with the first
    assert list(pal[2]) == [9] * 16 and list(pal[3]) == [0] * 16
    dst, total = orc.palette_layout(first, cnt)
    assert list(dst) == [0, 17, 34, 51] and total == 67
    pool = orc.palette_pack(attrs, first, pal, cnt, dst, total)
    idx = [order.index(v) for v in (5, 5, 7)]
    assert pool[16] == idx[0] | (idx[1] << 4) | (idx[2] << 8)
    assert list(pool[17:34]) == list(range(1, 18))            # overflow: 32-bit attributes
    assert list(pool[51:67]) == [0] * 16


def test_oracle_palette_empty_marker_and_collisions():
    # 0xFFFFFFFF is the table's empty marker: never inserted, packs as index 0
    pal, cnt = orc.palette_scan(np.array([OVER, 3, OVER], np.uint32), np.array([0, 3], np.uint32))
    assert cnt[0] == 1 and pal[0][0] == 3
    # two values with one home slot: the first inserted keeps it
    home = {}
    a = b = None
    for v in range(1, 100000):
        s = _hash(v) & 63
        if s in home:
            a, b = home[s], v
            break
        home[s] = v
    for seq in ([a, b], [b, a]):
        pal, cnt = orc.palette_scan(np.array(seq, np.uint32), np.array([0, 2], np.uint32))
        assert cnt[0] == 2 and list(pal[0][:2]) == seq


def _random_chunks(rng, count):
    sizes = rng.integers(0, 9000, count)
    sizes[::7] = 0
    first = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    attrs = np.empty(int(first[-1]), np.uint32)
    for c in range(count):
        k = int(rng.choice([1, 2, 5, 12, 16, 17, 40]))
        vals = rng.integers(1, 1 << 32, k, dtype=np.uint64).astype(np.uint32)
        if c % 3 == 0:   # values that share home slots
            vals = np.array([v for v in range(1, 5000) if _hash(v) & 63 in (3, 4)][:k], np.uint32)
        attrs[first[c]:first[c + 1]] = rng.choice(vals, int(sizes[c]))
    return attrs, first


def _check_against_oracle(attrs_host, attrs_dev, first):
    import torch
    from pyrit_b200 import gpu_build
    pal, cnt = gpu_build.palette_scan(attrs_dev, first)
    opal, ocnt = orc.palette_scan(attrs_host, first)
    assert np.array_equal(cnt, ocnt)
    keep = ocnt != OVER
    assert np.array_equal(pal.cpu().numpy().view(np.uint32)[keep], opal[keep])
    dst, total = gpu_build.palette_layout(first, cnt)
    odst, ototal = orc.palette_layout(first, ocnt)
    assert np.array_equal(dst, odst) and total == ototal
    pool = torch.zeros(max(total, 1), dtype=torch.int32, device="cuda")
    gpu_build.palette_pack(attrs_dev, first, pal, cnt, dst, pool)
    opool = orc.palette_pack(attrs_host, first, opal, ocnt, odst, ototal)
    assert np.array_equal(pool.cpu().numpy().view(np.uint32)[:total], opool)
    return cnt


@pytest.mark.gpu
def test_palette_random_chunks_match_oracle():
    from gpu_helpers import dev
    rng = np.random.default_rng(3)
    attrs, first = _random_chunks(rng, 300)
    cnt = _check_against_oracle(attrs, dev(attrs), first)
    assert (cnt == OVER).any() and (cnt != OVER).any()


@pytest.mark.gpu
def test_palette_of_a_chunk_batch_matches_oracle():
    """The install step after a batch build: palettes over the batch's attributes,
    chunk by chunk (first_voxel of the non-empty chunks, then voxel_count)."""
    from pyrit_b200 import gpu_build, workloads as wl
    log2s = wl.chunk_mix(64, 0)
    vox, offs = wl.mix_chunks_device(log2s, 0, 0)
    b = gpu_build.build_batch(log2s, 5, vox, offs)
    h = b.download()
    nonempty = [c for c in range(len(log2s)) if b.roots[c] != 0xFFFFFFFF]
    first = np.array([b.first_voxel[c] for c in nonempty] + [h.voxel_count], np.uint32)
    _check_against_oracle(h.attrs, b.attrs, first)
    b.free()


# Blocks of four steps of 4096 voxels: chunks that end around a step's and a block's last
# voxel, with one value, exactly as many as a palette holds and one more (all of them
# early, or the last one only at the chunk's end), and the table's empty marker among them.
@pytest.mark.gpu
@pytest.mark.parametrize("size", [1, 31, 4095, 4097, 16384, 16385, 40000])
def test_palette_steps_and_limits(size):
    from gpu_helpers import dev
    rng = np.random.default_rng(size)
    parts = []
    for k in (1, 2, 16, 17):
        vals = rng.integers(1, 1 << 31, k, dtype=np.uint64).astype(np.uint32)
        v = rng.choice(vals, size).astype(np.uint32)
        parts.append(v)
        late = rng.choice(vals[:-1] if k > 1 else vals, size).astype(np.uint32)
        late[-1] = vals[-1]
        parts.append(late)
        marked = np.sort(v)          # long runs
        marked[size // 2] = 0xFFFFFFFF
        parts.append(marked)
    first = np.arange(len(parts) + 1, dtype=np.uint32) * size
    attrs = np.concatenate(parts)
    _check_against_oracle(attrs, dev(attrs), first)


# Chunks of many blocks whose warps find the values beyond a palette's 16 at about the same
# time or one after another, beside chunks that just fit: the blocks' and warps' early ends.
@pytest.mark.gpu
@pytest.mark.parametrize("values", [17, 18, 64, 65, 5000])
def test_palette_early_ends(values):
    from gpu_helpers import dev
    rng = np.random.default_rng(values)
    parts = []
    for size in (256, 5000, 16384, 200_000):
        vals = rng.permutation(1 << 20)[:values].astype(np.uint32)
        parts.append(rng.choice(vals, size))                          # everywhere at once
        parts.append(np.sort(rng.choice(vals, size)))                 # in runs, warp after warp
        one = np.full(size, vals[0], np.uint32)                       # in the last rows only
        one[-min(values, size):] = vals[:min(values, size)]
        parts.append(one)
        parts.append(rng.choice(vals[:16], size))                     # a palette
    first = np.concatenate([[0], np.cumsum([len(v) for v in parts])]).astype(np.uint32)
    attrs = np.concatenate(parts).astype(np.uint32)
    cnt = _check_against_oracle(attrs, dev(attrs), first)
    assert (cnt == OVER).sum() >= 8 and (cnt[3::4] <= 16).all()


# Chunks whose voxels have the last indices of 32 bits: a block of 16384 voxels that starts
# there would end beyond them. The buffer holds these chunks only (an address that far below
# it stands for the attributes before them, which nothing reads).
@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1,), (16383,), (16384,), (16385, 4095), (3, 40000, 5000)])
def test_palette_of_the_last_voxel_indices(sizes):
    import torch
    from pyrit_b200 import gpu_build
    from gpu_helpers import dev
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    attrs = np.concatenate([rng.integers(0, 5 if c % 2 else 17, k) for c, k in enumerate(sizes)]).astype(np.uint32)
    ofirst = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    base = 0xFFFFFFFF - n
    first = (ofirst.astype(np.int64) + base).astype(np.uint32)
    assert first[-1] == 0xFFFFFFFF
    buf = dev(attrs)
    addr = buf.data_ptr() - 4 * base
    pal, cnt = gpu_build.palette_scan(addr, first)
    opal, ocnt = orc.palette_scan(attrs, ofirst)
    assert np.array_equal(cnt, ocnt)
    keep = ocnt != OVER
    assert np.array_equal(pal.cpu().numpy().view(np.uint32)[keep], opal[keep])
    dst, total = orc.palette_layout(ofirst, ocnt)
    pool = torch.zeros(max(total, 1), dtype=torch.int32, device="cuda")
    gpu_build.palette_pack(addr, first, pal, cnt, dst, pool)
    opool = orc.palette_pack(attrs, ofirst, opal, ocnt, dst, total)
    assert np.array_equal(pool.cpu().numpy().view(np.uint32)[:total], opool)


# The pack's table gives every palette entry a slot of its own, by the first of eight
# multipliers that does; these values share a slot under each of them. Palettes of the
# caller's may repeat entries and hold the table's empty marker; voxels outside have index 0.
@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["spread", "clash", "clash16", "repeats", "marker", "zero"])
def test_palette_pack_tables(kind):
    import torch
    from pyrit_b200 import gpu_build
    from gpu_helpers import dev
    rng = np.random.default_rng(len(kind))
    vals = [int(v) for v in rng.integers(1, 1 << 32, 16, dtype=np.uint64)]
    if kind.startswith("clash"):
        for t in range(8):
            m = (0x9E3779B1 + t * 0x3C6EF372) & 0xFFFFFFFF
            vals[t + 1] = (vals[t] + pow(m, -1, 1 << 32)) & 0xFFFFFFFF
            assert (vals[t] * m & 0xFFFFFFFF) >> 24 == (vals[t + 1] * m & 0xFFFFFFFF) >> 24
        if kind == "clash":
            vals[9:] = [vals[0]] * 7
    if kind == "repeats":
        vals = [vals[i] for i in (0, 1, 2, 1, 3, 2, 0, 4, 4, 4, 5, 1, 6, 6, 0, 0)]
    if kind == "marker":
        vals[5] = vals[9] = OVER
    if kind == "zero":
        vals[3] = 0
    pal = np.array([vals, vals[::-1]], np.uint32)
    outside = rng.integers(1, 1 << 32, 5, dtype=np.uint64).astype(np.uint32)
    pool = np.concatenate([pal[0], outside, np.array([0, OVER], np.uint32)])
    attrs = rng.choice(pool, 40_000).astype(np.uint32)
    first = np.array([0, 20_001, 40_000], np.uint32)
    cnt = np.array([16, 16], np.uint32)
    dst, total = orc.palette_layout(first, cnt)
    out = torch.zeros(total, dtype=torch.int32, device="cuda")
    gpu_build.palette_pack(dev(attrs), first, dev(pal), cnt, dst, out)
    want = orc.palette_pack(attrs, first, pal, cnt, dst, total)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    # the same values found by a scan
    if kind in ("spread", "clash", "clash16"):
        _check_against_oracle(np.resize(pal[0], 30_000), dev(np.resize(pal[0], 30_000)), np.array([0, 17, 30_000], np.uint32))
