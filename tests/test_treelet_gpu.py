"""The block-wise tree build and the one-launch build of small meshes (up to 1,024 triangles) give the
nodes of the leaf-by-leaf climb (which the batched build still is), byte for byte, around the block
sizes, on equal and comb-like keys, and where a coordinate is infinite or no number (whose boxes depend
on the order of the merges); 63-bit keys against the oracle."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 3, 31, 255, 256, 257, 511, 513, 1000, 1024, 1025, 4096, 66049]


def _vert(kind, n, seed):
    vert, faces = scenes.uniform_soup(n, sigma=0.01, seed=seed)
    tri = vert.reshape(n, 3, 3)
    if kind == "equal":
        tri[:] = tri[0]
    elif kind == "runs":  # long runs of equal keys
        tri[:] = tri[np.arange(n) // 300 * 300 % n]
    elif kind == "comb":  # cells at powers of two on a line: a deep, one-sided tree
        tri[:] = 0.0
        tri[:, :, 0] = (0.5 ** (np.arange(n) % 22))[:, None]
    elif kind in ("nan", "inf"):
        g = np.random.default_rng(seed)
        pick = g.integers(0, n, max(1, n // 400))
        tri[pick, g.integers(0, 3, pick.size), g.integers(0, 3, pick.size)] = np.nan if kind == "nan" else np.inf
    return tri.reshape(-1, 3).astype(np.float32), faces


@pytest.mark.parametrize("topo", ["refCompat", "karras"])
@pytest.mark.parametrize("kind", ["soup", "equal", "runs", "comb", "nan", "inf"])
@pytest.mark.parametrize("n", SIZES)
def test_equals_the_climb(gpu, n, kind, topo):
    import torch
    vert, faces = _vert(kind, n, n)
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    one = gpu.LBVH(n, 30, topo)
    got = one.build(v, f)
    again = gpu.empty_nodes(2 * n - 1)
    one.build_tree(v, f, again)  # from the same sorted keys: slots and root counter re-armed
    phases = gpu.LBVH(n, 30, topo)  # what a build leaves is what the phases leave
    phases.init_tri_data(v, f)
    phases.calc_morton(v, f)
    phases.sort(n)
    assert np.array_equal(one.scene_box(), phases.scene_box(), equal_nan=True)
    for done in (False, True):
        for a, b in zip(one.keys(n, done), phases.keys(n, done)):
            assert np.array_equal(a, b)
    batch = gpu.Batch([n], topology=topo)
    ref = batch.empty_nodes()
    batch.build(v, f, ref)
    torch.cuda.synchronize()
    assert torch.equal(got, ref) and torch.equal(again, ref)
    assert one.errors() == 0


@pytest.mark.parametrize("topo", ["refCompat", "karras"])
@pytest.mark.parametrize("kind", ["soup", "equal", "runs", "comb"])
@pytest.mark.parametrize("n", [2, 255, 257, 1000, 1024, 5000, 66049])
def test_long_keys(gpu, orc, n, kind, topo):
    import torch
    vert, faces = _vert(kind, n, n + 1)
    b = gpu.LBVH(n, 63, topo)
    got = b.build(torch.from_numpy(vert).cuda(), torch.from_numpy(faces.view(np.int32)).cuda())
    torch.cuda.synchronize()
    ref, _, _ = orc.lbvh_build(vert, faces, 63, 0 if topo == "refCompat" else 1)
    assert np.array_equal(gpu.nodes_to_numpy(got).view(np.uint8), ref.view(np.uint8))
    assert b.errors() == 0


def _from_keys(keys):
    """One degenerate triangle per 63-bit key, in the middle of its Morton cell, and the two that hold the
    scene box at [0, 1]."""
    cell = np.zeros((keys.size, 3), np.int64)
    for bit in range(21):
        for axis in range(3):
            cell[:, axis] |= ((keys >> (3 * bit + 2 - axis)) & 1) << bit
    p = ((cell + 0.5) / 2097152.0).astype(np.float32)
    p = np.concatenate([p, np.ones((1, 3), np.float32), np.zeros((1, 3), np.float32)])
    return np.repeat(p, 3, 0), np.arange(3 * len(p), dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("kind", ["peaks", "one nan"])
def test_lists_that_are_not_joined(gpu, orc, kind):
    """A comb on both sides of every 256th leaf leaves more roots than a joining block takes, over a part of
    the leaves; one NaN keeps a part of the lists, and the wider ones over it, from being joined."""
    import torch
    if kind == "peaks":
        g = np.random.default_rng(5)
        step, mid, bit = 2 ** 56, int("01" * 27, 2), 2 ** np.arange(54, dtype=np.int64)
        runs = [g.integers(1, step // 8, 227)]  # with the cell at the origin and 28 of a comb: 256
        for c in range(1, 41):  # deltas fall away from the middle, which is a block's first leaf, on both sides
            runs += [c * step + mid - bit[::2], [c * step + mid], c * step + mid + bit[1::2],
                     c * step + g.integers(step // 3, step // 2, 201)]
        vert, faces = _from_keys(np.concatenate(runs + [g.integers(48 * step, 120 * step, 60000)]))
    else:
        vert, faces = _vert("soup", 66049, 3)
        vert[3 * 20000 + 1, 2] = np.nan
    n = len(faces)
    bits = 63 if kind == "peaks" else 30
    b = gpu.LBVH(n, bits, "karras")
    v, f = torch.from_numpy(vert).cuda(), torch.from_numpy(faces.view(np.int32)).cuda()
    got = b.build(v, f)
    torch.cuda.synchronize()
    if kind == "peaks":
        ref, _, _ = orc.lbvh_build(vert, faces, 63, 1)
        assert np.array_equal(gpu.nodes_to_numpy(got).view(np.uint8), ref.view(np.uint8))
    else:
        batch = gpu.Batch([n], topology="karras")
        ref = batch.empty_nodes()
        batch.build(v, f, ref)
        assert torch.equal(got, ref)
    assert b.errors() == 0
