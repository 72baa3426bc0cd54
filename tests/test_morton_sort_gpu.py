"""The 63-bit Morton sort (upper bits, then groups of equal upper bits) is the stable sort of the keys,
around the longest group it orders itself, with groups across the ends of its tiles, on equal keys
and for more keys than its 32-bit cells are meant for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(cells, runs, seed, same=False):
    """Points in 'cells' cells of the upper 32 bits, 'runs' of them in each, in random order, apart in the
    lower bits (or, same: some of them on the same key)."""
    g = np.random.default_rng(seed)
    cell = np.repeat(np.arange(cells), runs)
    at = (g.integers(1, 1023, (cells, 3)) + 0.25) / 1024  # the middle of a cell of 1 / 2048
    p = at[cell] + g.uniform(-1, 1, (cell.size, 3)) / 10000
    if same:
        p = at[cell] + g.integers(0, 3, (cell.size, 3)) / 30000
    p = np.concatenate([g.permutation(p), [[0, 0, 0], [1, 1, 1]]])
    return np.repeat(p[:, None, :], 3, axis=1).astype(np.float32)


def _check(gpu, tri):
    import torch
    n = tri.shape[0]
    v = torch.from_numpy(np.ascontiguousarray(tri.reshape(-1, 3))).cuda()
    f = torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(n, 3)
    b = gpu.LBVH(n, 63, "karras")
    b.init_tri_data(v, f)
    b.calc_morton(v, f)
    b.sort(n)
    raw, _ = b.keys(n, False)
    keys, idx = b.keys(n, True)
    order = np.argsort(raw, kind="stable")
    assert np.array_equal(keys, raw[order])
    assert np.array_equal(idx, order.astype(np.uint32))
    assert b.errors() == 0
    b.close()
    return raw


@pytest.mark.parametrize("runs", [1, 2, 31, 255, 256, 257, 700])
@pytest.mark.parametrize("same", [False, True])
def test_group_lengths(gpu, runs, same):
    raw = _check(gpu, _points(max(2, 40000 // runs), runs, runs, same))
    top = np.unique(raw >> np.uint64(31), return_counts=True)[1].max()
    assert top >= runs


@pytest.mark.parametrize("n", [1, 2, 3, 1023, 1024, 1025, 1279, 1280, 1281, 2049, 8193])
def test_sizes(gpu, n):
    g = np.random.default_rng(n)
    _check(gpu, np.repeat(g.random((n, 1, 3)), 3, axis=1).astype(np.float32))
    _check(gpu, np.full((n, 3, 3), 0.25, np.float32))


def test_groups_across_tiles(gpu):
    """Groups of every length up to 256 in a row: their ends fall on every place of a tile."""
    lengths = np.concatenate([np.arange(1, 257), np.arange(256, 0, -1)])
    g = np.random.default_rng(7)
    cells = np.stack(np.meshgrid(np.arange(8), np.arange(8), np.arange(8), indexing="ij"), -1).reshape(-1, 3)
    at = (cells[: lengths.size] * 100 + 50.25) / 1024
    p = np.repeat(at, lengths, axis=0) + g.uniform(-1, 1, (lengths.sum(), 3)) / 10000
    p = np.concatenate([g.permutation(p), [[0, 0, 0], [1, 1, 1]]])
    _check(gpu, np.repeat(p[:, None, :], 3, axis=1).astype(np.float32))


def test_many_keys(gpu):
    import torch
    n = (1 << 23) + 12345  # 40 upper bits
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    p = torch.rand((n, 1, 3), generator=g, device="cuda")
    p[: n // 2] = p[: n // 2] * 0.01
    _check(gpu, p.expand(n, 3, 3).cpu().numpy())


@pytest.mark.parametrize("n", [1025, 5000, 262144, 1100000])
@pytest.mark.parametrize("full", [0.02, 0.5])
def test_full_cells(gpu, n, full):
    """A part of the triangles in one cell of the upper bits: the sort of all bits at once, and again from the
    same keys; then an even mesh in the same workspace, whose cells are counted afresh."""
    import torch
    b = gpu.LBVH(n, 63, "karras")
    for part in (full, 0.0):
        g = np.random.default_rng(n)
        p = g.random((n, 1, 3))
        p[:int(part * n)] = 0.3 + 1e-4 * p[:int(part * n)]
        v = torch.from_numpy(np.repeat(p, 3, 1).reshape(-1, 3).astype(np.float32)).cuda()
        f = torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(-1, 3)
        b.init_tri_data(v, f)
        b.calc_morton(v, f)
        keys, _ = b.keys(n, False)
        order = np.argsort(keys, kind="stable")
        for _ in range(2):
            b.sort(n)
            k, i = b.keys(n, True)
            assert np.array_equal(k, keys[order]) and np.array_equal(i, order.astype(np.uint32))
    assert b.errors() == 0
