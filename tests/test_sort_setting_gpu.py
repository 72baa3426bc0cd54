"""The process-wide tile of the sorts is the one they use: a pass over tiles of 8,192 keys has a scan launch
that the smaller tiles' passes do without, which the count of launches shows."""
import pytest

pytestmark = pytest.mark.gpu


def _launches(gpu, n, bytes_):
    import torch
    from bvhtest_gb300 import native
    lib = native.load()
    keys = torch.randint(0, 2 ** 31 - 1, (n,), device="cuda", dtype=torch.int32 if bytes_ == 4 else torch.int64)
    before = lib.bvhgb_launch_count()
    k, v = gpu.radix_sort_pairs(keys, torch.arange(n, dtype=torch.int32, device="cuda"))
    launches = lib.bvhgb_launch_count() - before
    ref, order = torch.sort(keys, stable=True)
    assert torch.equal(k, ref) and torch.equal(v, order.to(torch.int32))
    return launches


@pytest.mark.parametrize("bytes_", [4, 8])
@pytest.mark.parametrize("n", [4097, 200000, 262144, 300000])
def test_given_tile_is_used(gpu, n, bytes_):
    prev = gpu.sort_default_tile(2048)
    try:
        small = _launches(gpu, n, bytes_)
        gpu.sort_default_tile(4096)
        assert _launches(gpu, n, bytes_) == small
        gpu.sort_default_tile(8192)
        assert _launches(gpu, n, bytes_) == small + 1
    finally:
        assert gpu.sort_default_tile(prev) == 8192
    assert gpu.sort_default_tile(0) == prev
    assert _launches(gpu, 4000, bytes_) == 1  # the automatic choice again: placed by counting


@pytest.mark.parametrize("tile", [2048, 4096, 8192])
@pytest.mark.parametrize("n", [4097, 200000, 600000])
def test_morton_sort_with_a_given_tile(gpu, n, tile):
    """The 63-bit build's sort: even keys (upper bits, then groups), then the same with half of them in one cell
    (all bits)."""
    import numpy as np
    import torch
    p = torch.rand((n, 1, 3), device="cuda")
    f = torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(-1, 3)
    b = gpu.LBVH(n, 63, "karras")
    prev = gpu.sort_default_tile(tile)
    try:
        for _ in range(2):
            v = p.expand(n, 3, 3).reshape(-1, 3).contiguous()
            b.init_tri_data(v, f)
            b.calc_morton(v, f)
            b.sort(n)
            keys, _ = b.keys(n, False)
            order = np.argsort(keys, kind="stable")
            k, i = b.keys(n, True)
            assert np.array_equal(k, keys[order]) and np.array_equal(i, order.astype(np.uint32))
            p[: n // 2] = 0.3 + 1e-4 * p[: n // 2]
    finally:
        gpu.sort_default_tile(prev)
    assert b.errors() == 0
