"""A tree built on keys that a timed-out sort left in no order, with NaN boxes, which a block merges node by node:
the build ends, the sort's error bit stands, and the next build is a normal one. The order is made from that of a
finished sort of the same keys, so every face in it exists."""
import ctypes as C

import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
TIMEOUT_BIT = 1


@pytest.mark.parametrize("n", [200000, 1 << 20])
@pytest.mark.parametrize("bits", [30, 63])
def test_build_ends(gpu, n, bits):
    import torch
    from bvhtest_gb300 import native
    lib = native.load()
    vert, faces = scenes.uniform_soup(n, seed=n)
    vert[faces[::50, 0], 1] = np.nan  # in every block of leaves
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    b = gpu.LBVH(n, bits, "karras")
    nodes = gpu.empty_nodes(2 * n - 1)
    b.init_tri_data(v, f)
    b.calc_morton(v, f)
    b.sort(n)
    assert b.errors() == 0
    assert lib.bvhgb_sort_set_spin_limit(0, None) == 0
    try:
        b.sort(n)
        torch.cuda.synchronize()
    finally:
        assert lib.bvhgb_sort_set_spin_limit(0xFFFFFFFF, None) == 0
    keys, idx = b.keys(n, True)
    assert idx.max() < n
    flags = b.errors()
    b.build_tree(v, f, nodes)
    torch.cuda.synchronize()
    assert flags & TIMEOUT_BIT or (np.diff(keys.astype(np.float64)) >= 0).all()
    assert b.errors() & TIMEOUT_BIT == flags & TIMEOUT_BIT
    again = b.build(v, f)
    torch.cuda.synchronize()
    assert b.errors() == 0
    other = gpu.LBVH(n, bits, "karras")
    assert torch.equal(other.build(v, f), again)
    print("timed out", flags & TIMEOUT_BIT, "descents", int((np.diff(keys.astype(np.float64)) < 0).sum()))
