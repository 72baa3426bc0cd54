"""What the root's parent link holds is nobody's business: a tree whose root names no parent is optimised
like one whose root names node 0, without an error bit."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2], ids=["batched", "heap", "alt"])
@pytest.mark.parametrize("n,iters", [(3, 1), (40, 2), (600, 3)])
def test_root_without_a_parent(gpu, n, iters, mode):
    import torch
    vert, faces = scenes.uniform_soup(n, seed=n)
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    nodes = gpu.LBVH(n, 30, "refCompat").build(v, f)
    trees, stats, gains = [], [], []
    for parent in (0, 0xFFFFFFFF):
        t = gpu.nodes_to_numpy(nodes).copy()
        t["parent"][0] = parent
        dev = gpu.nodes_from_numpy(t)
        opt = gpu.Bittner13GPU(dev, num_nodes=2 * n - 1, batch_percent=75.0, num_chunks=2, search_mode=mode)
        gains.append(opt.gains(opt.inner_nodes()))
        opt.run(iters)
        torch.cuda.synchronize()
        stats.append(opt.stats())  # raises on a device error bit
        out = gpu.nodes_to_numpy(dev).copy()
        out["parent"][0] = 0
        trees.append(out)
        opt.close()
    assert torch.equal(gains[0].view(torch.int32), gains[1].view(torch.int32))
    assert stats[0] == stats[1]
    assert np.array_equal(trees[0].view(np.uint8), trees[1].view(np.uint8))
