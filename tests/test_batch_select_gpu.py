"""A batch of half a million inner nodes and more selects the nodes that its chunks read instead of
sorting all of them; every mesh's tree must still be that of the single-mesh optimizer, byte for byte:
around the sizes where a mesh keeps all its nodes and where its tiles end, with equal costs on both
sides of the last node kept (whose order is the index), and with other shares of the nodes."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
COUNTS = [2049, 2050, 1, 8193, 2, 8194, 16385, 300000, 40, 5000, 190000, 5000]


@pytest.mark.parametrize("chunks,percent", [(32, 1.0), (7, 2.5), (32, 12.0)])
def test_selection_equals_the_single_mesh_optimizer(gpu, chunks, percent):
    import torch
    verts = []
    for m, n in enumerate(COUNTS):
        v, _ = scenes.uniform_soup(n, sigma=0.01, seed=m)
        v = v.reshape(n, 3, 3)
        if n == 5000:
            v[:] = v[0] + (np.arange(n) % 16)[:, None, None].astype(np.float32)  # whole subtrees cost the same
        verts.append(v.reshape(-1, 3))
    base = np.cumsum([0] + COUNTS)
    v = torch.from_numpy(np.concatenate(verts).astype(np.float32)).cuda()
    f = torch.arange(3 * base[-1], dtype=torch.int32, device="cuda").reshape(-1, 3)
    b = gpu.Batch(COUNTS, num_chunks=chunks, batch_percent=percent)
    nodes = b.empty_nodes()
    b.build(v, f, nodes)
    b.optimize(nodes, 3)
    torch.cuda.synchronize()
    assert b.stats()[1] == 0
    for m, n in enumerate(COUNTS):
        mv, mf = v[3 * base[m]:3 * base[m + 1]], f[:n]
        ref = gpu.LBVH(n, 30).build(mv, mf)
        if n > 1:
            gpu.Bittner13GPU(ref, num_chunks=chunks, batch_percent=percent, num_nodes=2 * n - 1).run(3)
        assert torch.equal(b.mesh_nodes(nodes, m), ref[: 2 * n - 1]), (m, n)
