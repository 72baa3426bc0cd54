"""The optimizer's list of inner nodes is made on the device: ascending, for whole and ragged tiles of nodes and
for an array whose inner nodes are not in front."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 512, 513, 1024, 5000, 600000])
def test_ascending_inner_nodes(gpu, n):
    import torch
    vert, faces = scenes.uniform_soup(n, sigma=0.01, seed=n)
    nodes = gpu.LBVH(n, 30).build(torch.from_numpy(vert).cuda(), torch.from_numpy(faces.view(np.int32)).cuda())
    # more nodes than the tree has: what lies behind it is listed by its own flag
    more = torch.cat([nodes, nodes[n // 2:n + 7]])
    for a in (nodes, more):
        opt = gpu.Bittner13GPU(a, num_nodes=a.shape[0])
        flag = gpu.nodes_to_numpy(a)["isLeafFlag"]
        assert np.array_equal(opt.inner_nodes().cpu().numpy(), np.flatnonzero(flag == 0).astype(np.int32))
        opt.close()
