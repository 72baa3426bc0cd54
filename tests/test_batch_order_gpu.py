"""The batched trace takes a mesh's tree in any order of its nodes: root 0 and links within the mesh are all
that is asked of it. Meshes in another order than the build's, and one with a bad link, stand among others."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
BAD_INDEX = 4
COUNTS = np.array([2, 700, 3, 1, 4000, 64, 5, 900], np.uint32)


def _batch(gpu):
    import torch
    vert = np.concatenate([scenes.uniform_soup(int(n), sigma=0.05, seed=80 + k)[0] for k, n in enumerate(COUNTS)])
    v = torch.from_numpy(vert).cuda()
    f = torch.arange(vert.shape[0], dtype=torch.int32, device="cuda").reshape(-1, 3)
    b = gpu.Batch(COUNTS)
    nodes = b.empty_nodes()
    b.build(v, f, nodes)
    b.optimize(nodes, 1)
    return v, f, b, gpu.nodes_to_numpy(nodes).copy()


def _permute(t, g):
    """The same tree with its nodes but the root in another order."""
    order = np.concatenate([[0], 1 + g.permutation(t.shape[0] - 1)])  # new -> old
    place = np.argsort(order).astype(np.uint32)
    out = t[order].copy()
    inner = out["isLeafFlag"] == 0
    out["left"][inner], out["right"][inner] = place[out["left"][inner]], place[out["right"][inner]]
    out["parent"] = place[out["parent"]]
    return out


def _check(gpu, b, v, f, nodes, rays, skip=()):
    import torch
    hits, org, d = b.trace_random(nodes, v, f, rays, seed=9, with_rays=True)
    for m in range(len(COUNTS)):
        if m in skip:
            continue
        sl = slice(m * rays, (m + 1) * rays)
        fo = f[int(b.face_offsets[m]): int(b.face_offsets[m + 1])].contiguous()
        ref = gpu.trace_rays(b.mesh_nodes(nodes, m).contiguous(), v, fo, org[sl].contiguous(), d[sl].contiguous())
        assert torch.equal(hits[sl], ref), m
    return b.stats()[1]


@pytest.mark.parametrize("rays", [1, 33, 3000])
@pytest.mark.parametrize("meshes", [[7], [1, 4], list(range(8))])
def test_any_order(gpu, rays, meshes):
    v, f, b, t = _batch(gpu)
    g = np.random.default_rng(rays)
    mixed = t.copy()
    for m in meshes:
        a = int(b.node_offsets[m])
        mixed[a: a + 2 * int(COUNTS[m]) - 1] = _permute(t[a: a + 2 * int(COUNTS[m]) - 1], g)
    for nodes in (mixed, t, mixed):  # what one trace met does not stay for the next
        assert _check(gpu, b, v, f, gpu.nodes_from_numpy(nodes), rays) == 0


def test_bad_link(gpu):
    v, f, b, t = _batch(gpu)
    for m, link in ((1, 2 * 700 - 1), (4, 0xFFFFFFF0)):
        at = int(b.node_offsets[m])
        t["left"][at + int(t["left"][at])] = link  # the root's left child, an inner node
        assert t["isLeafFlag"][at + int(t["left"][at])] == 0
    assert _check(gpu, b, v, f, gpu.nodes_from_numpy(t), 3000, skip=(1, 4)) == BAD_INDEX
