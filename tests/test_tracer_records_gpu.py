"""A prepared tracer whose updates leave the rays' records out (it has traced pictures only): rays and bounces
that come all the same see the tree of the last update, in calls and beside replayed captures."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
N = 5000


def _tree(gpu, seed):
    import torch
    vert, faces = scenes.uniform_soup(N, sigma=0.05, seed=seed)
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    return v, f, gpu.LBVH(N, 30).build(v, f)


def _rays_of(gpu, tr, v, f, nodes):
    import torch
    cam = dict(scenes.camera_default(), width=60, height=40)
    org, d = scenes.random_rays(4000, (0,) * 3, (1,) * 3, seed=3)
    img, hits = gpu.trace_image(nodes, v, f, cam)
    for got, ref in ((tr.trace_rays(v, f, org, d), gpu.trace_rays(nodes, v, f, org, d)),
                     (tr.trace_bounce(v, f, cam, hits, seed=5)[0], gpu.trace_bounce(nodes, v, f, cam, hits, seed=5)[0]),
                     (tr.trace_image(v, f, cam)[0], img)):
        assert torch.equal(got, ref)


@pytest.mark.parametrize("pictures", [1, 3])
def test_rays_after_pictures(gpu, pictures):
    tr = gpu.Tracer(2 * N - 1)
    cam = dict(scenes.camera_default(), width=60, height=40)
    for seed in range(pictures + 1):  # the last update is behind a picture: without the rays' records
        v, f, nodes = _tree(gpu, seed)
        tr.update(nodes)
        if seed < pictures:
            tr.trace_image(v, f, cam)
    _rays_of(gpu, tr, v, f, nodes)
    for seed in (20, 21):
        v, f, nodes = _tree(gpu, seed)
        tr.update(nodes)
        _rays_of(gpu, tr, v, f, nodes)


def test_captured_updates(gpu):
    import torch
    (va, f, a), (vb, _, b) = _tree(gpu, 1), _tree(gpu, 2)
    cam = dict(scenes.camera_default(), width=60, height=40)
    held, vert = a.clone(), va.clone()
    tr = gpu.Tracer(2 * N - 1)
    tr.update(held).trace_image(vert, f, cam)
    held.copy_(b), vert.copy_(vb)
    tr.update(held)  # without the rays' records
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        tr.update(held)
        img, _ = tr.trace_image(vert, f, cam)
    _rays_of(gpu, tr, vert, f, held)  # not replayed yet
    held.copy_(a), vert.copy_(va)
    graph.replay()
    _rays_of(gpu, tr, vert, f, held)
    assert torch.equal(img, gpu.trace_image(held, vert, f, cam)[0])
    tr.update(held)
    held.copy_(b), vert.copy_(vb)
    graph.replay()
    _rays_of(gpu, tr, vert, f, held)
