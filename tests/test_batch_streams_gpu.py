"""Batched traces of one workspace on several streams at once, each with trees of its own: every one gives the
hits it gives alone, also where one of them is a replayed capture."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
COUNTS = np.tile(np.array([3000, 700, 1500, 64], np.uint32), 16)
RAYS = 8000


def _trees(gpu, b, seed):
    import torch
    vert = np.concatenate([scenes.uniform_soup(int(n), sigma=0.05, seed=seed + k)[0] for k, n in enumerate(COUNTS)])
    v = torch.from_numpy(vert).cuda()
    f = torch.arange(vert.shape[0], dtype=torch.int32, device="cuda").reshape(-1, 3)
    nodes = b.empty_nodes()
    b.build(v, f, nodes)
    hits = b.trace_random(nodes, v, f, RAYS, seed=seed)
    torch.cuda.synchronize()
    return nodes, v, f, hits


def test_two_streams(gpu):
    import torch
    b = gpu.Batch(COUNTS)
    sets = [_trees(gpu, b, 100), _trees(gpu, b, 300)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    got = []
    for _ in range(12):
        for k, (nodes, v, f, _) in enumerate(sets):
            with torch.cuda.stream(streams[k]):
                got.append((k, b.trace_random(nodes, v, f, RAYS, seed=(100, 300)[k], stream=streams[k])))
    torch.cuda.synchronize()
    assert all(torch.equal(h, sets[k][3]) for k, h in got)
    assert b.stats()[1] == 0


def test_run_beside_a_trace(gpu):
    """The captured pipeline on one stream (its own trees), given trees on another."""
    import torch
    b = gpu.Batch(COUNTS)
    sets = [_trees(gpu, b, 100), _trees(gpu, b, 300)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    nodes, hits = b.empty_nodes(), torch.empty_like(sets[0][3])
    torch.cuda.synchronize()
    got = []
    for _ in range(6):
        b.run(sets[0][1], sets[0][2], nodes, 0, RAYS, hits, seed=100, stream=streams[0])
        with torch.cuda.stream(streams[1]):
            got.append(b.trace_random(*sets[1][:3], RAYS, seed=300, stream=streams[1]))
    torch.cuda.synchronize()
    assert torch.equal(hits, sets[0][3]) and torch.equal(nodes, sets[0][0])
    assert all(torch.equal(h, sets[1][3]) for h in got)


def test_captured_trace(gpu):
    import torch
    b = gpu.Batch(COUNTS)
    sets = [_trees(gpu, b, 100), _trees(gpu, b, 300)]
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        held = b.trace_random(*sets[0][:3], RAYS, seed=100)
    got = []
    for _ in range(6):
        graph.replay()
        with torch.cuda.stream(s):
            got.append(b.trace_random(*sets[1][:3], RAYS, seed=300, stream=s))
    torch.cuda.synchronize()
    assert torch.equal(held, sets[0][3])
    assert all(torch.equal(h, sets[1][3]) for h in got)
