"""The Morton phase repeated on one scene box: the cells it samples are counted afresh each time, so the sort
takes the route that the keys call for, in calls and in the replays of a capture."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REPEATS = 45  # an uncleared sample of even keys would take 20 of them for a full cell
SIZES = [20000, 1100000]


def _mesh(n, cell):
    """Triangles at points; 'cell' of them in one cell of the keys' upper bits, none of those sampled."""
    import torch
    g = np.random.default_rng(n + cell)
    p = g.random((n, 3))
    at = np.flatnonzero(np.arange(n) % 16 != 0)[:cell]
    p[at] = 0.3001 + 1e-4 * g.random((len(at), 3))
    v = torch.from_numpy(np.repeat(p[:, None], 3, 1).reshape(-1, 3).astype(np.float32)).cuda()
    return v, torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(-1, 3)


def _fixed_box(b):
    from bvhtest_gb300.native import Aabb
    box = Aabb()
    box.mn[:], box.mx[:] = (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)
    import torch
    assert b.lib.bvhgb_lbvh_set_scene_box(b.ws, C.byref(box), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0


def _ordered(b, n):
    keys, _ = b.keys(n, False)
    k, i = b.keys(n, True)
    order = np.argsort(keys, kind="stable")
    return np.array_equal(k, keys[order]) and np.array_equal(i, order.astype(np.uint32))


@pytest.mark.parametrize("n", SIZES)
def test_repeated_phase(gpu, n):
    b = gpu.LBVH(n, 63, "karras")
    _fixed_box(b)
    v, f = _mesh(n, 0)
    for _ in range(REPEATS):
        b.calc_morton(v, f)
        b.sort(n)
        assert b.sort_route() == 0
    assert _ordered(b, n)
    b.calc_morton(*_mesh(n, 400))  # one group of 400, not sampled
    b.sort(n)
    assert b.sort_route() == 1 and _ordered(b, n)
    full = _mesh(n, n // 4)
    full[0].copy_(full[0].roll(3, 0))  # now sampled
    for _ in range(2):
        b.calc_morton(*full)
        b.calc_morton(*full)
        b.sort(n)
        assert b.sort_route() == 2 and _ordered(b, n)
    b.calc_morton(v, f)
    b.sort(n)
    assert b.sort_route() == 0 and _ordered(b, n)
    b.build(v, f)
    assert b.sort_route() == 0


@pytest.mark.parametrize("n", SIZES)
def test_replayed_phase(gpu, n):
    import torch
    b = gpu.LBVH(n, 63, "karras")
    v, f = _mesh(n, 0)
    b.build(v, f)  # before the capture: what is looked up once
    b.init_tri_data(v, f)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        b.calc_morton(v, f)
        b.sort(n)
    for _ in range(REPEATS):
        graph.replay()
    torch.cuda.synchronize()
    assert b.sort_route() == 0 and _ordered(b, n)
    b.calc_morton(v, f)
    b.sort(n)
    assert b.sort_route() == 0 and _ordered(b, n)
