"""The prepared tracer's four-wide traversal (bounce and given rays) gives the hits of the binary
traversal on the node array, bit for bit, where it can go wrong: the smallest trees, every remainder
of its runs of rays, leaves of several faces, flat and far-away boxes, rays along the axes and in
the planes of the boxes, distances below zero, and boxes that are on no finite grid."""
import numpy as np
import pytest

from bvhtest_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _scene(gpu, vert, faces, bits=30, topology="refCompat"):
    import torch
    v = torch.from_numpy(np.ascontiguousarray(vert, np.float32)).cuda()
    f = torch.from_numpy(np.ascontiguousarray(faces, np.uint32).view(np.int32)).cuda()
    b = gpu.LBVH(f.shape[0], bits, topology)
    nodes = b.build(v, f)
    return v, f, nodes, b


def _same(gpu, v, f, nodes, org, d, tmin=0.0, tmax=float("inf"), cull=False):
    import torch
    tr = gpu.Tracer(nodes.shape[0]).update(nodes)
    got = gpu.hits_to_numpy(tr.trace_rays(v, f, org, d, tmin=tmin, tmax=tmax, face_culling=cull))
    ref = gpu.hits_to_numpy(gpu.trace_rays(nodes, v, f, org, d, tmin=tmin, tmax=tmax, face_culling=cull))
    torch.cuda.synchronize()
    assert np.array_equal(got["prim"], ref["prim"])
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    assert gpu.trace_errors() == 0
    tr.close()
    return ref


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 100, 1000, 20001])
@pytest.mark.parametrize("rays", [1, 31, 33, 127, 129, 4097])
def test_sizes(gpu, n, rays):
    vert, faces = scenes.uniform_soup(n, sigma=0.2 / n ** (1 / 3), seed=n)
    v, f, nodes, _ = _scene(gpu, vert, faces)
    org, d = scenes.random_rays(rays, (-0.2,) * 3, (1.2,) * 3, seed=n + rays)
    _same(gpu, v, f, nodes, org, d)


def test_runs_are_stolen(gpu):
    """More runs than the chip holds warps."""
    vert, faces = scenes.uniform_soup(50000, sigma=0.01, seed=3)
    v, f, nodes, _ = _scene(gpu, vert, faces, 63, "karras")
    org, d = scenes.random_rays(1500017, (0,) * 3, (1,) * 3, seed=4)
    ref = _same(gpu, v, f, nodes, org, d)
    assert (ref["prim"] != 0xFFFFFFFF).mean() > 0.2


@pytest.mark.parametrize("tmin,tmax,cull", [(0.0, 0.3, False), (0.2, float("inf"), False), (-0.5, float("inf"), False),
                                            (-0.4, -0.1, False), (0.0, float("inf"), True)])
def test_ranges(gpu, tmin, tmax, cull):
    vert, faces = scenes.uniform_soup(5000, sigma=0.05, seed=8)
    v, f, nodes, _ = _scene(gpu, vert, faces)
    org, d = scenes.random_rays(20000, (0,) * 3, (1,) * 3, seed=9)
    ref = _same(gpu, v, f, nodes, org, d, tmin, tmax, cull)
    assert 0.05 < (ref["prim"] != 0xFFFFFFFF).mean() < 1.0


def test_axes_and_planes(gpu):
    """A grid of axis-aligned squares: flat boxes, rays along the axes, rays in the grid's own plane."""
    grid = scenes.ground_grid(24, 3.0).reshape(-1, 3)
    vert = np.concatenate([grid, grid[:, [1, 0, 2]] + np.float32([1.5, 0, 0]), grid[:, [0, 2, 1]]])
    faces = np.arange(vert.shape[0], dtype=np.uint32).reshape(-1, 3)
    v, f, nodes, _ = _scene(gpu, vert, faces, 63, "karras")
    g = np.random.default_rng(5)
    org = g.uniform(-1, 4, (30000, 3)).astype(np.float32)
    org[::3] = np.round(org[::3] * 8) / 8  # on the grid's lines and planes
    d = np.eye(3, dtype=np.float32)[g.integers(0, 3, 30000)] * g.choice(np.float32([-1, 1]), (30000, 1))
    two = g.normal(size=(10000, 3)).astype(np.float32)
    two[np.arange(10000), g.integers(0, 3, 10000)] = g.choice(np.float32([0.0, -0.0, 1e-30, -1e-42]), 10000)
    d[20000:] = two
    _same(gpu, v, f, nodes, org, d)


@pytest.mark.parametrize("offset,scale", [(0.0, 1.0), (1000.0, 1.0), (0.0, 1e-12), (0.0, 1e12), (3e6, 1.0)])
def test_magnitudes(gpu, offset, scale):
    """Boxes far from the origin for their size, and very small and large scenes."""
    vert, faces = scenes.uniform_soup(4000, sigma=0.05, seed=12)
    vert = ((vert + np.float32(offset)) * np.float32(scale)).astype(np.float32)
    v, f, nodes, _ = _scene(gpu, vert, faces)
    org, d = scenes.random_rays(8000, vert.min(0), vert.max(0), seed=13)
    far = org.copy()
    far[::2] -= d[::2] * np.float32(50.0 * scale)
    _same(gpu, v, f, nodes, far, d)


def test_leaves_of_several_faces(gpu):
    """Leaves of two faces (imported trees have them), among leaves of one and of none."""
    import torch
    n = 6000
    vert, faces = scenes.uniform_soup(n, sigma=0.05, seed=21)
    v, f, nodes, b = _scene(gpu, vert, faces)
    _, idx = b.keys(n, True)
    faces = faces[idx]  # sorted order is face order: leaf i is face i
    v, f, nodes, _ = _scene(gpu, vert, faces)
    t = gpu.nodes_to_numpy(nodes).copy()
    inner = np.flatnonzero(t["isLeafFlag"] == 0)
    l, r = t["left"][inner], t["right"][inner]
    both = (t["isLeafFlag"][l] == 1) & (t["isLeafFlag"][r] == 1)
    fl, fr = t["left"][l], t["left"][r]
    pick = inner[both & (fr == fl + 1)][::2]
    first = t["left"][t["left"][pick]]
    assert len(pick) > 300
    t["left"][pick], t["right"][pick], t["isLeafFlag"][pick] = first, 2, 1
    leaf = np.flatnonzero((t["isLeafFlag"] == 1) & (t["right"] == 1))
    t["right"][leaf[::50]] = 0
    nodes = gpu.nodes_from_numpy(t)
    org, d = scenes.random_rays(20000, (0,) * 3, (1,) * 3, seed=22)
    ref = _same(gpu, v, f, nodes, org, d)
    assert (ref["prim"] != 0xFFFFFFFF).any()


def test_boxes_on_no_grid(gpu):
    """A vertex at infinity makes the boxes above it infinite: they pass, and the finite ones still work."""
    vert, faces = scenes.uniform_soup(2000, sigma=0.05, seed=31)
    v, f, nodes, _ = _scene(gpu, vert, faces)
    t = gpu.nodes_to_numpy(nodes).copy()
    x = int(np.flatnonzero((t["isLeafFlag"] == 1))[700])
    for _ in range(64):  # the leaf's box and all above it
        t["mx"][x, 1] = np.inf
        if x == int(t["parent"][x]) or x == 0:
            break
        x = int(t["parent"][x])
    nodes = gpu.nodes_from_numpy(t)
    org, d = scenes.random_rays(5000, (0,) * 3, (1,) * 3, seed=32)
    _same(gpu, v, f, nodes, org, d)


@pytest.mark.parametrize("width,height", [(1, 1), (7, 3), (8, 4), (33, 17), (250, 131)])
def test_bounce(gpu, width, height):
    import torch
    vert, faces = scenes.uniform_soup(3000, sigma=0.08, seed=41)
    v, f, nodes, _ = _scene(gpu, vert, faces)
    cam = dict(scenes.camera_default(), width=width, height=height)
    tr = gpu.Tracer(nodes.shape[0]).update(nodes)
    _, hits = gpu.trace_image(nodes, v, f, cam)
    a, ao, ad = gpu.trace_bounce(nodes, v, f, cam, hits, seed=5, with_rays=True)
    b, bo, bd = tr.trace_bounce(v, f, cam, hits, seed=5, with_rays=True)
    c, _, _ = tr.trace_bounce(v, f, cam, hits, seed=5)
    torch.cuda.synchronize()
    assert torch.equal(a, b) and torch.equal(a, c)
    assert torch.equal(ao.view(torch.int32), bo.view(torch.int32)) and torch.equal(ad.view(torch.int32), bd.view(torch.int32))
    assert gpu.trace_errors() == 0


@pytest.mark.parametrize("rays", [1, 33, 500, 5000])
def test_batch(gpu, rays):
    """Meshes of 1, 2, 3 and more triangles in one launch, below and above the rule's line (a ray per
    eight inner nodes), against the single-mesh traversal on the node array."""
    import torch
    counts = np.array([1, 700, 2, 3, 5000, 64], np.uint32)
    parts = [scenes.uniform_soup(int(n), sigma=0.05, seed=60 + k)[0] for k, n in enumerate(counts)]
    vert = np.concatenate(parts)
    faces = np.arange(vert.shape[0], dtype=np.uint32).reshape(-1, 3)
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    b = gpu.Batch(counts)
    nodes = b.empty_nodes()
    b.build(v, f, nodes)
    b.optimize(nodes, 2)
    hits, org, d = b.trace_random(nodes, v, f, rays, seed=9, with_rays=True)
    for m in range(len(counts)):
        sl = slice(m * rays, (m + 1) * rays)
        fo = f[int(b.face_offsets[m]): int(b.face_offsets[m + 1])].contiguous()
        ref = gpu.trace_rays(b.mesh_nodes(nodes, m).contiguous(), v, fo, org[sl].contiguous(), d[sl].contiguous())
        assert torch.equal(hits[sl], ref), m
    assert b.stats()[1] == 0


def test_without_memory_for_the_records(gpu):
    """No memory for the wide records: the tracer is made all the same and traces on the node array."""
    import ctypes as C

    import torch
    from bvhtest_gb300 import native
    lib = native.load()
    vert, faces = scenes.uniform_soup(2000, sigma=0.05, seed=51)
    v, f, nodes, _ = _scene(gpu, vert, faces)
    org, d = scenes.random_rays(3000, (0,) * 3, (1,) * 3, seed=52)
    assert lib.bvhgb_debug_fail_allocations(1, None) == 0
    tr = gpu.Tracer(nodes.shape[0])
    assert lib.bvhgb_debug_fail_allocations(C.c_int64(-1), None) == 0
    tr.update(nodes)
    cam = dict(scenes.camera_default(), width=40, height=30)
    _, hits = tr.trace_image(v, f, cam)
    assert torch.equal(tr.trace_rays(v, f, org, d), gpu.trace_rays(nodes, v, f, org, d))
    assert torch.equal(tr.trace_bounce(v, f, cam, hits)[0], gpu.trace_bounce(nodes, v, f, cam, hits)[0])
