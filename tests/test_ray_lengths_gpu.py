"""Rays whose directions are not normalised: a prepared tracer gives the closest of all triangles (the oracle
tests every one) for every length of the direction, for components that are small beside the others, and from
origins that are far away for the size of the scene; and so the hits of the node array."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(gpu, scale=1.0, offset=0.0):
    import torch
    vert, faces = scenes.uniform_soup(3000, sigma=0.05, seed=71)
    vert = ((vert + np.float32(offset)) * np.float32(scale)).astype(np.float32)
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    return vert, faces, v, f, gpu.LBVH(3000, 30, "refCompat").build(v, f)


def _same(got, ref):
    assert np.array_equal(got["prim"], ref["prim"])
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))


def _hits(gpu, orc, org, d, least, **scene):
    vert, faces, v, f, nodes = _scene(gpu, **scene)
    tr = gpu.Tracer(nodes.shape[0]).update(nodes)
    got = gpu.hits_to_numpy(tr.trace_rays(v, f, org, d))
    ref = orc.trace_brute(org, d, vert, faces)
    assert (ref["prim"] != 0xFFFFFFFF).mean() >= least
    _same(got, ref)
    # the node array drops boxes where a component other than 0 has an infinite reciprocal
    if not ((d != 0) & (np.abs(d) < 3e-39)).any():
        _same(got, gpu.hits_to_numpy(gpu.trace_rays(nodes, v, f, org, d)))
    assert gpu.trace_errors() == 0
    tr.close()


def _directions(g, n):
    """Along an axis, in the plane of two, oblique, and with a component far below the largest."""
    d = g.normal(size=(n, 3))
    d /= np.abs(d).max(1, keepdims=True)
    k = g.integers(0, 3, n)
    d[: n // 4] = np.eye(3)[k[: n // 4]] * g.choice([-1.0, 1.0], (n // 4, 1))
    d[np.arange(n // 4, n // 2), k[n // 4: n // 2]] = g.choice([0.0, -0.0], n // 2 - n // 4)
    j = np.arange(n // 2, 3 * n // 4)
    d[j, k[j]] *= 10.0 ** g.uniform(-30, -1, j.size)
    return d


@pytest.mark.parametrize("length", [1e-37, 1e-30, 1e-25, 1e-24, 1e-22, 1e-12, 1.0, 1e12, 1e30])
def test_length(gpu, orc, length):
    g = np.random.default_rng(5)
    n = 6000
    org = g.uniform(0, 1, (n, 3)).astype(np.float32)
    org[::2] -= np.float32(5.0) * np.sign(org[::2] - 0.5)
    d = _directions(g, n)
    d[::2] = np.where(np.abs(d[::2]) > 0, np.abs(d[::2]), d[::2]) * np.sign(0.5 - org[::2])  # towards the scene
    org[: n // 4] = g.uniform(0, 1, (n // 4, 3))  # along an axis: from within, and from beside the scene
    k = np.abs(d[: n // 4]).argmax(1)
    org[np.arange(n // 4), k] -= np.float32(4.0) * np.sign(d[np.arange(n // 4), k]).astype(np.float32)
    _hits(gpu, orc, org, (d * length).astype(np.float32), 0.2)


@pytest.mark.parametrize("distance", [1e3, 1e9, 1e15, 1e24])
@pytest.mark.parametrize("length", [1e-24, 1.0])
def test_far_origins(gpu, orc, distance, length):
    """Along an axis, so that the other coordinates stay exact."""
    g = np.random.default_rng(6)
    n = 2000
    org = g.uniform(0, 1, (n, 3)).astype(np.float32)
    k, s = g.integers(0, 3, n), g.choice(np.float32([-1, 1]), n)
    d = np.zeros((n, 3), np.float32)
    d[np.arange(n), k] = s * np.float32(length)
    org[np.arange(n), k] = -s * np.float32(distance)
    _hits(gpu, orc, org, d, 0.2 if distance / length < 1e38 else 0.0)


def test_no_direction(gpu, orc):
    """A direction of zeros hits nothing."""
    g = np.random.default_rng(7)
    org = g.uniform(0, 1, (1000, 3)).astype(np.float32)
    d = g.normal(size=(1000, 3)).astype(np.float32)
    d[::3] = 0.0
    d[1::6] = -0.0
    _hits(gpu, orc, org, d, 0.1)


@pytest.mark.parametrize("scale,offset", [(1e-18, 0.0), (1e-3, 0.0), (1e9, 0.0), (1e12, 0.0), (1.0, 1000.0), (1e-6, 5e5)])
@pytest.mark.parametrize("length", [1e-20, 1.0, 1e20])
def test_scenes_of_every_size(gpu, orc, scale, offset, length):
    """Every kind of direction in scenes of every size, at the origin and far from it."""
    g = np.random.default_rng(8)
    n = 3000
    org = ((g.uniform(-0.5, 1.5, (n, 3)) + offset) * scale).astype(np.float32)
    d = (_directions(g, n) * length).astype(np.float32)
    _hits(gpu, orc, org, d, 0.05 if scale >= 1e-6 else 0.0, scale=scale, offset=offset)
