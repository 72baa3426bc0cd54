"""A workspace made while the default stream is busy is ready for a non-blocking stream at once."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [1000, 50000])
def test_build_beside_a_busy_default_stream(gpu, n, bits):
    import torch
    vert, faces = scenes.uniform_soup(n, seed=n)
    v = torch.from_numpy(vert).cuda()
    f = torch.from_numpy(faces.view(np.int32)).cuda()
    ref = gpu.LBVH(n, bits, "karras")
    expected, box = ref.build(v, f), ref.scene_box()
    nodes, side = torch.empty_like(expected), torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # a tenth of a second on the default stream
    busy = torch.cuda.Event()
    busy.record()
    b = gpu.LBVH(n, bits, "karras")
    b.build(v, f, nodes, stream=side)
    side.synchronize()
    assert not busy.query()
    torch.cuda.synchronize()
    assert np.array_equal(b.scene_box(stream=side), box)
    assert torch.equal(nodes, expected) and b.errors(stream=side) == 0


def test_calls_before_any_build(gpu):
    """A new workspace has an empty box and no errors, whatever its memory held."""
    import torch
    junk = [torch.full((64,), -1, dtype=torch.int32, device="cuda") for _ in range(2000)]
    del junk
    torch.cuda.empty_cache()
    for _ in range(20):
        b = gpu.LBVH(5000, 63, "karras")
        assert b.errors() == 0 and b.sort_route() == 0
        b.close()
