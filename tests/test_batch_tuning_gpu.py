"""The batched autotuner tries the tracer's block where the rays use it: on the node arrays (few rays). On
the records it stays as configured."""
import numpy as np
import pytest

from bvhtest_gb300 import scenes

pytestmark = pytest.mark.gpu
COUNTS = np.array([900, 2000, 40], np.uint32)


@pytest.mark.parametrize("rays,records", [(50, False), (500, True)])
def test_trace_block(gpu, rays, records):
    import torch
    vert = np.concatenate([scenes.uniform_soup(int(n), sigma=0.05, seed=k)[0] for k, n in enumerate(COUNTS)])
    v = torch.from_numpy(vert).cuda()
    f = torch.arange(vert.shape[0], dtype=torch.int32, device="cuda").reshape(-1, 3)
    b = gpu.Batch(COUNTS)
    b.set_config(traceBlock=192)
    nodes = b.empty_nodes()
    hits = torch.zeros(len(COUNTS) * rays, dtype=torch.int64, device="cuda")
    rep = b.autotune(v, f, nodes, rays, hits, seed=3)
    assert sorted(rep["trace_block"]) == [64, 128, 256]
    assert all((t == 0) == records for t in rep["trace_block"].values())
    assert (rep["chosen"]["traceBlock"] == 192) == records
    assert torch.equal(hits, b.trace_random(nodes, v, f, rays, seed=3))
