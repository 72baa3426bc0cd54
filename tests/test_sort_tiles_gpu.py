"""The tile that a sort picks by its size (2,048 to 8,192 keys, for whole and ragged last tiles): keys and
values against a stable sort."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bytes_", [4, 8])
@pytest.mark.parametrize("n", [262144, 262145, 524289, 700001, 1048576, 1500001, 2490368, 3500000, 4194305, 8388608, 8388609])
def test_stable_order(gpu, n, bytes_):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    top = 2 ** 31 - 1 if bytes_ == 4 else 2 ** 62
    keys = torch.randint(0, top, (n,), generator=g, device="cuda", dtype=torch.int32 if bytes_ == 4 else torch.int64)
    keys[n // 3:n // 2] = keys[0]  # many equal keys, whose order is the input's
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    k, v = gpu.radix_sort_pairs(keys, vals)
    ref, order = torch.sort(keys, stable=True)
    assert torch.equal(k, ref)
    assert torch.equal(v, order.to(torch.int32))
