"""The tile that a sort picks by its size (2,048 to 8,192 keys, for whole and ragged last tiles): keys and
values against a stable sort; and a few keys, which are placed by counting."""
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


@pytest.mark.parametrize("bytes_", [4, 8])
@pytest.mark.parametrize("bits", [(0, None), (8, 20), (3, 4)])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 255, 500, 1025, 4095, 4096, 4097])
def test_few_keys(gpu, n, bits, bytes_):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    dtype = torch.int32 if bytes_ == 4 else torch.int64
    keys = torch.randint(0, 2 ** 31 - 1, (n,), generator=g, device="cuda", dtype=dtype)
    keys[n // 3:n // 2] = -1  # the highest key
    vals = torch.randint(0, 2 ** 31 - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    k, v = gpu.radix_sort_pairs(keys, vals, *bits)
    end = 8 * bytes_ if bits[1] is None else bits[1]
    digits = (keys.to(torch.int64) & 0xFFFFFFFF if bytes_ == 4 else keys) >> bits[0] & 2 ** min(end - bits[0], 62) - 1
    if bytes_ == 8 and bits[1] is None:
        digits = torch.where(keys < 0, torch.full_like(keys, 2 ** 62), keys)  # read as unsigned
    order = torch.sort(digits, stable=True)[1]
    assert torch.equal(k, keys[order])
    assert torch.equal(v, vals[order])
