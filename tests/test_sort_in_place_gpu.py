"""Sorting pairs into their own arrays: an even number of passes goes through the scratch arrays first, and one
tile reads everything before it writes."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bytes_,bits", [(4, (0, 32)), (8, (0, 64)), (8, (0, 16)), (4, (8, 32)), (8, (3, 8))])
@pytest.mark.parametrize("n", [1, 2, 100, 1000, 2049, 4096, 4097, 8192, 100000])
@pytest.mark.parametrize("share", ["both", "keys", "values"])
def test_in_place(gpu, n, bytes_, bits, share):
    import torch
    from bvhtest_gb300 import native
    passes = -(-(bits[1] - bits[0]) // 8)
    if passes % 2 and n > 8192:
        return  # an odd number of passes ends in the arrays it starts from: several tiles would meet
    lib = native.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    keys = torch.randint(0, 2 ** 31 - 1, (n,), generator=g, device="cuda", dtype=torch.int32 if bytes_ == 4 else torch.int64)
    vals = torch.randint(0, 2 ** 31 - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    digits = keys.to(torch.int64) >> bits[0] & 2 ** min(bits[1] - bits[0], 62) - 1
    order = torch.sort(digits, stable=True)[1]
    need = C.c_size_t(0)
    assert lib.bvhgb_radix_sort_pairs(None, C.byref(need), None, None, None, None, n, bytes_, *bits, None) == 0
    temp = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    k, v = keys.clone(), vals.clone()
    ko = k if share in ("both", "keys") else torch.empty_like(k)
    vo = v if share in ("both", "values") else torch.empty_like(v)
    p = [C.c_void_p(x.data_ptr()) for x in (temp, k, ko, v, vo)]
    for _ in range(3):
        k.copy_(keys), v.copy_(vals)
        assert lib.bvhgb_radix_sort_pairs(p[0], C.byref(need), p[1], p[2], p[3], p[4], n, bytes_, *bits,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert torch.equal(ko, keys[order]) and torch.equal(vo, vals[order])
