"""Adam over a set of tensors in one launch equals the one-tensor call bit for bit: more tensors than one launch
holds, sizes around a block, an empty tensor, one larger than the grid covers at once."""
import ctypes as C

import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [0, 255, 256, 257], [200_000, 3, 592 * 256 + 1], [7 + i for i in range(33)]])
def test_adam_set_equals_adam(sizes):
    import torch

    dn = PKG.denoise if hasattr(PKG, "denoise") else __import__("importlib").import_module("gps-pbvr-web_b200.denoise")
    L = PKG.abi.lib()
    g = torch.Generator().manual_seed(len(sizes))
    one, many = [], []
    for n in sizes:
        t = [torch.randn(n, generator=g), torch.randn(n, generator=g), torch.randn(n, generator=g), torch.rand(n, generator=g)]
        one.append([x.cuda() for x in t])
        many.append([x.cuda() for x in t])
    ptr = C.c_void_p * len(sizes)
    w, gr, m, v = (ptr(*[t[k].data_ptr() for t in many]) for k in range(4))
    for t in (1, 2, 50):
        for x in one:
            if x[0].numel():
                assert L.gpsb_dn_adam(*[C.c_void_p(y.data_ptr()) for y in x], x[0].numel(), 1e-3, 0.9, 0.999, 1e-8, t, None, dn._stream()) == 0
        assert L.gpsb_dn_adam_set(len(sizes), w, gr, m, v, (C.c_int * len(sizes))(*sizes), 1e-3, 0.9, 0.999, 1e-8, t, dn._stream()) == 0
    torch.cuda.synchronize()
    for a, b in zip(one, many):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_adam_set_of_nothing():
    assert PKG.abi.lib().gpsb_dn_adam_set(0, None, None, None, None, None, 1e-3, 0.9, 0.999, 1e-8, 1, None) == 0
    assert PKG.abi.lib().gpsb_dn_adam_set(2, None, None, None, None, None, 1e-3, 0.9, 0.999, 1e-8, 1, None) != 0
