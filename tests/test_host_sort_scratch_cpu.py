"""The scratch of the pair sort (the runtime faked, fake_cudart.cpp): a sort allocates nothing after a sort of
at least as many pairs with as many key bits, as a captured or real-time caller relies on. Small sorts use
smaller, and so more, tiles than large ones."""
import pytest

from _fake_cuda import run


@pytest.mark.parametrize("digit_bits", [4, 6, 8])
def test_a_smaller_sort_allocates_nothing(digit_bits):
    run("""
big, line = 620_000, 600 * 1024
buf = [np.zeros(big, np.uint32) for _ in range(4)]
ptr = [C.c_void_p(b.ctypes.data) for b in buf]
for first in (big, line + 1, line, 100_000):
    r = PKG.GpsRenderer(16, 16, 1)
    r.set_tuning(sort_digit_bits=%d)
    L = PKG.abi.lib()
    assert L.gpsb_sort_pairs(r.handle, *ptr, first, 24) == 0
    before = fake.fake_mallocs()
    for n in (first, first - 1, line, line - 1, 400_000, 2049, 1):
        if n <= first:
            assert L.gpsb_sort_pairs(r.handle, *ptr, n, 24) == 0
            assert fake.fake_mallocs() == before, (first, n)
    r.close()
""" % digit_bits)
