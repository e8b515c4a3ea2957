"""How far the CPU check of the fast decisions pushes the exponential: the whole bound that the renderer checks
on the GPU, (6e-7 + 1.5e-7 |a|) relative at exp(a), its growth with the argument included."""
import math

import pytest

import oracle as O


@pytest.mark.parametrize("a", [0.0, -0.5, -3.0, -10.0, -14.0])
def test_exponential_reaches_the_edge_of_its_bound(a):
    x = a / math.log(2.0)
    import struct
    x = struct.unpack("f", struct.pack("f", x))[0]
    bound = 6e-7 + 1.5e-7 * abs(x) * math.log(2.0)
    for mode, sign in ((1, 1.0), (2, -1.0)):
        rel = O.lib().o2_fast_edge_ex2(x, mode) / 2.0 ** x - 1.0
        assert abs(rel - sign * bound) <= 0.01 * bound + 2.0 ** -24, (a, rel, bound)
