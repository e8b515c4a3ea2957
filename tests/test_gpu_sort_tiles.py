"""Radix sort at the sizes where its tiles can go wrong: one pair, a tile minus, plus and exactly its size
(2048 pairs for small sorts, 6912 and 3840 for large ones), both sides of the line between the two, a ragged last
tile, arrays that start off a 16-byte boundary, equal and sorted keys, every digit width. The
permutation must equal a stable sort's."""
import ctypes as C

import numpy as np
import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu

LINE = 600 * 1024


def sort(keys, key_bits, digit_bits, skew, noalloc):
    import torch

    n = len(keys)
    vals = np.random.default_rng(n).integers(0, 2**32, n, dtype=np.uint32)
    buf = [torch.zeros(n + 8, dtype=torch.int32, device="cuda") for _ in range(4)]
    view = [b[skew:skew + n] for b in buf]
    view[0].copy_(torch.from_numpy(keys.view(np.int32).copy()))
    view[1].copy_(torch.from_numpy(vals.view(np.int32).copy()))
    ptr = [C.c_void_p(v.data_ptr()) for v in view]
    torch.cuda.synchronize()
    L = PKG.abi.lib()
    if noalloc:
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        st = torch.cuda.current_stream()
        assert L.gpsb_sort_pairs_noalloc(*ptr, n, key_bits, C.c_void_p(st.cuda_stream), C.c_void_p(err.data_ptr())) == 0
        torch.cuda.synchronize()
        assert int(err.item()) == 0
    else:
        r = PKG.GpsRenderer(16, 16, 1)
        r.set_tuning(sort_digit_bits=digit_bits)
        assert L.gpsb_sort_pairs(r.handle, *ptr, n, key_bits) == 0
        r.wait_idle()
        assert r.debug_error_word() == 0
        r.close()
    order = np.argsort(keys, kind="stable")
    got = [v.cpu().numpy().view(np.uint32) for v in view[2:]]
    assert np.array_equal(got[0], keys[order])
    assert np.array_equal(got[1], vals[order])
    for b in buf[2:]:  # nothing written outside the outputs
        assert not b[:skew].any() and not b[skew + n:].any()


@pytest.mark.parametrize("digit_bits", [4, 6, 8])
@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 6913, LINE, LINE + 1, 90 * 6912, 90 * 6912 + 6911, 170 * 3840 + 1])
def test_sort_at_the_edges_of_its_tiles(n, digit_bits):
    keys = np.random.default_rng(n).integers(0, 1 << 24, n, dtype=np.uint32)
    sort(keys, 24, digit_bits, n % 4, False)


@pytest.mark.parametrize("n", [3, 2049, LINE, LINE + 1, 1 << 21])
@pytest.mark.parametrize("key_bits", [5, 32])
def test_sort_without_allocation_at_both_tile_sizes(n, key_bits):
    keys = np.random.default_rng(n).integers(0, 1 << key_bits, n, dtype=np.uint64).astype(np.uint32)
    sort(keys, key_bits, 8, 1, True)


@pytest.mark.parametrize("kind", ["equal", "sorted", "reversed", "two"])
def test_sort_of_keys_that_share_digits(kind):
    for n in (LINE - 5, 700_001):
        i = np.arange(n, dtype=np.uint32)
        keys = {"equal": i * 0 + 0xABCDEF, "sorted": i, "reversed": n - i, "two": (i & 1) * 0xFFFFFF}[kind].astype(np.uint32)
        sort(keys, 24, 8, 0, False)
