"""gpsb_sort_pairs captured into a graph after one larger uncaptured sort: the scratch is large enough for every
smaller one, also across the line between the tile sizes, and the replay equals a stable sort."""
import ctypes as C

import numpy as np
import pytest

from _parity import PKG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [600 * 1024, 400_001, 2048])
def test_replay_after_a_larger_sort(n):
    import torch
    L = PKG.abi.lib()
    stream = torch.cuda.Stream()
    r = PKG.GpsRenderer(16, 16, 1)
    r.set_stream(stream.cuda_stream)
    buf = [torch.zeros(700_000, dtype=torch.int32, device="cuda") for _ in range(4)]
    ptr = [C.c_void_p(b.data_ptr()) for b in buf]
    torch.cuda.synchronize()
    assert L.gpsb_sort_pairs(r.handle, *ptr, 700_000, 24) == 0
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        assert L.gpsb_sort_pairs(r.handle, *ptr, n, 24) == 0
    for seed in (1, 2):
        keys = np.random.default_rng(seed).integers(0, 1 << 24, n, dtype=np.uint32)
        with torch.cuda.stream(stream):
            buf[0][:n].copy_(torch.from_numpy(keys.view(np.int32)))
            buf[1][:n].copy_(torch.arange(n, dtype=torch.int32))
            graph.replay()
        stream.synchronize()
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(buf[2][:n].cpu().numpy().view(np.uint32), keys[order])
        assert np.array_equal(buf[3][:n].cpu().numpy(), order.astype(np.int32))
    assert r.debug_error_word() == 0
    del graph
    r.close()
