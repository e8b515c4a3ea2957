"""The bins of the sorted path: entries, bin ranges and the region blend at the sizes where they can go
wrong. The image and the sorted order must equal the CPU mirror's bit for bit: splats that cover every bin
beside ones that touch a single pixel, frames that are no multiple of a bin or region, frames of one
pixel and of more than 4 Mpixel (64 x 64 bins), every bin shape, no visible splat at all."""
import numpy as np
import pytest

import oracle as O
from _parity import PKG, lut

pytestmark = pytest.mark.gpu


def scene(n, seed, huge=0, behind=False):
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 16), np.float32)
    s[:, 0:2] = rng.uniform(-2.0, 2.0, (n, 2))
    s[:, 2] = rng.uniform(-6.0, -3.0, n) if behind else rng.uniform(3.0, 9.0, n)
    s[:, 3] = rng.uniform(0.0, 1.0, n)
    s[:, 4:7] = rng.normal(-4.0, 0.8, (n, 3))
    if huge:
        s[:huge, 4:7] = rng.normal(1.0, 0.4, (huge, 3))
        s[:huge, 2] = rng.uniform(2.0, 2.2, huge)
        s[:huge, 3] = 0.05
    s[:, 8:12] = rng.normal(size=(n, 4))
    s[:, 12:15] = rng.uniform(0, 1, (n, 3))
    return s


def check(splats, w, h, **tuning):
    cam = PKG.OracleCamera(focal_x=0.9 * w, focal_y=0.9 * w)
    p = PKG.RenderParams(spp_side=1)
    r = PKG.GpsRenderer(w, h, 1)
    r.set_gaussians(splats)
    if tuning:
        r.set_tuning(**tuning)
    for _ in range(2):  # the second frame reuses the buffers
        r.render_sorted(cam, p, 1)
    acc, (keys, vals) = r.read_accum(), r.read_sorted()
    assert r.debug_error_word() == 0
    r.close()
    oacc, _, okeys, ovals = O.o2_render_sorted(splats, None, 0, lut(), w, h, 1, cam.to_array(), p.to_c())
    assert np.array_equal(keys, okeys) and np.array_equal(vals, ovals)
    assert np.array_equal(acc.view(np.uint32), oacc.view(np.uint32))


@pytest.mark.parametrize("w,h", [(1, 1), (7, 9), (33, 31), (129, 65), (640, 361)])
@pytest.mark.parametrize("n,huge", [(1, 0), (1, 1), (33, 5), (5000, 40)])
def test_frames_and_counts(w, h, n, huge):
    check(scene(n, 7 + n, huge), w, h)


@pytest.mark.parametrize("shape", [(16, 16), (32, 8), (32, 32)])
def test_bin_shapes(shape):
    check(scene(3000, 3, 70), 321, 203, blend_tile_w=shape[0], blend_tile_h=shape[1])


def test_large_frame_uses_large_bins():
    check(scene(2000, 4, 3), 2600, 1700)


def test_no_visible_splat():
    check(scene(700, 5, behind=True), 100, 50)


def test_rank_ties_and_more_splats_than_a_block():
    s = scene(9000, 6, 300)
    s[:, 2] = np.float32(4.0)  # equal depth keys: order by index
    check(s, 200, 120)
