"""Every bin shape that can be set, on frames smaller and larger than a bin and no multiple of one, and the two that
a large frame chooses from, splats of one pixel and splats of many bins: the image and the sorted order
equal the CPU mirror's bit for bit."""
import pytest

from test_gpu_sorted_bins import check, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16), (32, 8), (64, 64), (1, 1)])
@pytest.mark.parametrize("w,h", [(9, 5), (321, 203)])
def test_shapes(shape, w, h):
    check(scene(3000, 3, 70), w, h, blend_tile_w=shape[0], blend_tile_h=shape[1])


@pytest.mark.parametrize("scale", [-6.0, -2.0])
@pytest.mark.parametrize("huge", [0, 9])
def test_large_frames(scale, huge):
    s = scene(4000, 11, huge)
    s[huge:, 4:7] += scale + 4.0
    check(s, 2600, 1700)
