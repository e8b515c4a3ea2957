"""The count scan on both sides of the line between its two forms (240 tiles of 2048 splats, counted over the
batch's ensembles): counts, statistics and image equal the CPU mirror's."""
import pytest

from _parity import PKG
from test_gpu_fast_flat import M, assert_bit_exact, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ens", [(239 * 2048, 1), (239 * 2048 + 1, 1), (75_000, 6), (75_000, 7)])
def test_both_forms(n, ens):
    s = scene(n, n, -6.0, lambda r, k: r.uniform(0.0, 1.0, k))
    s[: 1 + n // 5000, 4:7] = -2.0  # large means
    cam = PKG.OrbitCamera(distance=5.0).to_camera(160, 90)
    for method in (M.Gps, M.Extinction):
        assert_bit_exact(s, None, 0, 160, 90, 1, cam, PKG.RenderParams(spp_side=1, method=method, max_points_per_splat=500),
                         first_seed=5, count=ens)
