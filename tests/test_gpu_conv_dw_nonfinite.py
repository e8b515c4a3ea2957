"""An infinity or NaN of the layer's input at the image's last column or row stays in the taps that read it: the
pixels past the edge, which the kernel's K-steps and row blocks include, contribute nothing, not 0 x inf.
Widths that are and are not multiples of 16, of one K-step, of one pixel, of several segments; heights that
are and are not multiples of a row block. Finite sums as in the other tests."""
import pytest

from test_gpu_conv_dw import _dn, _ref_dw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(1, 1), (3, 7), (8, 16), (5, 16), (8, 17), (9, 33), (7, 112), (6, 113), (7, 250)])
@pytest.mark.parametrize("cin,cout", [(8, 32), (8, 64), (8, 128), (40, 32), (32, 64), (64, 128)])
def test_edges(H, W, cin, cout):
    import torch
    dn = _dn()
    B = 2
    g = torch.Generator(device="cuda").manual_seed(H * W + cin)
    dy = torch.randn(B, H, W, cout, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(B, H, W, cin, generator=g, device="cuda").to(torch.bfloat16)
    x[0, H - 1, W - 1, 1] = float("inf")
    x[1, H - 1, 0, 3] = float("nan")
    x[0, 0, W - 1, 4] = float("-inf")
    kp = dn.kp_of(cin)
    dw = torch.zeros(cout, kp, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dn.conv_dw(dn.to_planar(dy), dn.to_planar(x), cin, cout, dw, err=err)
    ref, mag = _ref_dw(dy.double(), x.double())
    got = dw[:, :9 * cin].double().reshape(cout, 9, cin)
    ok = ref.isfinite()
    assert torch.equal(got.isfinite(), ok), int((got.isfinite() != ok).sum())
    assert torch.all((got[ok] - ref[ok]).abs() <= mag[ok] * 2.0 ** -20 * (B * H * W) ** 0.5 + 1e-6)
    assert int(err.item()) == 0
