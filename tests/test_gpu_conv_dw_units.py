"""The weight-gradient kernel where a block works through dozens of units: both stages reused with either phase,
the accumulators read back and started afresh several times, the last run of units full, short, or the only
one. Every instance of the kernel, against float64. A block sums at most 168 K-steps in the tensor core,
each of which may drop up to 2^-23 of what it adds to, then adds one fp32 value per read-back, and its sum is
added to dw: the sum of the magnitudes times (2 * 168 + read-backs + blocks) 2^-24 bounds the error. A lost
read-back would be off by hundreds of times that."""
import pytest

from test_gpu_conv_dw import _dn, _ref_dw

pytestmark = pytest.mark.gpu

# cin, cout, rows of a unit
INSTANCES = [(8, 32, 8), (8, 64, 4), (8, 128, 2), (192, 32, 4), (192, 64, 4), (96, 128, 2)]


@pytest.mark.parametrize("cin,cout,rows", INSTANCES)
@pytest.mark.parametrize("runs,extra", [(1, False), (2, False), (2, True)])
def test_many_units_a_block(cin, cout, rows, runs, extra):
    import torch
    dn = _dn()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = max(sms // ((cin + 31) // 32), 1)  # of one group of input channels
    flush = 24 // rows  # units between read-backs
    units = blocks * runs * flush + (blocks // 2 if extra else 0)
    B, W = 2, 14 if extra else 16
    units += units % B
    H = units // B * rows - (1 if extra else 0)  # a ragged last row block
    g = torch.Generator(device="cuda").manual_seed(cin + cout + runs)
    dy = torch.randn(B, H, W, cout, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(B, H, W, cin, generator=g, device="cuda").to(torch.bfloat16)
    kp = dn.kp_of(cin)
    dw = torch.zeros(cout, kp, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dn.conv_dw(dn.to_planar(dy), dn.to_planar(x), cin, cout, dw, err=err)
    ref, mag = _ref_dw(dy.double(), x.double())
    tol = mag * (2 * 168 + runs + 1 + blocks) * 2.0 ** -24 + 1e-6
    diff = (dw[:, :9 * cin].double().reshape(cout, 9, cin) - ref).abs()
    assert torch.all(diff <= tol), float((diff / tol).max())
    assert int(err.item()) == 0
