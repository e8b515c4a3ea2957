"""The weight-gradient kernel (gpsb_dn_conv_dw in csrc/conv3x3.cu) and the vectorised element-wise steps of
the backward pass against float64 references, at the edges of their tiles: images narrower than a
16-pixel K-step, of one segment, one pixel more and several segments; fewer rows than a row block;
every pairing of input-group and output-plane instance; a channel slice of a wider tensor; added to what
dw holds. Tolerances: products of bf16 values are exact in fp32, so a sum of K of them accumulated
in fp32 is within K 2^-24 of the sum of the magnitudes; 2^-20 sqrt(K) of it leaves room for any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dn():
    from conftest import load_package
    load_package()
    from gps_pbvr_web_b200 import denoise as dn
    return dn


def _ref_dw(dy, x):
    """dy (B, H, W, co), x (B, H, W, ci) float64 -> (co, 9, ci), and the same of the magnitudes."""
    import torch
    B, H, W, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    out, mag = [], []
    for ky in range(3):
        for kx in range(3):
            s = p[:, ky:ky + H, kx:kx + W]
            out.append(torch.einsum("bhwo,bhwi->oi", dy, s))
            mag.append(torch.einsum("bhwo,bhwi->oi", dy.abs(), s.abs()))
    return torch.stack(out, 1), torch.stack(mag, 1)


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 3, 7), (1, 9, 16), (2, 5, 112), (1, 4, 113), (1, 7, 257)])
@pytest.mark.parametrize("cin,cout", [(8, 32), (8, 40), (8, 128), (16, 8), (32, 3), (40, 64), (96, 32), (64, 128), (192, 64)])
def test_weight_gradient(B, H, W, cin, cout):
    import torch
    dn = _dn()
    g = torch.Generator().manual_seed(1000 * cin + 10 * cout + W)
    coutp, ldx, xoff = (cout + 7) // 8 * 8, cin + 24, 16
    dy = torch.randn(B, H, W, coutp, generator=g)
    dy[..., cout:] = 7.0  # padding channels never reach dw
    x = torch.randn(B, H, W, ldx, generator=g)
    dy, x = dy.to(torch.bfloat16), x.to(torch.bfloat16)
    kp = dn.kp_of(cin)
    dw0 = torch.randn(cout, kp, generator=g)
    dw = dw0.cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dn.conv_dw(dn.to_planar(dy).cuda(), dn.to_planar(x).cuda(), cin, cout, dw, xoff=xoff, err=err)
    ref, mag = _ref_dw(dy.double()[..., :cout], x.double()[..., xoff:xoff + cin])
    got = (dw.cpu().double() - dw0.double())
    tol = mag * 2.0 ** -20 * (B * H * W) ** 0.5 + 2.0 ** -21 * (ref.abs() + dw0.double().abs()[:, :9 * cin].reshape(ref.shape)) + 1e-7
    diff = (got[:, :9 * cin].reshape(cout, 9, cin) - ref).abs()
    assert torch.all(diff <= tol), float((diff / tol).max())
    assert torch.equal(dw.cpu()[:, 9 * cin:], dw0[:, 9 * cin:]) and int(err.item()) == 0


@pytest.mark.parametrize("HW,C,ld", [(1, 3, 8), (255, 32, 32), (2048, 64, 96), (2049, 8, 8), (70_000, 128, 128)])
@pytest.mark.parametrize("shift", [0, 1])
def test_bias_gradient(HW, C, ld, shift):
    import ctypes
    import torch
    dn = _dn()
    B = 3
    g = torch.Generator().manual_seed(HW + C)
    flat = torch.randn(B * ld * HW + 8, generator=g).to(torch.bfloat16)
    dz = flat[shift:shift + B * ld * HW].reshape(B, ld // 8, HW, 8)
    db = torch.ones(C, device="cuda")
    dev = flat.cuda()
    dn._ck(dn._L().gpsb_dn_bias_grad(ctypes.c_void_p(dev.data_ptr() + 2 * shift), ld, B, HW, C, dn._p(db), dn._stream()), "bias")
    v = dz.double().permute(0, 1, 3, 2).reshape(B, ld, HW)[:, :C]
    tol = v.abs().sum((0, 2)) * 2.0 ** -20 + 1e-6
    assert torch.all((db.cpu().double() - 1.0 - v.sum((0, 2))).abs() <= tol)


@pytest.mark.parametrize("h,w,C,off,ld", [(1, 1, 32, 0, 32), (5, 27, 32, 64, 96), (13, 11, 64, 0, 64), (3, 50, 24, 8, 40), (4, 4, 3, 0, 3)])
def test_element_wise_backward(h, w, C, off, ld):
    import torch
    dn = _dn()
    L, st = dn._L(), dn._stream()
    B, H, W = 2, 2 * h, 2 * w
    g = torch.Generator().manual_seed(h * w + C)
    big = torch.randn(B, H, W, ld, generator=g).cuda()
    # ReLU backward into a chunk-planar tensor of ldo >= C channels
    ldo = (C + 7) // 8 * 8
    y = torch.randn(B, H, W, ldo + 8, generator=g).to(torch.bfloat16)
    for mask in (True, False):
        out = torch.full((B, ldo // 8, H, W, 8), 5.0, dtype=torch.bfloat16, device="cuda")
        yp = dn.to_planar(y).cuda()
        dn._ck(L.gpsb_dn_relu_bwd(dn._p(big), ld, off, dn._p(yp) if mask else None, ldo + 8, 8, B, H * W, C, dn._p(out), ldo, st),
               "relu")
        want = torch.zeros(B, H, W, ldo)
        want[..., :C] = big.cpu()[..., off:off + C]
        if mask:
            want[..., :C] *= (y[..., 8:8 + C].float() > 0)
        assert torch.equal(dn.from_planar(out).cpu(), want.to(torch.bfloat16))
    # 2x2 sums and spread averages
    up = torch.zeros(B, h, w, C, device="cuda")
    dn._ck(L.gpsb_dn_up2_bwd(dn._p(big), ld, off, B, h, w, C, dn._p(up), st), "up2_bwd")
    s = big[..., off:off + C]
    assert torch.equal(up, ((s[:, ::2, ::2] + s[:, ::2, 1::2]) + s[:, 1::2, ::2]) + s[:, 1::2, 1::2])
    small = torch.randn(B, h, w, C, generator=g).cuda()
    acc = big.clone()
    dn._ck(L.gpsb_dn_pool2_bwd_add(dn._p(small), B, h, w, C, dn._p(acc), ld, off, st), "pool2_bwd")
    want = big.clone()
    want[..., off:off + C] += 0.25 * small.repeat_interleave(2, 1).repeat_interleave(2, 2)
    assert torch.equal(acc, want)
