"""Backward kernels called on nothing (the runtime faked, fake_cudart.cpp): an empty batch, image or sample set is
refused, as the launch of an empty grid is, and no kernel runs; no channels to sum is no error."""
from _fake_cuda import run


def test_empty_inputs_are_refused():
    run("""
L = PKG.abi.lib()
buf = np.zeros(1 << 16, np.float32)
p = C.c_void_p((buf.ctypes.data + 255) & ~255)
E = C.c_void_p(0)
full = {
    "conv_dw": lambda B=1, H=4, W=16, cin=32: L.gpsb_dn_conv_dw(p, 32, p, 32, 0, cin, B, H, W, 32, 320, p, E, p),
    "l1": lambda B=1, H=4, W=16: L.gpsb_dn_l1(p, p, p, B * H * W, p, p, 1.0, E),
    "bias_grad": lambda B=1, H=4, W=16: L.gpsb_dn_bias_grad(p, 32, B, H * W, 32, p, E),
    "relu_bwd": lambda B=1, H=4, W=16: L.gpsb_dn_relu_bwd(p, 32, 0, p, 32, 0, B, H * W, 32, p, 32, E),
    "up2_bwd": lambda B=1, H=4, W=16: L.gpsb_dn_up2_bwd(p, 32, 0, B, H, W, 32, p, E),
    "pool2_bwd_add": lambda B=1, H=4, W=16: L.gpsb_dn_pool2_bwd_add(p, B, H, W, 32, p, 32, 0, E),
}
for name, call in full.items():
    fake.fake_clear()
    assert call() == 0 and fake.fake_launches() == 1, name
    for k in ("B", "H", "W"):
        fake.fake_clear()
        assert call(**{k: 0}) != 0 and fake.fake_launches() == 0, (name, k)
assert full["conv_dw"](cin=0) != 0
assert L.gpsb_dn_bias_grad(p, 32, 1, 64, 0, p, E) == 0
""")
