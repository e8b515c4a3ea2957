"""What a user of this renderer has it do, as cases that can be timed and compared.

Scenes follow the distributions of the package's synthetic scenes (`scenes.uniform_scene`,
`scenes.cluster_scene`), drawn on the GPU so that a case is prepared quickly. Every pass goes
through the public Python API or, where that has no wrapper, the C ABI. The accumulation of a
render call is returned as the renderer's own device buffer, as a headless program uses it.
"""
import importlib
import math

import numpy as np
import torch

gps = importlib.import_module("gps-pbvr-web_b200.gps")
abi = importlib.import_module("gps-pbvr-web_b200.abi")
denoise = importlib.import_module("gps-pbvr-web_b200.denoise")

UP = (0.0, -1.0, 0.0)
SH_FLOATS = {0: 0, 1: 9, 2: 24, 3: 45}


# ------------------------------------------------------------------------------------ the cases
def _frame(name, **kw):
    """A render_ensembles call into a fresh history."""
    c = dict(name=name, kind="frame", scene="cluster", n=560_000, sh=3, w=1280, h=720, spp=1, cap=16384, method="Extinction",
             calibration=3, radial=True, distance=7.0, ensembles=4, composite=False)
    c.update(kw)
    return c


def listed():
    return [
        # One GPS ensemble of a 10,000-splat object at 256x256: a thumbnail or a moving-camera tick,
        # where the launches of a frame count more than its work.
        _frame("gps 10k thumbnail", scene="uniform", n=10_000, sh=0, w=256, h=256, method="Gps", radial=False, distance=3.0,
               ensembles=1),
        # The viewer's default frame: GPS, 2x2 subpixels, 4 ensembles, composited to RGBA8 on the host.
        _frame("gps viewer frame", spp=2, cap=65536, method="Gps", radial=False, composite=True),
        # PBVR Extinction C3+R from inside the scene: nearly all particles leave the screen.
        _frame("pbvr near", distance=2.5),
        # The same scene framed normally.
        _frame("pbvr mid", ensembles=8),
        # A whole accumulation of 64 ensembles from far away: many ensembles with few particles each.
        _frame("pbvr far 64", distance=20.0, ensembles=64),
        # Part of an orbit of a 2M-splat scene at 1920x1080 with ScreenOccupancy, accumulations kept
        # on the device (offline rendering, training data).
        dict(name="occupancy orbit", kind="orbit", n=2_000_000, sh=3, w=1920, h=1080, spp=1, cap=16384, method="ScreenOccupancy",
             distance=7.0, cameras=2, ensembles=2),
        # The depth-sorted frame the session's Auto path shows for ordinary views.
        dict(name="sorted 720p", kind="sorted", n=560_000, sh=3, w=1280, h=720, distance=7.0),
        # The largest sorted frame: 6M splats at 3840x2160.
        dict(name="sorted 4k", kind="sorted", n=6_000_000, sh=3, w=3840, h=2160, distance=7.0),
        # A denoised preview: 4 far-view ensembles, the U-Net, the colours on the host.
        dict(name="denoised frame", kind="denoised", n=560_000, sh=3, w=1280, h=720, distance=20.0, ensembles=4),
        # One training step of the denoiser on a batch of eight 256x256 crops.
        dict(name="denoiser training step", kind="train", batch=8, w=256, h=256),
        # The stand-alone (key, value) sort on 24-bit depth keys.
        dict(name="sort 16M pairs", kind="sort", n=1 << 24, bits=24),
        # Opening a scene: host arrays uploaded, then the first preview ensemble.
        dict(name="open scene", kind="open", n=560_000, sh=3, w=1280, h=720, distance=20.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["orbit", "sorted", "sorted", "denoised", "train", "sort", "open"])
    w, h = int(_log(rng, 200, 1920)), int(_log(rng, 150, 1080))
    n = int(_log(rng, 10_000, 560_000))
    sh = rng.choice([0, 1, 2, 3, 3, 3])
    d = round(_log(rng, 2.5, 20.0), 3)
    if kind == "frame":
        method = rng.choice(["Gps", "Gps", "Proportional", "Extinction", "Extinction", "Extinction", "ViewConditioned",
                             "ScreenOccupancy"])
        spp = rng.choice([1, 1, 2, 3])
        # the per-ensemble work falls with the distance squared and grows with splats and subpixels
        e = max(1, min(int(_log(rng, 1, 64)), int(4 * 560_000 / n * (d / 2.5) ** 1.5 / spp ** 2 * 921_600 / (w * h))))
        return dict(kind=kind, scene="cluster", n=n, sh=sh, w=w, h=h, spp=spp, cap=rng.choice([4096, 16384, 65536]), method=method,
                    calibration=3 if method == "Extinction" else rng.choice([2, 3]), radial=rng.random() < 0.7, distance=d,
                    ensembles=e, composite=rng.random() < 0.3)
    if kind == "orbit":
        return dict(kind=kind, n=n, sh=sh, w=w, h=h, spp=rng.choice([1, 2]), cap=16384,
                    method=rng.choice(["ScreenOccupancy", "Extinction"]), distance=round(_log(rng, 5.0, 20.0), 3),
                    cameras=rng.randint(1, 4), ensembles=rng.randint(1, 3))
    if kind == "sorted":
        big = rng.random() < 0.5
        return dict(kind=kind, n=int(_log(rng, 10_000, 4_000_000)), sh=sh, w=w * 2 if big else w, h=h * 2 if big else h,
                    distance=round(_log(rng, 4.0, 20.0), 3))
    if kind == "denoised":
        return dict(kind=kind, n=n, sh=sh, w=4 * (w // 4), h=4 * (h // 4), distance=round(_log(rng, 7.0, 20.0), 3), ensembles=4)
    if kind == "train":
        return dict(kind=kind, batch=rng.randint(1, 8), w=4 * rng.randint(16, 64), h=4 * rng.randint(16, 64))
    if kind == "sort":
        return dict(kind=kind, n=int(_log(rng, 10_000, 1 << 24)), bits=rng.choice([8, 13, 16, 24, 24, 32]))
    return dict(kind="open", n=n, sh=sh, w=w, h=h, distance=round(_log(rng, 7.0, 20.0), 3))


# ------------------------------------------------------------------------------------ inputs
def _scene(kind, n, sh, seed):
    """(splats (n, 16), SH rest (n * 3 * ((d+1)^2 - 1)) or None) float32 CUDA tensors of the
    package's scene distributions."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def uni(lo, hi, *s):
        return torch.rand(*s, generator=g, device="cuda", dtype=torch.float32) * (hi - lo) + lo

    def nor(m, sd, *s):
        return torch.randn(*s, generator=g, device="cuda", dtype=torch.float32) * sd + m

    if kind == "uniform":
        pos, log_scale, logit = uni(-1, 1, n, 3), nor(-4.0, 0.5, n, 3), nor(0.0, 1.5, n)
    else:
        centres, stds = uni(-5, 5, 64, 3), uni(0.05, 0.8, 64, 3)
        which = torch.randint(0, 64, (n,), generator=g, device="cuda")
        pos = centres[which] + nor(0, 1, n, 3) * stds[which]
        pos[int(0.9 * n):] = uni(-5, 5, n - int(0.9 * n), 3)
        pos = pos[torch.randperm(n, generator=g, device="cuda")]
        log_scale, logit = nor(-3.5, 0.7, n, 3), nor(0.5, 2.0, n)
    s = torch.zeros(n, 16, device="cuda")
    s[:, 0:3], s[:, 3] = pos, torch.sigmoid(logit)
    s[:, 4:7] = log_scale
    s[:, 8:12] = torch.nn.functional.normalize(nor(0, 1, n, 4), dim=1)
    s[:, 12:15] = uni(0, 1, n, 3)
    rest = nor(0.0, 0.05, n * SH_FLOATS[sh]) if sh else None
    return s, rest


class _Accum:
    """A renderer's accumulation buffer as torch.as_tensor reads it; the tensor keeps the renderer,
    which owns the memory, alive."""

    def __init__(self, r, w, h):
        self.renderer = r
        self.__cuda_array_interface__ = {"data": (r.accum_device_ptr(), False), "shape": (h * w, 4), "typestr": "<f4",
                                         "version": 3}


def _camera(c, k=0):
    return gps.OrbitCamera(target=(0.0, 0.0, 0.0), distance=c["distance"], yaw=0.6 + 0.4 * k, pitch=0.25, up=UP,
                           fov_y=0.9).to_camera(c["w"], c["h"])


def _params(c):
    p = gps.RenderParams(spp_side=c.get("spp", 1), max_points_per_splat=c.get("cap", 16384),
                         method=gps.Method[c.get("method", "Extinction")])
    p.pbvr.calibration = gps.Calibration(c.get("calibration", 3))
    p.pbvr.radial_correction = bool(c.get("radial", True))
    return p


def _renderer(c, seed, scene="cluster"):
    r = gps.GpsRenderer(c["w"], c["h"], c.get("spp", 1))
    s, rest = _scene(scene, c["n"], c["sh"], seed)
    torch.cuda.synchronize()
    r.set_gaussians_device(s.data_ptr(), c["n"], rest.data_ptr() if rest is not None else None,
                           rest.numel() if rest is not None else 0, c["sh"])
    return r


def prepare(case, seed):
    c, st = case, {"case": case, "seed": seed & 0x3FFFFFFF}
    kind = c["kind"]
    if kind in ("frame", "orbit", "sorted", "denoised"):
        st["r"] = r = _renderer(c, seed, c.get("scene", "cluster"))
        st["p"] = _params(c)
        st["cams"] = [_camera(c, k) for k in range(c.get("cameras", 1))]
        st["accum"] = torch.as_tensor(_Accum(r, c["w"], c["h"]), device="cuda")
        if kind == "orbit":
            st["out"] = torch.zeros(c["cameras"], c["h"] * c["w"], 4, device="cuda")
        if kind == "denoised":
            st["net"] = denoise.NativeDenoiser()
    elif kind == "open":
        s, rest = _scene("cluster", c["n"], c["sh"], seed)
        st["splats"], st["rest"] = s.cpu().numpy(), (rest.cpu().numpy() if rest is not None else None)
        st["r"] = r = gps.GpsRenderer(c["w"], c["h"], 1)
        st["p"], st["cams"] = _params(c), [_camera(c)]
        st["accum"] = torch.as_tensor(_Accum(r, c["w"], c["h"]), device="cuda")
    elif kind == "train":
        st["net"] = denoise.Denoiser(seed=seed & 0xFFFF)
        st["x"], st["base"], st["target"] = _crops(c, seed)
    else:
        st["keys"], st["vals"] = _pairs(c, seed)
        st["work"] = [torch.empty_like(st["keys"]) for _ in range(4)]
        st["r"] = gps.GpsRenderer(16, 16, 1)
        st["stream"] = torch.cuda.Stream()  # the sort and the copies of its input run in order on one stream
        st["r"].set_stream(st["stream"].cuda_stream)
    return st


def _crops(c, seed):
    """A batch as the renderer gives it: smooth colours, few-ensemble noise around them, coverage,
    depth / (1 + depth) and the per-pixel standard deviation; channels 6 and 7 are padding."""
    b, h, w = c["batch"], c["h"], c["w"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def smooth(ch, cells):
        t = torch.rand(b, ch, cells, cells, generator=g, device="cuda")
        return torch.nn.functional.interpolate(t, size=(h, w), mode="bilinear", align_corners=False).permute(0, 2, 3, 1)

    target = smooth(3, 12).contiguous()
    alpha, depth, sd = smooth(1, 16), smooth(1, 8), 0.3 * smooth(1, 24)
    base = (target + 0.5 * sd * torch.randn(b, h, w, 3, generator=g, device="cuda")).clamp(min=0.0).contiguous()
    x = torch.cat([base, depth, alpha, sd, torch.zeros(b, h, w, 2, device="cuda")], dim=3).to(torch.bfloat16).contiguous()
    return x, base, target


def _pairs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    hi = 1 << c["bits"]
    keys = torch.randint(0, hi, (c["n"],), dtype=torch.int64, generator=g, device="cuda")
    keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)
    vals = torch.randperm(c["n"], generator=g, device="cuda").to(torch.int32)
    return keys, vals


# ------------------------------------------------------------------------------------ one pass
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "frame":
        r = state["r"]
        r.reset_accum()
        r.render_ensembles(state["cams"][0], state["p"], state["seed"], c["ensembles"])
        return {"rgba8": r.composite(state["p"])} if c["composite"] else {"accum": state["accum"]}
    if kind == "orbit":
        state["r"].render_trajectory(state["cams"], state["p"], state["seed"], c["ensembles"], state["out"].data_ptr())
        return {"accum": state["out"]}
    if kind == "sorted":
        state["r"].render_sorted(state["cams"][0], state["p"], 1)
        return {"accum": state["accum"]}
    if kind == "denoised":
        rgb, used, check = state["net"].render(state["r"], state["cams"][0], state["p"], state["seed"], ensembles=c["ensembles"],
                                               gate_limit=10.0)
        return {"rgb": rgb, "used": used, "check": check}
    if kind == "open":
        r = state["r"]
        if state["rest"] is None:
            r.set_gaussians(state["splats"])
        else:
            r.set_gaussians_sh(state["splats"], state["rest"], c["sh"])
        r.render_ensembles(state["cams"][0], state["p"], state["seed"], 1)
        return {"accum": state["accum"]}
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["base"], state["target"], lr=1e-3)
        q = net.p
        return {"loss": loss, "gw": {n: q[n]["gw"] for n in q}, "gb": {n: q[n]["gb"] for n in q},
                "w": {n: q[n]["w"] for n in q}}
    ka, va, kb, vb = state["work"]
    with torch.cuda.stream(state["stream"]):
        ka.copy_(state["keys"])  # the sort overwrites its input
        va.copy_(state["vals"])
        status = abi.lib().gpsb_sort_pairs(state["r"].handle, ka.data_ptr(), va.data_ptr(), kb.data_ptr(), vb.data_ptr(), c["n"],
                                           c["bits"])
    if status != abi.GPSB_OK:
        raise RuntimeError("gpsb_sort_pairs: status %d" % status)
    return {"keys": kb, "vals": vb}


# ------------------------------------------------------------------------------------ what a pass needs
def _project(splats, c, k=0):
    """Of every splat, in 64 bits: (in front of the camera, image mean, covariance a b c, depth)."""
    cam = _camera(c, k)
    s = splats.double()
    rot = torch.as_tensor(np.asarray(cam.view_rot, np.float64).reshape(3, 3), device=s.device)
    pos = torch.as_tensor(np.asarray(cam.view_pos, np.float64), device=s.device)
    cx, cy = (cam.cx, cam.cy) if (cam.cx, cam.cy) != (0.0, 0.0) else (0.5 * c["w"], 0.5 * c["h"])
    p = (s[:, 0:3] - pos) @ rot.T
    z = p[:, 2]
    front = z > 0.05
    zs = torch.where(front, z, torch.ones_like(z))
    tx = (p[:, 0] / zs).clamp(-5.2, 5.2)
    ty = (p[:, 1] / zs).clamp(-5.2, 5.2)
    zero = torch.zeros_like(z)
    j0 = torch.stack([cam.focal_x / zs, zero, -cam.focal_x * tx / zs], 1) @ rot
    j1 = torch.stack([zero, cam.focal_y / zs, -cam.focal_y * ty / zs], 1) @ rot
    q = s[:, 8:12] / s[:, 8:12].norm(dim=1, keepdim=True)
    qw, qx, qy, qz = q.unbind(1)
    cols = torch.stack([torch.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy + qw * qz), 2 * (qx * qz - qw * qy)], 1),
                        torch.stack([2 * (qx * qy - qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz + qw * qx)], 1),
                        torch.stack([2 * (qx * qz + qw * qy), 2 * (qy * qz - qw * qx), 1 - 2 * (qx * qx + qy * qy)], 1)], 1)
    sd = s[:, 4:7].exp()
    u = torch.einsum("nkj,nj->nk", cols, j0) * sd
    v = torch.einsum("nkj,nj->nk", cols, j1) * sd
    a, b, cc = (u * u).sum(1) + cam.low_pass, (u * v).sum(1), (v * v).sum(1) + cam.low_pass
    return front, cam.focal_x * p[:, 0] / zs + cx, cam.focal_y * p[:, 1] / zs + cy, a, b, cc, z


def _particles(c, k=0):
    """Expected particles of one ensemble of the case's scene (of seed 0), from the method's counts."""
    splats, _ = _scene(c.get("scene", "cluster"), c["n"], 0, 0)
    front, mx, my, a, b, cc, z = _project(splats, c, k)
    o = splats[:, 3].double().clamp(0, 1 - 1e-6)
    tau = -torch.log1p(-o)
    area = c.get("spp", 1) ** 2 * 2 * math.pi * (a * cc - b * b).sqrt()
    method = c.get("method", "Extinction")
    if method == "ScreenOccupancy":  # one Bernoulli per subpixel of the splat's screen rectangle
        r = (2 * torch.log((o * 255).clamp(min=1))).sqrt()
        wx = (mx + r * a.sqrt()).clamp(0, c["w"]) - (mx - r * a.sqrt()).clamp(0, c["w"])
        wy = (my + r * cc.sqrt()).clamp(0, c["h"]) - (my - r * cc.sqrt()).clamp(0, c["h"])
        n = wx * wy * c.get("spp", 1) ** 2 * tau.clamp(max=1)
    elif method == "Gps":
        n = area * o  # Li2(o) >= o
        off = (mx + 5.9 * a.sqrt() < 0) | (mx - 5.9 * a.sqrt() >= c["w"]) | (my + 5.9 * cc.sqrt() < 0) | \
            (my - 5.9 * cc.sqrt() >= c["h"])
        n = torch.where(off, torch.zeros_like(n), n).clamp(max=c["cap"])
    else:
        n = area * tau if c.get("calibration", 3) == 3 and method != "ViewConditioned" else 512.0 * tau
        n = n.clamp(max=c.get("cap", 16384))
    return float(torch.where(front, n, torch.zeros_like(n)).sum())


def work(case):
    """Bytes: the scene read once, the outputs written once. Flops of a particle: about 200 (its
    random numbers, three normal pairs, the transform, the projection, the keep test) for the PBVR
    methods, 60 for the others; of a blended splat and pixel: 20."""
    c = case
    kind = c["kind"]
    if kind == "sort":
        return {"bytes": 16 * c["n"], "flops": 0}
    if kind == "train":
        px = c["batch"] * c["w"] * c["h"]
        flops = 0.0
        for (_, cin, cin_real, cout), level in zip(denoise.LAYERS, [1, 1, 4, 4, 16, 16, 4, 4, 1, 1, 1]):
            flops += 2.0 * 9 * cin_real * cout * px / level * 3  # forward, data gradient, weight gradient
        return {"bytes": px * (16 + 12 + 12) + 472_000 * 4 * 7, "flops": flops}
    scene = c["n"] * (64 + 4 * SH_FLOATS[c["sh"]])
    px = c["w"] * c["h"]
    per = 60 if c.get("method", "Extinction") in ("Gps", "ScreenOccupancy") else 200
    if kind == "sorted":
        return {"bytes": scene + 16 * px, "flops": 20.0 * 64 * px}
    if kind == "orbit":
        n = sum(_particles(c, k) for k in range(c["cameras"]))
        return {"bytes": scene + 16 * px * c["cameras"], "flops": per * n * c["ensembles"]}
    n = _particles(c) * c.get("ensembles", 1)
    if kind == "denoised":
        net = sum(2.0 * 9 * l[2] * l[3] * px / v for l, v in zip(denoise.LAYERS, [1, 1, 4, 4, 16, 16, 4, 4, 1, 1, 1]))
        return {"bytes": scene + 12 * px, "flops": per * n + net}
    return {"bytes": scene + (4 if c.get("composite") else 16) * px, "flops": per * n}


# ------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """Monte Carlo frames have no value of their own in 64 bits: the particles of a seed are defined
    by 32-bit random numbers and land on whole subpixels. The sort, the training step and the sorted
    frame have one."""
    c = case
    if c["kind"] == "sort":
        keys, vals = _pairs(c, seed)
        k = keys.to(torch.int64) & 0xFFFFFFFF
        order = torch.argsort(k, stable=True)
        return {"keys": keys[order], "vals": vals[order]}
    if c["kind"] == "train":
        return _exact_train(c, seed)
    if c["kind"] == "sorted" and c["n"] <= 1_000_000:
        return {"accum": _exact_sorted(c, seed)}
    return None


def _exact_train(c, seed):
    net = denoise.Denoiser(seed=seed & 0xFFFF)  # only its initial weights
    x, base, target = _crops(c, seed)
    w, b = {}, {}
    for name, q in net.p.items():
        cin, cout = q["cin"], q["cout"]
        rows = q["w"][:, :9 * cin].to(torch.bfloat16).double().reshape(cout, 3, 3, cin)
        w[name] = rows.permute(0, 3, 1, 2).contiguous().requires_grad_(True)
        b[name] = q["b"].double().clone().requires_grad_(True)
    F = torch.nn.functional

    def conv(n, t):  # nine shifted products: no convolution library needed in 64 bits
        h, wd = t.shape[2:]
        p = F.pad(t, (1, 1, 1, 1))
        out = b[n].view(1, -1, 1, 1)
        for dy in range(3):
            for dx in range(3):
                out = out + torch.einsum("oc,bchw->bohw", w[n][:, :, dy, dx], p[:, :, dy:dy + h, dx:dx + wd])
        return out

    def act(n, t):
        return conv(n, t).relu()

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3)

    t0 = x.double().permute(0, 3, 1, 2)
    s1 = act("c1b", act("c1a", t0))
    s2 = act("c2b", act("c2a", F.avg_pool2d(s1, 2)))
    s3 = act("c3b", act("c3a", F.avg_pool2d(s2, 2)))
    d2 = act("c4b", act("c4a", torch.cat([up(s3), s2], 1)))
    d1 = act("c5b", act("c5a", torch.cat([up(d2), s1], 1)))
    pred = base.double() + conv("c6", d1).permute(0, 2, 3, 1)
    loss = (pred - target.double()).abs().mean()
    loss.backward()
    out = {"loss": loss.detach().reshape(1), "gw": {}, "gb": {}, "w": {}}
    for name, q in net.p.items():
        g = torch.zeros(q["cout"], q["kp"], dtype=torch.float64, device="cuda")
        g[:, :9 * q["cin"]] = w[name].grad.permute(0, 2, 3, 1).reshape(q["cout"], -1)
        out["gw"][name], out["gb"][name] = g, b[name].grad
        out["w"][name] = q["w"].double() - 1e-3 * g / (g.abs() + 1e-8)  # Adam's first step
    return out


def _exact_sorted(c, seed):
    """The depth-sorted alpha image: splats far to near by the 24-bit depth key (ties by index, the
    last one in front), alpha = min(o exp(-r2 / 2), 0.99), splats beyond K standard deviations or
    under 1 / 255 left out, blended front to back until under 1e-4 of the light is left."""
    w, h = c["w"], c["h"]
    splats, rest = _scene("cluster", c["n"], c["sh"], seed)
    cam, bg = _camera(c), (0.05, 0.05, 0.08)
    front, mx, my, a, b, cc, z = _project(splats, c)
    o = splats[:, 3].double()
    kk = (2 * torch.log((o * 255).clamp(min=1.0))).sqrt()
    det = a * cc - b * b
    ex, ey = kk * a.sqrt(), kk * cc.sqrt()
    keep = front & (o >= 1 / 255) & (mx + ex >= 0) & (mx - ex < w) & (my + ey >= 0) & (my - ey < h)
    ids = keep.nonzero().squeeze(1)
    near = z[ids].float().view(torch.int32) >> 8
    ids = ids[torch.argsort(near, stable=True, descending=True)].flip(0)  # nearest first
    mx, my, a, b, cc, o, kk, det, ex, ey = (t[ids] for t in (mx, my, a, b, cc, o, kk, det, ex, ey))
    pos = torch.as_tensor(np.asarray(cam.view_pos, np.float64), device="cuda")
    col = _colour(splats[ids].double(), None if rest is None else rest.double().reshape(c["n"], -1)[ids], pos, c["sh"])
    img = torch.zeros(h * w, 4, dtype=torch.float64, device="cuda")
    x0, x1 = (mx - ex - 0.5).ceil().clamp(0, w - 1).long(), (mx + ex - 0.5).floor().clamp(-1, w - 1).long()
    y0, y1 = (my - ey - 0.5).ceil().clamp(0, h - 1).long(), (my + ey - 0.5).floor().clamp(-1, h - 1).long()
    rows = max(1, min(h, 16))
    for top in range(0, h, rows):
        end = min(h, top + rows)
        ya, yb = y0.clamp(min=top), y1.clamp(max=end - 1)
        wide, tall = (x1 - x0 + 1).clamp(min=0), (yb - ya + 1).clamp(min=0)
        cnt = wide * tall
        who = torch.repeat_interleave(torch.arange(len(cnt), device="cuda"), cnt)  # in depth order
        k = torch.arange(len(who), device="cuda") - (cnt.cumsum(0) - cnt)[who]
        px, py = x0[who] + k % wide[who], ya[who] + k // wide[who]
        dx, dy = px + 0.5 - mx[who], py + 0.5 - my[who]
        r2 = (cc[who] * dx * dx - 2 * b[who] * dx * dy + a[who] * dy * dy) / det[who]
        al = (o[who] * torch.exp(-0.5 * r2)).clamp(max=0.99)
        ok = (r2 <= kk[who] ** 2) & (al >= 1 / 255)
        pix, al, who = ((py - top) * w + px)[ok], al[ok], who[ok]
        order = torch.argsort(pix, stable=True)
        pix, al, who = pix[order], al[order], who[order]
        lg = torch.log1p(-al)
        run_ = lg.cumsum(0) - lg  # light left before each entry, relative to the row band's start
        first = torch.ones_like(pix, dtype=torch.bool)
        first[1:] = pix[1:] != pix[:-1]
        start = torch.zeros((end - top) * w, dtype=torch.float64, device="cuda")
        start[pix[first]] = run_[first]
        before = torch.exp(run_ - start[pix])
        live = before >= 1e-4
        wgt = torch.where(live, before * al, torch.zeros_like(al))
        acc = torch.zeros((end - top) * w, 3, dtype=torch.float64, device="cuda")
        acc.index_add_(0, pix, wgt[:, None] * col[who])
        left = torch.zeros((end - top) * w, dtype=torch.float64, device="cuda")
        left.index_add_(0, pix, torch.where(live, lg, torch.zeros_like(lg)))
        img[top * w:end * w, :3] = acc + torch.exp(left)[:, None] * torch.tensor(bg, dtype=torch.float64, device="cuda")
    img[:, 3] = 1.0
    return img


def _colour(s, rest, pos, deg):
    """The view-dependent colour of splats s (m, 16) with SH rest (m, 3 * r), channel-major."""
    base = s[:, 12:15]
    if rest is None or deg == 0:
        return base.clamp(min=0)
    d = torch.nn.functional.normalize(s[:, 0:3] - pos, dim=1)
    x, y, z = d.unbind(1)
    f = [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if deg >= 2:
        f += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * z * z - x * x - y * y),
              -1.0925484305920792 * x * z, 0.5462742152960396 * (x * x - y * y)]
    if deg >= 3:
        f += [-0.5900435899266435 * y * (3 * x * x - y * y), 2.890611442640554 * x * y * z,
              -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
              0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
              -0.4570457994644658 * x * (4 * z * z - x * x - y * y), 1.445305721320277 * z * (x * x - y * y),
              -0.5900435899266435 * x * (x * x - 3 * y * y)]
    f = torch.stack(f, 1)
    return (base + torch.einsum("mk,mck->mc", f, rest.reshape(len(s), 3, -1))).clamp(min=0)
