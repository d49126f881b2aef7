"""The work that users of this framework have it do, as timed and checked cases.

Each case is one call (or the few calls of one step) through the public entry
points: the host-pointer drop-in ABI, the device plans, the batched 2D
operators, SIRT3D, the TV flow, the warm-start network and the curved-detector
FDK.  ``exact`` restates each operator in plain 64-bit torch.

Geometry fields of a cone case: nt, ns, nz voxels over st, ss, sz mm; views
over a full turn; cols x rows detector samples at pp, px mm at the rotation
centre; source-to-centre distance dist.  A fan case: n x n pixels of 1 mm,
views, bins, dist.
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path.cwd()
PKG = ROOT / "ct-research_gb300"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

MATLAB_EPS = 2.220446049250313e-16
F64 = torch.float64


# -- the cases ------------------------------------------------------------------
def _cone(kind, name, nt, ns, nz, views, cols, rows, size=None, pitch=None, **kw):
    """A cone scan like the 512^3 workload's (200 x 200 x 150 mm seen by a
    307.2 x 204.8 mm detector at the centre) at other sizes."""
    m = max(nt, ns)
    if size is None:
        size = (200.0 * nt / m, 200.0 * ns / m, 150.0 * nz / m)
    if pitch is None:
        pitch = (307.2 / cols, 204.8 * size[2] / 150.0 / rows)
    return dict(name=name, kind=kind, nt=nt, ns=ns, nz=nz, st=float(size[0]), ss=float(size[1]), sz=float(size[2]),
                views=views, cols=cols, rows=rows, pp=float(pitch[0]), px=float(pitch[1]), dist=600.0, **kw)


def _fan(kind, name, n, views, bins, **kw):
    return dict(name=name, kind=kind, n=n, views=views, bins=bins, dist=500.0, **kw)


def listed():
    return [
        # a script that calls the 2D filtered backprojection of the drop-in ABI on host arrays, slice by slice
        _fan("dropin_fbp", "dropin_fbp_256", 256, 360, 512),
        # one SIRT iteration of a small 2D fan slice on the device: launch latency counts
        _fan("fan_sirt", "fan_sirt_128", 128, 90, 256),
        # the filtered backprojection of a large 2D fan slice through its plan
        _fan("fan_fbp", "fan_fbp_512", 512, 720, 1024),
        # one SIRT iteration of the batch of 64 uneven fan slices
        dict(name="fan_batch_64", kind="fan_batch", slices=64, mix=4),
        # SIRT3D of a small scan with odd sizes on every axis: a whole call, normalisers included
        _cone("sirt3d", "sirt3d_odd", 151, 133, 97, 77, 221, 143, iters=4),
        # the forward projection of the 512^3 / 360-view throughput workload
        _cone("cone_fp", "cone_fp_512", 512, 512, 512, 360, 768, 512),
        # its backprojection
        _cone("cone_bp", "cone_bp_512", 512, 512, 512, 360, 768, 512),
        # FDK of the 256^3 scan (128 mm, 512 x 384 at 0.4 mm), filter and backprojection in the reference's modes
        _cone("fdk", "fdk_256", 256, 256, 256, 360, 512, 384, size=(128.0, 128.0, 128.0), pitch=(0.4, 0.4)),
        # the TV phase between two SIRT updates: 20 sub-steps on a noisy volume
        dict(name="tv_256", kind="tv", nt=256, ns=256, nz=256, iters=20),
        # the warm-start network applied to a volume (shipped weights): a whole call
        dict(name="unet_forward_256", kind="unet_forward", nx=256, ny=256, nz=256),
        # one training step of the network at the training size: forward, all gradients, Adam
        dict(name="unet_train_128", kind="unet_train", nx=128, ny=128, nz=128),
        # the curved-detector short-scan FDK of the scanner set-up
        dict(name="curved_fdk", kind="curved", gammas=936, rows=80, views=800, n=512, nz=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin_fbp", "fan_sirt", "fan_fbp", "fan_batch", "sirt3d", "cone_fp", "cone_bp", "fdk", "tv",
                       "unet_forward", "unet_train", "curved"])
    if kind in ("dropin_fbp", "fan_sirt", "fan_fbp"):
        c = _fan(kind, "", _log(rng, 96, 512), _log(rng, 60, 720), _log(rng, 160, 1024))
    elif kind == "fan_batch":
        c = dict(name="", kind=kind, slices=_log(rng, 4, 48), mix=rng.randrange(1000))
    elif kind == "sirt3d":
        n = _log(rng, 48, 160)
        c = _cone(kind, "", n, n + rng.randint(-5, 5), n + rng.randint(-9, 0), _log(rng, 40, 120),
                  int(n * rng.uniform(1.3, 1.6)), int(n * rng.uniform(0.9, 1.1)), iters=rng.randint(2, 5))
    elif kind == "tv":
        n = _log(rng, 48, 400)
        c = dict(name="", kind=kind, nt=n, ns=n + rng.randint(-9, 9), nz=max(32, n - rng.randint(0, n // 3)),
                 iters=rng.randint(5, 20))
    elif kind == "unet_forward":
        c = dict(name="", kind=kind, nx=2 ** rng.randint(6, 8), ny=2 ** rng.randint(6, 8), nz=16 * rng.randint(2, 16))
    elif kind == "unet_train":
        c = dict(name="", kind=kind, nx=2 ** rng.randint(6, 7), ny=2 ** rng.randint(6, 7), nz=16 * rng.randint(2, 8))
    elif kind == "curved":
        c = dict(name="", kind=kind, gammas=_log(rng, 240, 936), rows=_log(rng, 16, 80), views=_log(rng, 120, 800),
                 n=_log(rng, 96, 512), nz=_log(rng, 12, 50))
    else:
        top = 320 if kind == "fdk" else 480
        m = _log(rng, 64, top)
        c = _cone(kind, "", m, max(48, m - rng.randint(0, m // 4)), max(40, m - rng.randint(0, m // 3)),
                  _log(rng, 45, 360), int(m * rng.uniform(1.2, 1.6)), int(m * rng.uniform(0.8, 1.1)))
    c.pop("name")
    return c


# -- inputs (plain torch and numpy) -----------------------------------------------
def _libm(name):
    f = getattr(ctypes.CDLL("libm.so.6"), name)
    f.restype, f.argtypes = ctypes.c_float, [ctypes.c_float]
    return f


def _angles(views):
    return np.arange(1, views + 1, dtype=np.float64) * (2 * np.pi / views)


def _cone_arrays(c):
    beta = _angles(c["views"]).astype(np.float32)
    P = ((np.arange(c["cols"]) - (c["cols"] - 1) / 2.0) * c["pp"]).astype(np.float32)
    xi = ((np.arange(c["rows"]) - (c["rows"] - 1) / 2.0) * c["px"]).astype(np.float32)
    return beta, P, xi


def _fan_arrays(n, views, bins):
    maxp = 1.1 * n * np.sqrt(2.0) / 2.0
    return _angles(views), np.linspace(-maxp, maxp, bins)


def _batch_scans(c):
    rng = np.random.default_rng(c["mix"])       # the ranges of the batched 2D workload
    return [(int(rng.integers(128, 513)), int(rng.integers(90, 721)), int(rng.integers(256, 1025)))
            for _ in range(c["slices"])]


def _ellipsoids(seed, count=10):
    """Rows (amplitude, a, b, c, x0, y0, z0, phi) in units of the half extents."""
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(count, 3))
    v *= (0.5 * rng.uniform(0, 1, count) ** (1 / 3) / np.linalg.norm(v, axis=1))[:, None]
    return np.column_stack([rng.uniform(0.1, 0.5, count), rng.uniform(0.08, 0.45, (count, 3)), v,
                            rng.uniform(0, np.pi, count)])


def _volume(shape, seed):
    """float32 [z][s][t]: a sum of ellipsoids, clipped to [0, 1], with 1% texture."""
    nz, ns, nt = shape
    g = torch.Generator(device="cuda").manual_seed(seed)
    ax = [((torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * (2.0 / n) - 1.0) for n in (nt, ns, nz)]
    x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    vol = torch.zeros(shape, device="cuda")
    for A, a, b, cc, x0, y0, z0, phi in _ellipsoids(seed):
        co, si = math.cos(phi), math.sin(phi)
        q = (((x - x0) * co + (y - y0) * si) / a) ** 2 + (((y - y0) * co - (x - x0) * si) / b) ** 2
        vol += A * (q + ((z - z0) / cc) ** 2 <= 1.0)
    noise = torch.rand(shape, device="cuda", generator=g)
    return vol.clamp_(0.0, 1.0).mul_(noise.mul_(0.02).add_(0.99)).contiguous()


def _line_integrals(src, d, half, seed):
    """Line integrals of the ellipsoids (src, d: three broadcastable tensors each, relative to the centre)."""
    norm = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    out = 0.0
    for A, a, b, cc, x0, y0, z0, phi in _ellipsoids(seed):
        co, si = math.cos(phi), math.sin(phi)
        r = min(half[0], half[1])
        p = (src[0] - x0 * half[0], src[1] - y0 * half[1], src[2] - z0 * half[2])
        u = ((p[0] * co + p[1] * si) / (a * r), (p[1] * co - p[0] * si) / (b * r), p[2] / (cc * half[2]))
        w = ((d[0] * co + d[1] * si) / (a * r), (d[1] * co - d[0] * si) / (b * r), d[2] / (cc * half[2]))
        ww = w[0] * w[0] + w[1] * w[1] + w[2] * w[2]
        uw = u[0] * w[0] + u[1] * w[1] + u[2] * w[2]
        uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        disc = (uw * uw - ww * (uu - 1.0)).clamp_min(0.0)
        out = out + A * 2.0 * torch.sqrt(disc) / ww * norm
    return out


def _cone_sino(c, seed):
    """float32 [beta][xi][P]: the ellipsoids' line integrals with 0.3% noise."""
    beta, P, xi = _cone_arrays(c)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    half = (c["st"] / 2, c["ss"] / 2, c["sz"] / 2)
    Pt = torch.from_numpy(P).cuda()[None, None, :]
    Xt = torch.from_numpy(xi).cuda()[None, :, None]
    out = torch.empty((len(beta), len(xi), len(P)), device="cuda")
    step = max(1, (1 << 25) // (len(P) * len(xi)))
    for v in range(0, len(beta), step):
        b = torch.from_numpy(beta[v:v + step]).cuda()[:, None, None]
        s, k = torch.sin(b), torch.cos(b)
        D = c["dist"]
        src = (-D * s, D * k, torch.zeros_like(b))
        d = (Pt * k + D * s, Pt * s - D * k, Xt)
        q = _line_integrals(src, d, half, seed)
        out[v:v + step] = q * (1.0 + 0.003 * torch.randn(q.shape, device="cuda", generator=g))
    return out


def _fan_sino(n, views, bins, dist, seed):
    beta, P = _fan_arrays(n, views, bins)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    Pt = torch.from_numpy(P).cuda().float()[None, :]
    b = torch.from_numpy(beta).cuda().float()[:, None]
    s, k = torch.sin(b), torch.cos(b)
    zero = torch.zeros_like(b)
    q = _line_integrals((-dist * s, dist * k, zero), (Pt * k + dist * s, Pt * s - dist * k, zero),
                        (n / 2, n / 2, 1.0), seed)
    return (q * (1.0 + 0.003 * torch.randn(q.shape, device="cuda", generator=g))).contiguous()


def _tv_input(c, seed):
    """A volume over a background, with noise: 2% of a full amplitude, as a SIRT update leaves it."""
    g = torch.Generator(device="cuda").manual_seed(seed + 3)
    vol = _volume((c["nz"], c["ns"], c["nt"]), seed)
    return (0.2 + 0.6 * vol + 0.02 * torch.randn(vol.shape, device="cuda", generator=g)).contiguous()


def _curved_arrays(c):
    """The scanner's set-up (ImplementUIData.m): 936 gammas over the fan, 80 rows, 240 degrees; other
    sample counts cover the same fan, height and arc."""
    gama = -(np.arange(c["gammas"]) - (c["gammas"] - 1) / 2) * (9.7527e-4 * 936 / c["gammas"])
    xi = (np.arange(c["rows"]) - (c["rows"] - 1) / 2) * (0.915 * 80 / c["rows"])
    b0 = math.radians(1.5466)
    beta = b0 + math.radians(240 / c["views"]) * np.arange(c["views"])
    # a hair more than the detector's own fan angle: the edge samples stay clear of the ramps' poles
    fan = 1.001 * abs(gama[-1] - gama[0])
    return dict(gama=gama, xi=xi, beta=beta, b0=b0, fan=fan, D=570.0, ds2d=1060.2,
                size=np.array([c["n"], c["n"], 23], np.int32), nz=c["nz"])


def _curved_input(c, seed):
    a = _curved_arrays(c)
    g = torch.Generator(device="cuda").manual_seed(seed)
    b = torch.tensor(a["beta"], device="cuda").view(-1, 1, 1)
    x = torch.tensor(a["xi"], device="cuda").view(1, -1, 1)
    gm = torch.tensor(a["gama"], device="cuda").view(1, 1, -1)
    gm = gm / gm.abs().max()
    ph = np.random.default_rng(seed).uniform(0, 6, 3)
    R = (1.0 + 0.3 * torch.cos(b + 0.01 * x + ph[0]) + 0.2 * torch.cos(3 * b + ph[1]) * gm) * (1 - gm * gm)
    noise = torch.randn(R.shape, device="cuda", dtype=F64, generator=g)
    return (R * (1.0 + 0.003 * noise)).contiguous()


def _net_input(c, seed):
    """A volume smoothed and noisy, and the volume itself, as [1][z][y][x]."""
    y = _volume((c["nz"], c["ny"], c["nx"]), seed)[None]
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    x = torch.nn.functional.avg_pool3d(y[None], 3, stride=1, padding=1)[0]
    return (x + 0.02 * torch.randn(x.shape, device="cuda", generator=g)).contiguous(), y


# -- the framework's objects --------------------------------------------------------
def _cone_plan(c):
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry
    return ConePlan(ConeGeometry(c["nt"], c["ns"], c["nz"], (c["st"], c["ss"], c["sz"]), *_cone_arrays(c), c["dist"]))


def _fan_geom(n, views, bins, dist):
    from ctgb.geometry import FanGeometry
    return FanGeometry(n, n, (n, n), *_fan_arrays(n, views, bins), dist)


def prepare(case, seed):
    import ctgb
    ctgb.load()
    k = case["kind"]
    s = {"kind": k}
    if k in ("dropin_fbp", "fan_sirt", "fan_fbp"):
        n, views, bins, dist = case["n"], case["views"], case["bins"], case["dist"]
        sino = _fan_sino(n, views, bins, dist, seed)
        if k == "dropin_fbp":
            beta, P = _fan_arrays(n, views, bins)
            s |= dict(case=case, R=sino.cpu().numpy(), beta=beta.astype(np.float32), P=P.astype(np.float32),
                      size=np.array([n, n], np.float64), out=np.empty((n, n), np.float32))
            return s
        from ctgb.device import FanPlan
        plan = s["plan"] = FanPlan(_fan_geom(n, views, bins, dist))
        s["b"] = sino
        if k == "fan_sirt":
            s["rowsum"] = plan.fp(torch.ones((n, n), device="cuda"))
            s["colsum"] = plan.bp(torch.ones_like(sino))
            s["x"] = 0.5 * _volume((1, n, n), seed)[0]
            s["e"] = torch.empty_like(sino)
            s["norms"] = torch.zeros(2, dtype=F64, device="cuda")
    elif k == "fan_batch":
        from ctgb.batch import FanBatch
        scans = _batch_scans(case)
        batch = s["batch"] = FanBatch([_fan_geom(*q, 500.0) for q in scans])
        s["b"] = batch.pack_sinos([_fan_sino(*q, 500.0, seed + i) for i, q in enumerate(scans)])
        s["x"] = batch.pack_images([0.5 * _volume((1, q[0], q[0]), seed + i)[0] for i, q in enumerate(scans)])
        s["rowsum"] = batch.fp(torch.ones(batch.n_img, device="cuda"))
        s["colsum"] = batch.bp(torch.ones(batch.n_sino, device="cuda"))
        s["e"] = torch.empty_like(s["b"])
        s["norms"] = torch.zeros(len(scans), 2, dtype=F64, device="cuda")
    elif k in ("cone_fp", "cone_bp", "fdk", "sirt3d"):
        plan = s["plan"] = _cone_plan(case)
        if k == "cone_fp":
            s["vol"] = _volume((case["nz"], case["ns"], case["nt"]), seed)
            s["proj"] = plan.new_sino()
        else:
            s["b"] = _cone_sino(case, seed)
            s["out"] = plan.new_volume()
        if k == "sirt3d":
            from ctgb.sirt import SirtConfig
            s["cfg"] = SirtConfig(iters=case["iters"], check_every=case["iters"])
    elif k == "tv":
        s["x0"] = _tv_input(case, seed)
        s["x"], s["work"] = torch.empty_like(s["x0"]), torch.empty_like(s["x0"])
        s["scratch"] = torch.zeros(2, dtype=F64, device="cuda")
        s["iters"] = case["iters"]
    elif k in ("unet_forward", "unet_train"):
        from ctgb import warmstart
        s["net"] = warmstart.load()
        s["x"], s["y"] = _net_input(case, seed)
    elif k == "curved":
        s |= _curved_arrays(case)
        s["R"] = _curved_input(case, seed)
        s["rcov"] = torch.empty(s["R"].shape, dtype=torch.float32, device="cuda")
        s["disp"] = torch.empty((case["nz"], case["n"], case["n"]), dtype=F64, device="cuda")
    else:
        raise ValueError(k)
    return s


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def run(s):
    k = s["kind"]
    if k == "dropin_fbp":
        from ctgb import _lib
        c = s["case"]
        _lib.call("ct_FBPfan", _p(s["out"]), _p(s["R"]), _p(s["P"]), _p(s["beta"]), len(s["beta"]), len(s["P"]),
                  _p(s["size"]), c["n"], c["n"], c["dist"])
        return s["out"]
    if k == "fan_sirt":
        s["plan"].fp_residual(s["x"], s["b"], s["rowsum"], MATLAB_EPS, out=s["e"], norms=s["norms"])
        s["plan"].bp_update(s["e"], s["colsum"], s["x"], lam=2.0, eps=MATLAB_EPS, lo=0.0, hi=1.0)
        return {"e": s["e"], "x": s["x"]}
    if k == "fan_fbp":
        return s["plan"].fbp(s["b"])
    if k == "fan_batch":
        s["norms"].zero_()
        s["batch"].fp_residual(s["x"], s["b"], s["rowsum"], MATLAB_EPS, s["e"], s["norms"])
        s["batch"].bp_update(s["e"], s["colsum"], s["x"], 2.0, MATLAB_EPS, 0.0, 1.0)
        return {"e": s["e"], "x": s["x"], "norms": s["norms"].float()}
    if k == "cone_fp":
        return s["plan"].fp(s["vol"], s["proj"])
    if k == "cone_bp":
        return s["plan"].bp(s["b"], s["out"])
    if k == "fdk":
        return s["plan"].fdk(s["b"], s["out"])
    if k == "sirt3d":
        from ctgb.sirt import sirt3d
        res = sirt3d(s["plan"], s["b"], s["cfg"])
        return {"x": res.x, "residual": torch.tensor([r for _, r in res.residuals], dtype=torch.float32)}
    if k == "tv":
        from ctgb.device import tv_flow
        s["x"].copy_(s["x0"])
        return tv_flow(s["x"], s["iters"], 1e-3, work=s["work"], scratch=s["scratch"])
    if k == "unet_forward":
        return s["net"].forward(s["x"])
    if k == "unet_train":
        net = s["net"]
        out = net.forward(s["x"], keep=True)
        grads = net.backward((2.0 / out.numel()) * (out - s["y"]))
        net.adam_step(grads, lr=1e-5)
        return {"out": out, "grads": grads}
    if k == "curved":
        from ctgb.device import fdkui_bp, fdkui_filter
        fdkui_filter(s["R"], s["xi"], s["gama"], s["beta"], s["b0"], s["fan"], s["D"], s["ds2d"], s["rcov"])
        fdkui_bp(s["rcov"], s["xi"], s["gama"], s["beta"], s["D"], s["ds2d"], s["size"], s["nz"], s["disp"])
        return {"filtered": s["rcov"], "display": s["disp"]}
    raise ValueError(k)


# -- the work each case cannot do without -----------------------------------------------
def _net_flops(vox):
    """Multiply-adds x 2 of the 17 convolutions and the head: 4.2e5 per voxel."""
    per = 0.0
    for lvl, layers in ((1, ((27, 32), (27 * 32, 32), (27 * 64, 32), (27 * 32, 32), (32, 1))),
                        (8, ((27 * 32, 64), (27 * 64, 64), (27 * 128, 64), (27 * 64, 64), (64, 32))),
                        (64, ((27 * 64, 128), (27 * 128, 128), (27 * 256, 128), (27 * 128, 128), (128, 64))),
                        (512, ((27 * 128, 256), (27 * 256, 256), (256, 128)))):
        per += sum(2.0 * k * m for k, m in layers) / lvl
    return per * vox


def work(case):
    k = case["kind"]
    # Siddon segments per ray: 0.22 (cone: 4.85e10 of 1.42e8 rays at 512^3) and 0.8 (fan) of the sum of the sizes
    if k in ("dropin_fbp", "fan_sirt", "fan_fbp", "fan_batch"):
        scans = _batch_scans(case) if k == "fan_batch" else [(case["n"], case["views"], case["bins"])]
        by = fl = 0.0
        for n, v, p in scans:
            if k in ("dropin_fbp", "fan_fbp"):
                by += 4.0 * (v * p + n * n)
                fl += 2.0 * v * p * p + 8.0 * n * n * v
            else:
                by += 4.0 * (3 * v * p + 3 * n * n)
                fl += 2.0 * 0.8 * n * v * p + 12.0 * n * n * v
        return {"bytes": by, "flops": fl}
    if k in ("unet_forward", "unet_train"):
        vox = case["nx"] * case["ny"] * case["nz"]
        f = 1 if k == "unet_forward" else 3
        return {"bytes": 8.0 * vox + f * 2.0 * 3.9e6, "flops": f * _net_flops(vox)}
    if k == "curved":
        r = case["gammas"] * case["rows"] * case["views"]
        vox = case["n"] ** 2 * case["nz"]
        return {"bytes": 12.0 * r + 8.0 * vox, "flops": 2.0 * r * case["gammas"] + 11.0 * vox * case["views"]}
    vox = case["nt"] * case["ns"] * case["nz"]
    if k == "tv":
        return {"bytes": 8.0 * vox, "flops": case["iters"] * 30.0 * vox}
    rays = case["views"] * case["cols"] * case["rows"]
    fp = 2.0 * 0.22 * (case["nt"] + case["ns"] + case["nz"]) * rays
    bp = 11.0 * vox * case["views"]
    one = 4.0 * (vox + rays)
    if k == "cone_fp":
        return {"bytes": one, "flops": fp}
    if k == "cone_bp":
        return {"bytes": one, "flops": bp}
    if k == "fdk":
        return {"bytes": one, "flops": bp + 2.0 * rays * case["cols"]}
    return {"bytes": one, "flops": (case["iters"] + 1) * (fp + bp)}


# -- the same results in 64 bits ------------------------------------------------------------
def _siddon64(vol, n, res, src, d):
    """Line integrals of vol (flat float64, n[0] fastest) along src + a d (three tensors each), stepping all rays at once."""
    d = [torch.where(x == 0, torch.full_like(x, 1e-300), x) for x in d]
    lo = torch.full_like(d[0], -1e300)
    hi = torch.full_like(d[0], 1e300)
    for a in range(3):
        t0, t1 = (0.0 - src[a]) / d[a], (n[a] * res[a] - src[a]) / d[a]
        lo, hi = torch.maximum(lo, torch.minimum(t0, t1)), torch.minimum(hi, torch.maximum(t0, t1))
    acc = torch.zeros_like(lo)
    hi = torch.maximum(lo, hi)
    nxt, step = [], []
    for a in range(3):
        p = (src[a] + lo * d[a]) / res[a]
        k = torch.where(d[a] > 0, torch.floor(p + 1e-9) + 1, torch.ceil(p - 1e-9) - 1)
        nxt.append((k * res[a] - src[a]) / d[a])
        step.append(res[a] / d[a].abs())
    cur = lo
    for it in range(sum(n) + 8):
        if it % 32 == 31 and not bool((cur < hi).any()):
            break
        end = torch.minimum(torch.minimum(nxt[0], nxt[1]), torch.minimum(nxt[2], hi))
        mid = 0.5 * (cur + end)
        idx = torch.zeros_like(mid, dtype=torch.int64)
        for a in (2, 1, 0):
            v = torch.floor((src[a] + mid * d[a]) / res[a]).to(torch.int64).clamp_(0, n[a] - 1)
            idx = idx * n[a] + v
        acc += (end - cur) * vol[idx]
        for a in range(3):
            nxt[a] = torch.where(nxt[a] <= end, nxt[a] + step[a], nxt[a])
        cur = end
    return acc * torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)


def _trig32(beta):
    s, k = _libm("sinf"), _libm("cosf")
    return [(float(s(float(b))), float(k(float(b)))) for b in beta]


def _cone_fp64(c, vol):
    beta, P, xi = _cone_arrays(c)
    n, res = (c["nt"], c["ns"], c["nz"]), (c["st"] / c["nt"], c["ss"] / c["ns"], c["sz"] / c["nz"])
    v = vol.double().reshape(-1)
    Pt = torch.from_numpy(P).cuda().double()[None, None, :]
    Xt = torch.from_numpy(xi).cuda().double()[None, :, None]
    out = torch.empty((len(beta), len(xi), len(P)), dtype=F64, device="cuda")
    tr = _trig32(beta)
    step = max(1, (1 << 24) // (len(P) * len(xi)))
    D = c["dist"]
    for k in range(0, len(beta), step):
        t = torch.tensor(tr[k:k + step], dtype=F64, device="cuda")
        s, co = t[:, 0, None, None], t[:, 1, None, None]
        full = torch.zeros((t.shape[0], len(xi), len(P)), dtype=F64, device="cuda")
        src = [c["st"] / 2 - D * s + full, c["ss"] / 2 + D * co + full, c["sz"] / 2 + full]
        d = [Pt * co + D * s + full, Pt * s - D * co + full, Xt + full]
        out[k:k + step] = _siddon64(v, n, res, src, d)
    return out


def _cone_bp64(c, R, fdk=False):
    """Chord-weighted backprojection, or FDK's with a column's last in-range value kept above the detector."""
    beta, P, xi = _cone_arrays(c)
    nt, ns, nz = c["nt"], c["ns"], c["nz"]
    rt, rs, rz = c["st"] / nt, c["ss"] / ns, c["sz"] / nz
    it = ((torch.arange(nt, device="cuda", dtype=F64) + 0.5) * rt - c["st"] / 2)[None, :]
    is_ = ((torch.arange(ns, device="cuda", dtype=F64) + 0.5) * rs - c["ss"] / 2)[:, None]
    iz = ((torch.arange(nz, device="cuda", dtype=F64) + 0.5) * rz - c["sz"] / 2)[:, None, None]
    Pt, Xt = torch.from_numpy(P).cuda().double(), torch.from_numpy(xi).cuda().double()
    pint, xint = float(abs(P[1] - P[0])), float(abs(xi[1] - xi[0]))
    bint = float(abs(beta[1] - beta[0]))
    D = c["dist"]
    acc = torch.zeros((nz, ns, nt), dtype=F64, device="cuda")
    for v, (s, k) in enumerate(_trig32(beta)):
        R2 = R[v].double()
        dt, ds = it * k + is_ * s, -it * s + is_ * k
        lr = D / (D - ds)
        Pq = dt * lr
        pin = (Pq >= float(P.min())) & (Pq < float(P.max()))
        p1 = torch.floor((Pq - Pt[0]).abs() / pint).long().clamp_(0, len(P) - 2)
        wp1, wp0 = (Pq - Pt[p1]).abs() / pint, (Pt[p1 + 1] - Pq).abs() / pint
        X = iz * lr
        zin = (X >= float(xi.min())) & (X < float(xi.max()))
        if fdk:
            last = torch.where(zin, torch.arange(nz, device="cuda")[:, None, None], 0).amax(0)   # last in-range z
            top = torch.gather(X, 0, last[None])
            above = torch.arange(nz, device="cuda")[:, None, None] > last[None]
            some = zin.any(0)
            X = torch.where(above, top, X)
            zin = (zin | above) & some
        x1 = torch.floor((X - Xt[0]).abs() / xint).long().clamp_(0, len(xi) - 2)
        wx1, wx0 = (X - Xt[x1]).abs() / xint, (Xt[x1 + 1] - X).abs() / xint
        flat = R2.reshape(-1)
        o = x1 * len(P) + p1
        val = wx0 * (wp0 * flat[o] + wp1 * flat[o + 1]) + wx1 * (wp0 * flat[o + len(P)] + wp1 * flat[o + len(P) + 1])
        if fdk:
            w = lr * lr * bint
        else:
            ex, ey = it + D * s, is_ - D * k
            m = torch.minimum(torch.minimum(rt / 2 / ex.abs(), rs / 2 / ey.abs()), rz / 2 / iz.abs())
            w = 2.0 * m * torch.sqrt(ex * ex + ey * ey + iz * iz)
        acc += torch.where(zin & pin, val * w, torch.zeros_like(val))
    return acc


def _taps64(pint, np_):
    n = torch.arange(-(np_ - 1), np_, dtype=F64, device="cuda")
    a = (math.pi * pint) ** 2
    return torch.where(n == 0, torch.full_like(n, 1.0 / a), -1.0 / a / (4 * n * n - 1)).float().double()


def _ramp64(R, weight, pint, tile, row_block, rows_mod):
    """Rows of R (last axis) through the Shepp-Logan taps, the pre-weight applied in the launch order of the
    reference: an output tile sees the tiles launched up to its own weighted and the later ones raw."""
    np_ = R.shape[-1]
    G = _taps64(pint, np_)
    i = torch.arange(np_, device="cuda")
    T = G[(np_ - 1) + i[None, :] - i[:, None]]            # [q][p]
    nfull, resid = np_ // tile, np_ % tile
    tiles = nfull + (1 if resid else 0)
    raw = R.double()
    wt = raw * weight
    out = torch.empty_like(raw)
    ridx = torch.arange(rows_mod, device="cuda")
    late = (rows_mod % row_block != 0) & (ridx >= (rows_mod // row_block) * row_block)
    for sel, first in ((~late, False), (late, True)):
        if not bool(sel.any()):
            continue
        def pos(k):
            return (0 if k == nfull else k + 1) if (first and resid) else k
        for k in range(tiles):
            seen = torch.tensor([pos(j) <= pos(k) for j in range(tiles)], device="cuda")[i // tile]
            a, b = k * tile, min(np_, (k + 1) * tile)
            mix = torch.where(seen, wt[..., sel, :], raw[..., sel, :])
            out[..., sel, a:b] = pint * (mix @ T[:, a:b])
    return out


def _fdk64(c, b):
    beta, P, xi = _cone_arrays(c)
    w = c["dist"] / torch.sqrt(c["dist"] ** 2 + torch.from_numpy(P).cuda().double()[None, :] ** 2 +
                               torch.from_numpy(xi).cuda().double()[:, None] ** 2)
    filt = torch.empty(b.shape, dtype=F64, device="cuda")
    for v in range(0, len(beta), 16):
        filt[v:v + 16] = _ramp64(b[v:v + 16], w, float(abs(P[1] - P[0])), 256, 256, len(xi))
    return _cone_bp64(c, filt, fdk=True)


def _fan_fp64(n, views, bins, dist, img):
    beta, P = _fan_arrays(n, views, bins)
    b = torch.from_numpy(beta).cuda()[:, None]
    Pt = torch.from_numpy(P).cuda()[None, :]
    full = torch.zeros((views, bins), dtype=F64, device="cuda")
    s, k = torch.sin(b), torch.cos(b)
    src = [n / 2 - dist * s + full, n / 2 + dist * k + full, 0.5 + full]
    d = [Pt * k + dist * s + full, Pt * s - dist * k + full, full]
    return _siddon64(img.double().reshape(-1), (n, n, 1), (1.0, 1.0, 1.0), src, d)


def _fan_bp64(n, views, bins, dist, R, fbp):
    beta, P = _fan_arrays(n, views, bins)
    bf, Pf = beta.astype(np.float32), P.astype(np.float32)
    Pt = torch.from_numpy(Pf).cuda().double()
    pint, bint = float(abs(Pf[1] - Pf[0])), float(abs(bf[1] - bf[0]))
    t = torch.arange(n, device="cuda", dtype=F64)
    it, is_ = (t + 0.5 - n / 2)[None, :], (t + 0.5 - n / 2)[:, None]
    acc = torch.zeros((n, n), dtype=F64, device="cuda")
    for v, (s, k) in enumerate(_trig32(bf)):
        u = (dist - (is_ * k - it * s)) / dist
        pd = (it * k + is_ * s) / u
        ok = (pd >= float(Pf.min())) & (pd < float(Pf.max()))
        p1 = torch.floor((pd - Pt[0]).abs() / pint).long().clamp_(0, bins - 2)
        row = R[v].double()
        val = (Pt[p1 + 1] - pd).abs() / pint * row[p1] + (pd - Pt[p1]).abs() / pint * row[p1 + 1]
        if fbp:
            acc += torch.where(ok, val / (u * u) * bint, torch.zeros_like(val))
            continue
        st, ss = n / 2 - dist * s, n / 2 + dist * k
        th = torch.atan(pd / dist)
        a, cr = 2 * dist * torch.sin(th), dist - 2 * dist * torch.cos(th)
        et, es = n / 2 + a * k - cr * s, n / 2 + a * s + cr * k
        gt, gs = et - st, es - ss
        lo_t, lo_s = t[None, :], t[:, None]
        at_s = ss + (lo_t - st) * (gs / torch.where(gt == 0, torch.full_like(gt, 1e-15), gt)).clamp(-1e16, 1e16)
        at_t = st + (lo_s - ss) * (gt / torch.where(gs == 0, torch.full_like(gs, 1e-15), gs)).clamp(-1e16, 1e16)
        one = (at_s >= 0) & (at_s <= lo_s + 1)
        two = ~one & (at_t >= 0) & (at_t <= lo_t + 1)
        T1 = torch.where(one, lo_t.expand(n, n), at_t)
        S1 = torch.where(one, at_s, lo_s.expand(n, n))
        w = 2.0 * torch.sqrt((T1 - et) ** 2 + (S1 - es) ** 2)
        acc += torch.where(ok & (one | two), val * w, torch.zeros_like(val))
    return acc


def _fan_fbp64(n, views, bins, dist, sino):
    P = _fan_arrays(n, views, bins)[1].astype(np.float32)
    w = dist / torch.sqrt(dist ** 2 + torch.from_numpy(P).cuda().double() ** 2)
    filt = _ramp64(sino[None], w, float(abs(P[1] - P[0])), 128, 128, views)[0]
    return _fan_bp64(n, views, bins, dist, filt, True)


def _fan_sirt64(n, views, bins, dist, b, x):
    q = (n, views, bins, dist)
    rowsum = _fan_fp64(*q, torch.ones((n, n), device="cuda"))
    colsum = _fan_bp64(*q, torch.ones((views, bins), device="cuda"), False)
    r = b.double() - _fan_fp64(*q, x)
    e = r / (rowsum + MATLAB_EPS)
    new = (x.double() + 2.0 * _fan_bp64(*q, e, False) / (colsum + MATLAB_EPS)).clamp(0.0, 1.0)
    return e, new, r.square().sum(), b.double().square().sum()


def _tv_grad64(x, eps):
    def fd(dim):
        d = torch.zeros_like(x)
        d.narrow(dim, 0, x.shape[dim] - 1).copy_(x.narrow(dim, 1, x.shape[dim] - 1) - x.narrow(dim, 0, x.shape[dim] - 1))
        return d
    d = [fd(a) for a in range(3)]
    inv = 1.0 / torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + eps * eps)
    g = torch.zeros_like(x)
    for a in range(3):
        q = d[a] * inv
        g -= q
        g.narrow(a, 1, x.shape[a] - 1).add_(q.narrow(a, 0, x.shape[a] - 1))
    return g


def _tv64(x, iters, step, eps):
    for _ in range(iters):
        g = _tv_grad64(x, eps)
        x = (x - step * torch.sqrt(x.numel() / g.square().sum()) * g).clamp_min(0.0)
    return x


def _sirt3d64(c, b):
    """SIRT3D: relaxation 1, x >= 0, zero start; the residual is that of the x entering the last iteration."""
    ones_v = torch.ones((c["nz"], c["ns"], c["nt"]), device="cuda")
    rowsum, colsum = _cone_fp64(c, ones_v), _cone_bp64(c, torch.ones_like(b))
    x = torch.zeros_like(ones_v, dtype=F64)
    res = 0.0
    for _ in range(c["iters"]):
        r = b.double() - _cone_fp64(c, x)
        res = float(r.norm() / b.double().norm())
        x = (x + _cone_bp64(c, r / (rowsum + 1e-9)) / (colsum + 1e-9)).clamp_min(0.0)
    return x, res


def _curved64(c, R):
    a = _curved_arrays(c)
    gm, xi, be = (torch.tensor(a[k], device="cuda") for k in ("gama", "xi", "beta"))
    lg, lx, nb = len(gm), len(xi), len(be)
    gint, xint, bint = (float((q[1] - q[0]).abs()) for q in (gm, xi, be))
    D, ds, b0, fan = a["D"], a["ds2d"], a["b0"], a["fan"]
    i = torch.arange(lg, device="cuda")
    filt = torch.empty(R.shape, dtype=F64, device="cuda")
    for x in range(lx):
        pr = ds / math.sqrt(ds * ds + a["xi"][x] ** 2)
        bp, gp, b0p, mg = be[:, None] * pr, gm[None, :] * pr, b0 * pr, fan * pr
        up = torch.sin(math.pi / 4 * bp / (mg / 2 - gp)) ** 2
        down = torch.sin(math.pi / 4 * (math.pi + mg - bp) / (mg / 2 + gp)) ** 2
        W = torch.where((bp >= b0p) & (bp < b0p + mg - 2 * gp), up,
                        torch.where((bp >= b0p + mg - 2 * gp) & (bp <= b0p + math.pi - 2 * gp), torch.ones_like(up),
                                    torch.where((bp > b0p + math.pi - 2 * gp) & (bp <= b0p + math.pi + mg), down,
                                                torch.zeros_like(up))))
        n = torch.arange(-(lg - 1), lg, dtype=F64, device="cuda")
        sn = torch.where(n == 0, torch.ones_like(n), torch.sin(n * gint * pr))
        G = torch.where(n == 0, 2.0 / (math.pi * gint * pr) ** 2 + 0 * n,
                        -2.0 * n * n / math.pi ** 2 / (4 * n * n - 1) / sn ** 2)
        filt[:, x] = gint * pr * ((R[:, x] * (D / pr) * torch.cos(gp) * W) @ G[(lg - 1) + i[None, :] - i[:, None]])
    nn, nz = c["n"], c["nz"]
    half = a["size"][0] // 2
    t = torch.arange(nn, device="cuda", dtype=F64) - 0.5 - float(half)
    it, is_ = t[None, :], t[:, None]
    iz = ((torch.arange(nz, device="cuda", dtype=F64) - 0.5) * (23.0 / nz) - float(23 // 2))[:, None, None]
    acc = torch.zeros((nz, nn, nn), dtype=F64, device="cuda")
    for v in range(nb):
        bt = float(be[v])
        k, s = math.cos(bt), math.sin(bt)
        st, ss = D * math.cos(bt + math.pi / 2), D * math.sin(bt + math.pi / 2)
        l2xy = (it - st) ** 2 + (is_ - ss) ** 2
        L2 = l2xy + iz * iz
        Gm = torch.atan((it * k + is_ * s) / (D - (-it * s + is_ * k)))
        X = ds * iz / torch.sqrt(l2xy)
        ok = ((Gm >= gm.min()) & (Gm < gm.max())) & (X >= xi.min()) & (X < xi.max())
        x1 = torch.floor((X - xi[0]).abs() / xint).long().clamp_(0, lx - 2)
        g1 = torch.floor((Gm - gm[0]).abs() / gint).long().clamp_(0, lg - 2)
        wx1, wx2 = (X - xi[x1]).abs(), (xi[x1 + 1] - X).abs()
        wg1, wg2 = (Gm - gm[g1]).abs(), (gm[g1 + 1] - Gm).abs()
        f = filt[v].reshape(-1)
        o = x1 * lg + g1
        val = wx2 * (wg2 * f[o] + wg1 * f[o + 1]) + wx1 * (wg2 * f[o + lg] + wg1 * f[o + lg + 1])
        val = val / (gint * xint) / L2 * (bint * torch.sqrt(l2xy) / torch.sqrt(L2))
        acc += torch.where(ok, val, torch.zeros_like(val))
    return filt, acc


def _net64(x, y):
    """The network on the stored weights in 64 bits: its output and, with y, the gradients of the mean squared error."""
    d = np.load(PKG / "ctgb" / "weights" / "warmstart_unet.npz")
    par = {k: torch.from_numpy(d[k]).view(torch.bfloat16).double().cuda().requires_grad_(y is not None)
           for k in d.files if k != "meta"}
    F = torch.nn.functional

    def conv(name, t, taps, relu):
        w = par[name + ".w"]
        k = 3 if taps == 27 else 1
        o = F.conv3d(t, w.permute(0, 2, 1).reshape(w.shape[0], w.shape[2], k, k, k), par[name + ".b"], padding=k // 2)
        return F.relu(o) if relu else o

    with torch.set_grad_enabled(y is not None):
        xin = x.double().unsqueeze(1)
        pad = F.pad(xin, (1,) * 6)
        nz, ny, nx = x.shape[1:]
        g = torch.cat([pad[:, :, i:i + nz, j:j + ny, k:k + nx] for i in range(3) for j in range(3) for k in range(3)] +
                      [torch.zeros_like(xin)] * 5, 1)
        e1 = conv("e1b", conv("e1a", g, 1, True), 27, True)
        e2 = conv("e2b", conv("e2a", F.max_pool3d(e1, 2), 27, True), 27, True)
        e3 = conv("e3b", conv("e3a", F.max_pool3d(e2, 2), 27, True), 27, True)
        t = conv("b2", conv("b1", F.max_pool3d(e3, 2), 27, True), 27, True)
        for skip, u, a, b in ((e3, "u3", "d3a", "d3b"), (e2, "u2", "d2a", "d2b"), (e1, "u1", "d1a", "d1b")):
            t = F.interpolate(conv(u, t, 1, False), scale_factor=2, mode="nearest")
            t = conv(b, conv(a, torch.cat([skip, t], 1), 27, True), 27, True)
        out = (t * par["head.w"].view(1, 32, 1, 1, 1)).sum(1) + par["head.b"] + x.double()
        if y is None:
            return out
        ((out - y.double()) ** 2).mean().backward()
    return {"out": out.detach(), "grads": {k: p.grad for k, p in par.items()}}


def exact(case, seed):
    k = case["kind"]
    if k in ("dropin_fbp", "fan_fbp", "fan_sirt"):
        q = (case["n"], case["views"], case["bins"], case["dist"])
        sino = _fan_sino(*q, seed)
        if k != "fan_sirt":
            return _fan_fbp64(*q, sino)
        e, x, _, _ = _fan_sirt64(*q, sino, 0.5 * _volume((1, q[0], q[0]), seed)[0])
        return {"e": e, "x": x}
    if k == "fan_batch":
        if case["slices"] > 16:
            return None                     # over 20 seconds
        got = []
        for i, q in enumerate(_batch_scans(case)):
            q = (*q, 500.0)
            got.append(_fan_sirt64(*q, _fan_sino(*q, seed + i), 0.5 * _volume((1, q[0], q[0]), seed + i)[0]))
        return {"e": torch.cat([g[0].reshape(-1) for g in got]), "x": torch.cat([g[1].reshape(-1) for g in got]),
                "norms": torch.stack([torch.stack([g[2], g[3]]) for g in got])}
    if k in ("unet_forward", "unet_train"):
        if case["nx"] * case["ny"] * case["nz"] > 2 ** 18:
            return None                     # over 20 seconds (64-bit convolutions)
        x, y = _net_input(case, seed)
        return _net64(x, None) if k == "unet_forward" else _net64(x, y)
    if k == "curved":
        f, d = _curved64(case, _curved_input(case, seed))
        return {"filtered": f, "display": d}
    if k == "tv":
        return _tv64(_tv_input(case, seed).double(), case["iters"], 1e-3, 1e-8)
    vox, rays = case["nt"] * case["ns"] * case["nz"], case["views"] * case["cols"] * case["rows"]
    steps = rays * (case["nt"] + case["ns"] + case["nz"])
    if k == "cone_fp" and steps > 6e10:
        return None                         # over 20 seconds
    if k == "cone_fp":
        return _cone_fp64(case, _volume((case["nz"], case["ns"], case["nt"]), seed))
    if vox * case["views"] > 2e10:
        return None                         # over 20 seconds
    b = _cone_sino(case, seed)
    if k == "cone_bp":
        return _cone_bp64(case, b)
    if k == "fdk":
        return _fdk64(case, b)
    x, r = _sirt3d64(case, b)
    return {"x": x, "residual": torch.tensor([r], dtype=F64)}
