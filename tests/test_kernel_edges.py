"""Kernels at the sizes where their tiles, groups and rules change, against the
oracle (FP32 against the reference's FP64 arithmetic: rel-L2 <= 1e-5)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


# (nt, ns), views, bins, detector half width over the image half width, descending, first spacing over the rest
FAN_BP = [
    ((5, 3), 1, 2, 1.6, False, 1.0),          # fewer views than groups, one bin pair
    ((8, 4), 7, 3, 1.6, True, 1.0),
    ((33, 1), 8, 4, 1.6, False, 1.0),         # two pixel tiles, the second of one lane
    ((31, 33), 37, 50, 1.6, False, 1.0),
    ((64, 65), 40, 333, 0.7, True, 1.0),      # truncated detector: off-detector pixels and edge bins
    ((64, 64), 64, 90, 1.6, False, 1.02),     # uneven samples
    ((48, 96), 128, 70, 1.6, False, 1.0),     # views on the diagonals: ties of the pixel edges
]


@pytest.mark.parametrize("shape,views,bins,width,down,first", FAN_BP)
def test_fan_backprojection_groups_and_edges(oracle, shape, views, bins, width, down, first):
    import torch
    from ctgb.device import FanPlan
    from ctgb.geometry import FanGeometry
    nt, ns = shape
    rng = np.random.default_rng(nt * views + bins)
    half = width * 0.5 * max(nt, ns)
    step = np.full(bins - 1, 1.0)
    step[0] = first
    P = np.concatenate([[0.0], np.cumsum(step)])
    P = (P / P[-1] * 2 - 1) * half
    P = P[::-1].copy() if down else P
    beta = np.arange(1, views + 1) * (2 * np.pi / views)
    size, D = np.array([float(nt), float(ns)]), 2.5 * max(nt, ns)
    # smooth rows: the FP32 detector coordinate (~1e-7 of the scan's extent) then costs
    # ~1e-6; on white noise it costs its error in bins, 1.3e-5 at these 0.14 mm bins
    phase = rng.uniform(0, 6, (views, 1))
    R = (1.5 + np.cos(phase + np.linspace(0, 5, bins)[None, :])).astype(np.float32)
    b32, p32 = beta.astype(np.float32), P.astype(np.float32)
    plan = FanPlan(FanGeometry(nt, ns, tuple(size), beta, P, D))
    d = torch.from_numpy(R).cuda()
    assert rel_l2(plan.bp(d).cpu().numpy(), oracle.fan_bp(R, b32, p32, size, (ns, nt), D)) <= TOL
    filt = oracle.fbpfan_filter(R, p32, D, mode=0)
    assert rel_l2(plan.fbp(d, filter_mode=0).cpu().numpy(), oracle.fbpfan_bp(filt, b32, p32, size, (ns, nt), D)) <= TOL


# bins around the 4-output groups, the P-tiles (128 fan, 256 cone) and the longest single-pass row; views around the
# residual row tile of 128
@pytest.mark.parametrize("views,bins", [(1, 2), (3, 5), (130, 127), (128, 130), (2, 1023), (2, 1024), (2, 1025)])
@pytest.mark.parametrize("scale", [1.0, 1e-35, 1e33])
def test_row_filter_tiles_and_scales(oracle, views, bins, scale):
    """Both orders of the pre-weight on rows at the edges of the kernel's tiles, scaled to the ends of the normal
    float range (the kernel scales each row to 1)."""
    import torch
    from ctgb.device import FanPlan
    from ctgb.geometry import FanGeometry
    rng = np.random.default_rng(views + bins)
    P = np.linspace(-40.0, 40.0, bins)
    beta = np.arange(1, views + 1) * (2 * np.pi / views)
    R = (rng.random((views, bins)) * scale).astype(np.float32)
    p32, b32 = P.astype(np.float32), beta.astype(np.float32)
    plan = FanPlan(FanGeometry(8, 8, (8.0, 8.0), beta, P, 100.0))
    for mode in (0, 1):
        filt = oracle.fbpfan_filter(R, p32, 100.0, mode=mode)
        ref = oracle.fbpfan_bp(filt, b32, p32, (8.0, 8.0), (8, 8), 100.0)
        got = plan.fbp(torch.from_numpy(R).cuda(), filter_mode=mode).cpu().numpy()
        assert rel_l2(got, ref) <= TOL


def test_row_filter_infinities_stay_in_their_row():
    """An infinity or NaN spoils its own row's outputs only."""
    import torch
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry, centred_domain, view_angles
    plan = ConePlan(ConeGeometry(4, 4, 4, (4.0, 4.0, 4.0), view_angles(3), centred_domain(300, 0.1),
                                 centred_domain(5, 0.1), 50.0), fdk_filter=0)
    R = torch.rand((3, 5, 300), device="cuda")
    good = plan.fdk_filter(R)
    bad = R.clone()
    bad[1, 2, 7] = float("inf")
    bad[2, 0, 299] = float("nan")
    out = plan.fdk_filter(bad)
    assert not torch.isfinite(out[1, 2]).any() and not torch.isfinite(out[2, 0]).any()
    out[1, 2], out[2, 0] = good[1, 2], good[2, 0]
    assert torch.equal(out, good)


# (nt, ns, nz), views, (cols, rows), detector rows per voxel in z (below and above one), descending rows, source distance
CONE_BP = [
    ((33, 5, 16), 3, (40, 24), 0.7, False, 5.0),        # one z tile of 16, a second t tile of one column
    ((31, 4, 17), 4, (40, 30), 1.3, False, 5.0),        # the last tile holds one slice
    ((20, 18, 40), 9, (30, 20), 0.6, True, 5.0),        # rows descending: the quotient falls with z
    ((24, 24, 64), 8, (40, 30), 0.9, False, 2.0),       # the cone leaves the detector in z, diagonal views
    ((300, 260, 33), 2, (200, 60), 0.8, False, 4.0),    # wide enough for 32 z per thread
    ((300, 260, 70), 2, (200, 90), 2.2, False, 4.0),
]


@pytest.mark.parametrize("shape,views,det,rows,down,dist", CONE_BP)
def test_cone_backprojection_tiles_and_row_steps(oracle, shape, views, det, rows, down, dist):
    import torch
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry
    nt, ns, nz = shape
    rng = np.random.default_rng(nt + nz)
    cols, nx = det
    P = (np.arange(cols) - (cols - 1) / 2) * (1.5 * max(nt, ns) / cols)
    xi = (np.arange(nx) - (nx - 1) / 2) / rows
    xi = xi[::-1].copy() if down else xi
    beta = np.arange(1, views + 1) * (2 * np.pi / views)
    size, D = (float(nt), float(ns), float(nz)), dist * max(nt, ns)
    g = ConeGeometry(nt, ns, nz, size, beta, P, xi, D)
    R = rng.random(g.sino_shape).astype(np.float32)
    d = torch.from_numpy(R).cuda()
    assert rel_l2(ConePlan(g).bp(d).cpu().numpy(), oracle.cone_bp(R, g.beta, g.P, g.xi, size, D, (nz, ns, nt))) <= TOL
    for sticky in (0, 1):
        ref = oracle.fdk_bp(R, g.beta, g.P, g.xi, size, D, (nz, ns, nt), sticky=sticky)
        assert rel_l2(ConePlan(g, fdk_bp=sticky).fdk_bp(d).cpu().numpy(), ref) <= TOL


def _curved(lg, lx, views):
    """Equiangular detector of lg gammas and lx rows around a 90 mm display at distance 300."""
    gama = -(np.arange(lg) - (lg - 1) / 2) * (0.4 / lg)
    xi = (np.arange(lx) - (lx - 1) / 2) * (60.0 / lx)
    beta = 0.03 + np.arange(views) * (4.2 / views)
    return gama, xi, beta, 0.03, 1.001 * abs(gama[-1] - gama[0]), 300.0, 560.0


@pytest.mark.parametrize("lg", [2, 3, 5, 64, 66, 127, 1030])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e30])
def test_curved_filter_row_lengths(oracle, lg, scale):
    """Rows around the 4-output groups, the 64-sample sums and the block's 1024 outputs: the filter rounds a ~2^-40
    sum to a float, so it agrees with the FP64 sum to a float's rounding (6e-8 rms of each value)."""
    import torch
    from ctgb.device import fdkui_filter
    gama, xi, beta, b0, fan, D, ds = _curved(lg, 3, 4)
    R = (1.0 + np.random.default_rng(lg).random((4, 3, lg))) * scale
    ref = oracle.fdkui_filter(R, xi, gama, beta, b0, fan, D, ds)
    got = fdkui_filter(torch.from_numpy(R).cuda(), xi, gama, beta, b0, fan, D, ds).cpu().numpy()
    assert rel_l2(got, ref) <= 2e-7


def test_curved_backprojection_in_view_chunks(oracle):
    """More views than the records of one launch hold (170 at 512 x 512 columns), one and 17 slices."""
    import torch
    from ctgb.device import fdkui_bp
    for n, nz, views in ((512, 1, 172), (40, 17, 9)):
        gama, xi, beta, _, _, D, ds = _curved(60, 8, views)
        D, ds = D * n / 90, ds * n / 90
        xi = xi * (n / 90)
        size = np.array([n, n, 2 if nz == 1 else n // 4], np.int32)
        rc = np.random.default_rng(n).random((views, 8, 60)).astype(np.float32)
        ref = oracle.fdkui_bp(rc, size, nz, beta, D, ds, gama, xi)
        got = fdkui_bp(torch.from_numpy(rc).cuda(), xi, gama, beta, D, ds, size, nz).cpu().numpy()
        assert rel_l2(got, ref) <= TOL


@pytest.mark.parametrize("n,views,bins", [(5, 4, 3), (64, 4, 41), (97, 8, 33), (300, 4, 601)])
@pytest.mark.parametrize("parallel", [False, True])
def test_grazing_rays_by_warps_and_split_rays(oracle, n, views, bins, parallel):
    """Rays on grid lines (odd bins, views on the axes) around 32 steps and more, short rays that are not split, and a
    sinogram above the size that is."""
    import torch
    from ctgb.device import FanPlan, ParPlan
    from ctgb.geometry import FanGeometry
    if parallel and n % 2:
        pytest.skip("no parallel ray on a grid line")
    views = 256 if bins == 601 and not parallel else views     # parallel: every ray runs along a grid line
    rng = np.random.default_rng(n)
    img = rng.random((n, n)).astype(np.float32)
    ang = np.arange(1, views + 1) * (2 * np.pi / views)
    P = (np.arange(bins) - (bins - 1) // 2) * 1.0
    if parallel:
        plan = ParPlan(n, n, (1.0, 1.0), ang, P)
        ref = oracle.par_fp(img, ang, P, (float(n), float(n)))
    else:
        plan = FanPlan(FanGeometry(n, n, (float(n), float(n)), ang, P, 3.0 * n))
        ref = oracle.fan_fp(img, ang, P, (float(n), float(n)), 3.0 * n)
    got = plan.fp(torch.from_numpy(img).cuda()).cpu().numpy()
    assert plan.grazing_rays() > 0 or n % 2
    assert rel_l2(got, ref) <= TOL


# (nz, ny, nx) around the gradient's warps (30 columns, 4 rows, 16 rows per block) and runs of planes
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 5, 7), (2, 4, 30), (3, 17, 31), (40, 16, 61), (33, 33, 90), (70, 3, 121)])
@pytest.mark.parametrize("offset", [0, 1])
def test_tv_gradient_tiles_and_alignment(shape, offset):
    """One sub-step, its move 0.05 rms on values of ~0.5: FP32 rounding leaves ~1e-6 of the move.  offset: x starts 4
    bytes off a 16-byte boundary."""
    import torch
    from ctgb.device import tv_flow
    from oracle.oracle import tv_flow as tv_ref
    n = int(np.prod(shape))
    x = (0.5 + 0.2 * np.random.default_rng(n).normal(size=shape)).astype(np.float32)
    buf = torch.zeros(n + 4, device="cuda")
    t = buf[offset:offset + n].view(shape)
    t.copy_(torch.from_numpy(x))
    got = tv_flow(t, 1, 0.05, 1e-8, -1e9).cpu().numpy().astype(np.float64) - x
    ref = tv_ref(x, 1, 0.05, 1e-8, -1e9) - x.astype(np.float64)
    assert rel_l2(got, ref) <= TOL


def test_dropin_2d_plans_kept_between_calls(oracle):
    """More geometries than plans are kept, of equal sizes but other contents, from several threads, twice, and after a
    release."""
    from concurrent.futures import ThreadPoolExecutor
    from ctgb import _lib, ops
    rng = np.random.default_rng(11)
    size, n, nb, bins = np.array([24.0, 24.0]), 24, 20, 31
    cases = []
    for k in range(6):
        beta = (np.arange(1, nb + 1) * (2 * np.pi / nb) + 0.01 * k).astype(np.float32)
        P = (np.linspace(-30, 30, bins) * (1 + 0.01 * k)).astype(np.float32)
        R = rng.random((nb, bins)).astype(np.float32)
        D = 70.0 + (k == 5)
        filt = oracle.fbpfan_filter(R, P, D, mode=1)
        cases.append((R, beta, P, D, oracle.fbpfan_bp(filt, beta, P, size, (n, n), D),
                      oracle.fan_bp(R, beta, P, size, (n, n), D)))

    def check(k):
        R, beta, P, D, fbp, bp = cases[k]
        return (rel_l2(ops.FBPfan(R.ravel(), beta, P, size, n, n, D), fbp.ravel()),
                rel_l2(ops.BackprojectionFan2D(R.ravel(), beta, P, size, n, n, D), bp.ravel()))

    for rounds in range(2):
        with ThreadPoolExecutor(4) as ex:
            for errs in ex.map(check, [0, 0, 1, 2, 3, 4, 5, 0, 3]):
                assert max(errs) <= TOL
        _lib.call("ct_dropin_release")


# channel-major x-shifted copies: whole 16-byte groups, channel tiles that end inside 32, 64-voxel blocks that end
# inside a volume, an x of one group, and sizes and views that take the element-wise kernel.  The copies are exact.
@pytest.mark.gpu
@pytest.mark.parametrize("c,nb,nz,ny,nx,off", [(32, 2, 3, 5, 8, 0), (40, 1, 2, 3, 24, 8), (8, 1, 1, 1, 8, 0),
                                               (64, 2, 4, 4, 64, 32), (32, 1, 2, 3, 12, 0), (12, 2, 2, 2, 16, 4),
                                               (32, 1, 3, 3, 72, 1)])
def test_shift_copies_groups_and_remainders(c, nb, nz, ny, nx, off):
    import torch
    from ctgb import _lib
    from ctgb.unet import _tptr, _stream
    g = torch.Generator(device="cuda").manual_seed(c + nx)
    x = torch.randn((nb, nz, ny, nx, c), device="cuda", generator=g).to(torch.bfloat16)
    ctot = c + off + 3
    outs = [torch.full((nb, ctot, nz, ny, nx), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    for skip in (None, 0, 2):
        ptr = [None if skip == k else _tptr(o) for k, o in enumerate(outs)]
        for o in outs:
            o.fill_(7.0)
        _lib.call("ct_unet_shift_t", _tptr(x), c, nb, nz, ny, nx, *ptr, ctot, off, _stream())
        t = x.permute(0, 4, 1, 2, 3)
        for k, o in enumerate(outs):
            ref = torch.full_like(o, 7.0)
            if k != skip:
                want = torch.zeros_like(t)
                if k == 0:
                    want[..., 1:] = t[..., :-1]
                elif k == 1:
                    want[...] = t
                else:
                    want[..., :-1] = t[..., 1:]
                ref[:, off:off + c] = want
            assert torch.equal(o, ref), (k, skip)


# z-marching convolution: one slice, fewer slices than accumulators, chunks along z with several items per CTA, two
# inputs, a split output with masks.  Products of bf16 numbers are exact in FP32, so only the order of the sums
# differs from torch's FP32 result: 27 cin terms of size ~1 err by at most 27 cin 2^-24 of their absolute sum, far
# below the bf16 step; outputs equal but for roundings at a tie (at least 99 in 100, 2e-3 of the norm).
@pytest.mark.gpu
@pytest.mark.parametrize("c1,c2,cout,nb,nz,ny,nx,split,masked", [
    (32, 0, 32, 5, 1, 128, 128, None, False), (32, 0, 32, 3, 2, 128, 128, None, True),
    (32, 32, 32, 2, 3, 128, 128, None, False), (32, 0, 64, 2, 5, 96, 128, 32, True), (32, 0, 64, 2, 70, 32, 64, 48, True),
    (32, 32, 32, 2, 45, 64, 64, None, True), (32, 0, 32, 3, 33, 48, 72, 16, False), (64, 0, 64, 1, 29, 48, 64, 48, True)])
def test_conv3d_marching_along_z(c1, c2, cout, nb, nz, ny, nx, split, masked):
    import torch
    import torch.nn.functional as F
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(c1 + c2 + cout + nz)
    bf = torch.bfloat16

    def rnd(*shape):
        return torch.randn(shape, device="cuda", generator=g)

    x1 = rnd(nb, nz, ny, nx, c1).to(bf)
    x2 = rnd(nb, nz, ny, nx, c2).to(bf) if c2 else None
    w = (rnd(cout, 27, c1 + c2) * 0.05).to(bf)
    bias = rnd(cout)
    co = [cout] if split is None else [split, cout - split]
    masks = tuple(rnd(nb, nz, ny, nx, k).to(bf) for k in co) if masked else ()
    masks = masks + (None,) * (2 - len(masks))
    out = unet.conv3d(x1, w, bias, relu=not masked, x2=x2, split=split, masks=masks)
    assert unet.status() == 0
    x = x1 if x2 is None else torch.cat((x1, x2), -1)
    ref = F.conv3d(x.float().permute(0, 4, 1, 2, 3), w.float().permute(0, 2, 1).reshape(cout, c1 + c2, 3, 3, 3), bias,
                   padding=1).permute(0, 2, 3, 4, 1)
    ref = ref if masked else ref.relu()
    outs, at = ((out,) if split is None else out), 0
    for k, o in enumerate(outs):
        r = ref[..., at:at + co[k]]
        at += co[k]
        if masked:
            r = r * (masks[k].float() > 0)
        r = r.to(bf).float()
        err = float((o.float() - r).norm() / r.norm())
        assert err <= 2e-3 and float((o.float() == r).float().mean()) >= 0.99, err


# weight gradient from channels-last tensors: one slice, partial sums of one tile and of a number that does not divide
# the tiles, more items than CTAs, two inputs, three chunks, one tap, a y that the tiles do not fit.  Against FP64 sums
# of the same bf16 values: FP32 sums of at most 2^14 products between two additions, so 2^14 2^-24 = 1e-3 of the
# absolute sum at the very worst and, rounding at random, about 2^7 2^-24 = 8e-6 of the norm; 1e-4 leaves ten times that.
@pytest.mark.gpu
@pytest.mark.parametrize("cins,cout,taps,nb,nz,ny,nx,kper", [
    ((32,), 32, 27, 1, 1, 16, 8, 1), ((32,), 64, 27, 2, 2, 16, 24, 6), ((64, 32), 32, 27, 1, 7, 32, 16, 10),
    ((32,), 32, 27, 3, 21, 64, 72, None), ((32, 32), 64, 1, 2, 5, 48, 40, 14), ((128,), 128, 27, 1, 3, 16, 16, 4),
    ((32,), 32, 27, 1, 3, 24, 16, 4)])
def test_conv3d_wgrad_channels_last(cins, cout, taps, nb, nz, ny, nx, kper):
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(sum(cins) + cout + nz)
    xs = [torch.randn((nb, nz, ny, nx, c), device="cuda", generator=g).to(torch.bfloat16) for c in cins]
    dy = torch.randn((nb, nz, ny, nx, cout), device="cuda", generator=g).to(torch.bfloat16)
    dw = unet.conv3d_wgrad(xs, dy, taps, kper=kper)
    assert unet.status() == 0
    r = 1 if taps == 27 else 0
    x = torch.nn.functional.pad(torch.cat(xs, -1).double(), (0, 0) + (r,) * 6)
    ref = torch.zeros_like(dw, dtype=torch.float64)
    for t in range(taps):
        a, b, e = (t // 9, t // 3 % 3, t % 3) if r else (0, 0, 0)
        ref[:, t] = dy.double().reshape(-1, cout).t() @ x[:, a:a + nz, b:b + ny, e:e + nx].reshape(-1, sum(cins))
    assert float((dw.double() - ref).norm() / ref.norm()) <= 1e-4


# channel sums: 8 channels per thread at every channel count, lanes that the voxels do not fill, an unaligned tensor
# (the 2-byte kernel).  FP32 sums of n values of size 1 against FP64: n 2^-24 of the absolute sum at the very worst.
@pytest.mark.gpu
@pytest.mark.parametrize("c,n,off", [(8, 1, 0), (8, 70001, 0), (32, 33, 0), (32, 500003, 0), (128, 4097, 0), (256, 7, 0),
                                     (256, 100003, 0), (16, 1001, 2), (4, 999, 0)])
def test_channel_sums(c, n, off):
    import torch
    from ctgb import _lib
    from ctgb.unet import _tptr, _stream
    g = torch.Generator(device="cuda").manual_seed(c + n)
    x = torch.randn(n * c + off, device="cuda", generator=g).to(torch.bfloat16)[off:]
    db = torch.ones(c, device="cuda")
    _lib.call("ct_unet_colsum", _tptr(x), c, n, _tptr(db), _stream())
    v = x.reshape(n, c).double()
    assert bool(((db.double() - 1 - v.sum(0)).abs() <= (n + 8) * 2.0 ** -24 * (1 + v.abs().sum(0))).all())


# one fused Adam pass against the same formula in FP64: a dozen FP32 roundings (2^-24 each) of m, v and the step; the
# bf16 copy is the rounding of the new parameter.  The element-wise path of a non-contiguous gradient agrees with it.
@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 255, 70001])
def test_adam_pass_and_flipped_weights(n):
    import torch
    from ctgb import unet
    net = unet.UNet3D()
    g = torch.Generator(device="cuda").manual_seed(n)
    net.params = {"a.w": torch.randn(n, device="cuda", generator=g), "head.b": torch.randn(1, device="cuda", generator=g)}
    ref = {k: v.double() for k, v in net.params.items()}
    other = {k: v.clone() for k, v in net.params.items()}
    s = net.adam
    m = {k: torch.zeros_like(v) for k, v in ref.items()}
    v2 = {k: torch.zeros_like(v) for k, v in ref.items()}
    twin = unet.UNet3D()
    twin.params = other
    for t in range(1, 4):
        gr = {k: torch.randn(v.shape, device="cuda", generator=g) for k, v in net.params.items()}
        net.adam_step(gr, lr=1e-2)
        twin.adam_step({k: torch.stack((v, v), -1)[..., 0] for k, v in gr.items()}, lr=1e-2)
        for k in ref:
            gd = gr[k].double()
            m[k] = s.b1 * m[k] + (1 - s.b1) * gd
            v2[k] = s.b2 * v2[k] + (1 - s.b2) * gd * gd
            ref[k] -= 1e-2 * (m[k] / (1 - s.b1 ** t)) / ((v2[k] / (1 - s.b2 ** t)).sqrt() + s.eps)
            tol = 3 * 2.0 ** -24 * (ref[k].abs() + 1) * 4
            assert bool(((net.params[k].double() - ref[k]).abs() <= tol).all())
            assert bool(((twin.params[k].double() - ref[k]).abs() <= tol).all())
    assert set(net.wb) == set(twin.wb) == {"a"} and torch.equal(net.wb["a"], net.params["a.w"].to(torch.bfloat16))
    for shape in ((32, 27, 64), (64, 1, 32), (40, 27, 33)):
        net.wb["w"] = torch.randn(shape, device="cuda", generator=g).to(torch.bfloat16)
        net.wt.pop("w", None)
        assert torch.equal(net._wt("w"), net.wb["w"].flip(1).transpose(0, 2).contiguous())


# the first convolution from the volume itself: the same instructions on the same bf16 values as the gathered tensor's
# 1-tap convolution, so the same bits; one tile, tiles across x rows, slices and samples, thin volumes.
@pytest.mark.gpu
@pytest.mark.parametrize("nb,nz,ny,nx,relu,biased", [(1, 1, 1, 128, True, True), (1, 16, 16, 16, True, True),
                                                     (2, 5, 16, 24, False, True), (3, 64, 48, 80, True, False),
                                                     (1, 2, 64, 1, True, True)])
def test_conv_first_matches_gathered_taps(nb, nz, ny, nx, relu, biased):
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(nz + nx)
    vol = torch.randn((nb, nz, ny, nx), device="cuda", generator=g)
    w = torch.randn((32, 1, 32), device="cuda", generator=g)
    w[:, :, 27:] = 0
    w = w.to(torch.bfloat16)
    bias = torch.randn(32, device="cuda", generator=g) if biased else None
    out = unet.conv_first(vol, w, bias, relu)
    assert unet.status() == 0
    taps = unet.im2col27(vol).reshape(1, 1, -1, 128, 32)      # as rows of 128 voxels: a shape the 1-tap kernel takes
    assert torch.equal(out.reshape(-1), unet.conv3d(taps, w, bias, relu=relu, ntaps=1).reshape(-1))


# the head taken from the convolution's accumulators: the same bf16 values summed in the same order as from the stored
# activation, so the same bits; one slice, fewer slices than accumulators, several items per group, no base.
@pytest.mark.gpu
@pytest.mark.parametrize("nb,nz,ny,nx,base", [(1, 1, 16, 8, True), (2, 5, 32, 24, False), (2, 37, 64, 72, True)])
def test_conv_head_without_stored_activation(nb, nz, ny, nx, base):
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(nz)
    x = torch.randn((nb, nz, ny, nx, 32), device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn((32, 27, 32), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    bias, hw, hb = (torch.randn(k, device="cuda", generator=g) for k in (32, 32, 1))
    b = torch.randn((nb, nz, ny, nx), device="cuda", generator=g) if base else None
    out = unet.conv3d_head(x, w, bias, True, hw, hb, b)
    assert unet.status() == 0
    assert torch.equal(out, unet.head(unet.conv3d(x, w, bias, relu=True), hw, hb, b))


# one Adam launch for many tensors: more than one launch's table, sizes around a block's 1024 elements; against the
# element-wise expressions (a dozen FP32 roundings apart).  Pooling gradient added to a skip gradient: the same bits as
# the two passes.
@pytest.mark.gpu
def test_adam_of_many_tensors_and_pool_gradient_sum():
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(5)
    sizes = [1, 3, 1023, 1024, 1025, 2048, 5000] * 8
    net, twin = unet.UNet3D(), unet.UNet3D()
    net.params = {f"{i}.w": torch.randn(n, device="cuda", generator=g) for i, n in enumerate(sizes)}
    twin.params = {k: v.clone() for k, v in net.params.items()}
    for _ in range(2):
        gr = {k: torch.randn(v.shape, device="cuda", generator=g) for k, v in net.params.items()}
        net.adam_step(gr, lr=1e-2)
        twin.adam_step({k: torch.stack((v, v), -1)[..., 0] for k, v in gr.items()}, lr=1e-2)
    for k, v in net.params.items():
        assert bool(((v - twin.params[k]).abs() <= 24 * 2.0 ** -24 * (v.abs() + 1)).all()), k
        assert torch.equal(net.wb[k[:-2]], v.to(torch.bfloat16))
    x = torch.relu(torch.randn((2, 4, 6, 8, 40), device="cuda", generator=g)).to(torch.bfloat16)
    y = unet.pool2(x)
    dy = torch.randn(y.shape, device="cuda", generator=g).to(torch.bfloat16)
    skip = torch.randn(x.shape, device="cuda", generator=g).to(torch.bfloat16)
    assert torch.equal(unet.pool2_bwd(x, y, dy, skip), skip + unet.pool2_bwd(x, y, dy))


# 8 z per thread (enough blocks at 8, too few at 16), a last tile of one and of three slices, and 4 z with a last tile
# of one: the bounds of the other tile sizes' test above
@pytest.mark.gpu
@pytest.mark.parametrize("shape,views,det,rows,down,dist", [
    ((100, 100, 41), 5, (130, 60), 0.9, False, 3.0), ((97, 101, 43), 4, (120, 90), 1.4, True, 3.0),
    ((40, 30, 9), 6, (60, 24), 0.8, False, 2.0)])
def test_cone_backprojection_small_scans(oracle, shape, views, det, rows, down, dist):
    test_cone_backprojection_tiles_and_row_steps(oracle, shape, views, det, rows, down, dist)
