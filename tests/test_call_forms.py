"""Forms of a call that a kernel's split, its range tests or its kept state must not change: operands that share memory,
steps of either sign, uneven detector samples, calls on other streams, threads and after a device reset."""
import numpy as np
import pytest

from conftest import rel_l2


# The row filter in place: rows of several blocks (600, 1300 columns), few short rows (200 columns, a block per warp),
# rows of one block, the smoothing window, and launch order on rows above its limit
@pytest.mark.gpu
@pytest.mark.parametrize("views,rows,cols,window", [(9, 7, 768, 0), (3, 2, 200, 0), (4, 3, 1300, 5), (40, 64, 128, 0),
                                                    (2, 2, 2100, 0)])
@pytest.mark.parametrize("mode", [0, 1])
def test_row_filter_in_place(views, rows, cols, window, mode):
    import torch
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry, centred_domain, view_angles
    geom = ConeGeometry(8, 8, 8, (8.0, 8.0, 8.0), view_angles(views), centred_domain(cols, 0.05),
                        centred_domain(rows, 0.1), 80.0)
    plan = ConePlan(geom, fdk_filter=mode).set_filter("shepp-logan", window)
    R = torch.rand((views, rows, cols), device="cuda")
    ref = plan.fdk_filter(R)
    assert torch.equal(plan.fdk_filter(R, out=R), ref)


# A negative step moves against the flow, as written: from the same start the two moves are opposite (FP32 rounding of
# values near 0.5: 6e-8 of them, against moves of 0.05).  The ASD-POCS phase with a negative alpha likewise.
@pytest.mark.gpu
def test_tv_flow_steps_of_either_sign():
    import torch
    from ctgb.device import tv_flow, tv_flow_asd
    x0 = 0.5 + 0.2 * torch.randn((9, 20, 33), device="cuda")
    up, down = tv_flow(x0.clone(), 1, -0.05, lo=-1e9), tv_flow(x0.clone(), 1, 0.05, lo=-1e9)
    assert float((down - x0).abs().max()) > 0.01
    assert float((up + down - 2 * x0).abs().max()) <= 4e-7
    got = []
    for alpha in (-0.2, 0.2):
        x, prev = x0.clone(), x0 + 0.1
        state = torch.tensor([alpha, 0.0, 0.0], dtype=torch.float64, device="cuda")
        tv_flow_asd(x, prev, torch.empty_like(x), torch.zeros(2, dtype=torch.float64, device="cuda"), state, 1, lo=-1e9)
        got.append(x - x0)
    assert float(got[1].abs().max()) > 0.001
    assert float((got[0] + got[1]).abs().max()) <= 4e-7


# A detector that the image's shadow passes, with a first spacing wider than the rest (the grid it implies runs 0.7 to 22
# bins past the last sample, as 12000 even float samples' does by 4): pixel-views past the last sample get nothing.
# FP32 against the reference's FP64 arithmetic on smooth rows: rel-L2 <= 1e-5, as for even samples.
@pytest.mark.gpu
@pytest.mark.parametrize("n,views,bins,down,first", [(64, 64, 90, False, 1.02), (64, 40, 333, True, 1.02),
                                                     (65, 37, 90, True, 1.5), (64, 40, 50, False, 2.0)])
def test_fan_backprojection_past_uneven_samples(oracle, n, views, bins, down, first):
    import torch
    from ctgb.batch import FanBatch
    from ctgb.device import FanPlan
    from ctgb.geometry import FanGeometry
    half = 0.35 * n
    step = np.full(bins - 1, 1.0)
    step[0] = first
    P = np.concatenate([[0.0], np.cumsum(step)])
    P = (P / P[-1] * 2 - 1) * half
    P = -P if down else P
    beta = np.arange(1, views + 1) * (2 * np.pi / views)
    size, D = np.array([float(n), float(n)]), 2.5 * n
    phase = np.random.default_rng(bins).uniform(0, 6, (views, 1))
    R = (1.5 + np.cos(phase + np.linspace(0, 5, bins)[None, :])).astype(np.float32)
    b32, p32 = beta.astype(np.float32), P.astype(np.float32)
    geom = FanGeometry(n, n, tuple(size), beta, P, D)
    plan, d = FanPlan(geom), torch.from_numpy(R).cuda()
    got = plan.bp(d)
    assert rel_l2(got.cpu().numpy(), oracle.fan_bp(R, b32, p32, size, (n, n), D)) <= 1e-5
    filt = oracle.fbpfan_filter(R, p32, D, mode=0)
    assert rel_l2(plan.fbp(d, filter_mode=0).cpu().numpy(), oracle.fbpfan_bp(filt, b32, p32, size, (n, n), D)) <= 1e-5
    assert torch.equal(FanBatch([geom]).bp(d.reshape(-1)), got.reshape(-1))


# Detector columns that lie closer than the first two, so that a voxel's column weights sum to less than 1, under a
# volume of flat voxels whose z faces limit most chords: FP32 against the reference's FP64 arithmetic
@pytest.mark.gpu
@pytest.mark.parametrize("rest,down", [(0.5, False), (0.8, True), (0.05, False)])
def test_cone_backprojection_uneven_columns(oracle, rest, down):
    import torch
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry
    nt, ns, nz, cols, rows, views = 16, 12, 400, 60, 80, 7
    P = np.concatenate([[0.0, 1.0], 1.0 + rest * np.arange(1, cols - 1)])
    P = (P / P[-1] * 2 - 1) * 14.0
    P = -P if down else P
    xi = (np.arange(rows) - (rows - 1) / 2) * (56.0 / rows)
    beta = np.arange(1, views + 1) * (2 * np.pi / views)
    size, D = (16.0, 12.0, 40.0), 100.0
    g = ConeGeometry(nt, ns, nz, size, beta, P, xi, D)
    R = np.random.default_rng(cols).random(g.sino_shape).astype(np.float32)
    got = ConePlan(g).bp(torch.from_numpy(R).cuda()).cpu().numpy()
    assert rel_l2(got, oracle.cone_bp(R, g.beta, g.P, g.xi, size, D, (nz, ns, nt))) <= 1e-5


# The curved-detector stages of two scans queued one behind the other on a stream of their own, which the copies of the
# second scan's tables do not wait for: each gives what it gives alone
@pytest.mark.gpu
def test_curved_fdk_scans_back_to_back_on_a_stream():
    import torch
    from ctgb.device import fdkui_bp, fdkui_filter

    def scan(lg, lx, nb, dg):
        gama = (np.arange(lg) - (lg - 1) / 2) * dg
        fan = abs(gama[-1] - gama[0])
        return dict(gama=gama, xi=(np.arange(lx) - (lx - 1) / 2) * 1.5, beta=np.arange(nb) * ((np.pi + fan) / (nb - 1)),
                    fan=fan, R=torch.rand((nb, lx, lg), dtype=torch.float64, device="cuda"))

    def run(c):
        rows = fdkui_filter(c["R"], c["xi"], c["gama"], c["beta"], 0.0, c["fan"], 110.0, 200.0)
        rows.nan_to_num_(0.0, 0.0, 0.0)
        return rows, fdkui_bp(rows, c["xi"], c["gama"], c["beta"], 110.0, 200.0, np.array([96, 96, 21], np.int32), 20)

    a, b = scan(700, 24, 300, 0.0012), scan(700, 24, 300, 0.0011)
    alone = [run(a), run(b)]
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        got = [run(c) for c in (a, b, a, b)]
    s.synchronize()
    for k, (rows, disp) in enumerate(got):
        assert torch.equal(rows, alone[k % 2][0]) and torch.equal(disp, alone[k % 2][1])


RESET_CHILD = r'''
import ctypes as C, sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/ct-research_gb300"]
from ctgb import _lib
lib = _lib.lib()
rt = C.CDLL("libcudart.so.13")
rt.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
p = lambda a: a.ctypes.data_as(C.c_void_p)
n, nb, bins = 24, 20, 31
beta = (np.arange(1, nb + 1) * (2 * np.pi / nb)).astype(np.float32)
P = np.linspace(-30, 30, bins).astype(np.float32)
R = np.random.default_rng(1).random((nb, bins)).astype(np.float32)
size, out = np.array([24.0, 24.0]), []
for k in range(3):
    if k:
        # memory of other owners at the addresses that the reset set free, in the sizes that the call uses
        blocks = []
        for nbytes in [4 * nb * bins, 4 * n * n, 512, 2048, 1 << 16, 1 << 20] * 8:
            d = C.c_void_p()
            assert rt.cudaMalloc(C.byref(d), nbytes) == 0
            mark = np.full(nbytes, 0xA5, np.uint8)
            assert rt.cudaMemcpy(d, p(mark), nbytes, 1) == 0
            blocks.append((d, nbytes))
    img = np.zeros((n, n), np.float32)
    assert lib.ct_FBPfan(p(img), p(R), p(P), p(beta), nb, bins, p(size), n, n, C.c_double(70.0)) == 0, lib.ct_last_error()
    out.append(img)
    if k:
        for d, nbytes in blocks:
            got = np.empty(nbytes, np.uint8)
            assert rt.cudaMemcpy(p(got), d, nbytes, 2) == 0
            assert (got == 0xA5).all(), nbytes
    assert rt.cudaDeviceReset() == 0
assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2]) and out[0].any()
print("kept apart")
'''


# A 2D host-pointer call after a device reset that nobody announced, with the freed addresses in other hands: the same
# image, and the others' memory untouched
@pytest.mark.gpu
def test_2d_calls_after_a_device_reset():
    import subprocess
    import sys
    from pathlib import Path
    r = subprocess.run([sys.executable, "-c", RESET_CHILD, str(Path(__file__).resolve().parents[1])], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "kept apart" in r.stdout, r.stdout + r.stderr


# 2D calls of eight threads on six scans, two of them alike, with a release among them: every result is the one of a call
# alone
@pytest.mark.gpu
def test_2d_calls_of_several_threads():
    from concurrent.futures import ThreadPoolExecutor
    from ctgb import _lib, ops
    rng = np.random.default_rng(5)
    scans = []
    for n, nb, bins in ((24, 20, 31), (33, 17, 40), (24, 20, 31), (200, 90, 300), (64, 50, 91), (24, 21, 31)):
        P = np.linspace(-0.9 * n, 0.9 * n, bins).astype(np.float32)
        beta = (np.arange(1, nb + 1) * (2 * np.pi / nb)).astype(np.float32)
        scans.append((rng.random((nb, bins)).astype(np.float32), beta, P, np.array([float(n)] * 2), n))

    def call(k):
        R, beta, P, size, n = scans[k % len(scans)]
        return ops.FBPfan(R.ravel(), beta, P, size, n, n, 3.0 * n), ops.BackprojectionFan2D(R.ravel(), beta, P, size, n, n, 3.0 * n)

    alone = [call(k) for k in range(len(scans))]
    _lib.call("ct_dropin_release")
    with ThreadPoolExecutor(8) as ex:
        for k, got in enumerate(ex.map(call, range(60))):
            for a, b in zip(got, alone[k % len(scans)]):
                assert np.array_equal(a, b)
            if k == 20:
                _lib.call("ct_dropin_release")


# The chunk that is reported is the one in effect: automatic chunks where the set-up's records bound them (64 views of
# 1024^2 columns, evened out), and a set value up to the view count, in one pass
@pytest.mark.gpu
def test_backprojection_chunk_in_effect():
    import torch
    from ctgb import _lib
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry, centred_domain, view_angles
    lib = _lib.lib()
    geom = ConeGeometry(1024, 1024, 3, (100.0, 100.0, 0.3), view_angles(100), centred_domain(60, 3.0),
                        centred_domain(6, 0.2), 400.0)
    R, got = torch.rand(geom.sino_shape, device="cuda"), []
    for views, chunk, launches in ((0, 50, 3 + 3 * 2), (100, 100, 6), (1000, 100, 6), (70, 70, 9)):
        plan = ConePlan(geom).set_bp_chunk(views)
        assert plan.bp_chunk_views() == chunk and plan.launches_per_pair() == launches
        got.append(plan.bp(R))
        size = lib.ct_cone_plan_workspace_bytes(plan._h)
        need = chunk * (8 * 60 * 6 + 32 * 1024 * 1024)
        assert need <= size <= need + (1 << 20)
    for v in got[1:]:
        assert rel_l2(v.cpu().numpy(), got[0].cpu().numpy()) <= 1e-6


# Columns of many slices: the row quotient is stepped from the set-up's first slice.  On rows that alternate between 0 and
# 1 an error of the quotient is one of the value; FP32 arithmetic leaves 2^-22 at most.
@pytest.mark.gpu
@pytest.mark.parametrize("nz", [500, 60000])
def test_cone_backprojection_of_tall_columns(oracle, nz):
    import torch
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry
    rows, size, D = 6000, (2.0, 2.0, 50.0), 100.0
    P, xi = np.arange(8) - 3.5, (np.arange(rows) - (rows - 1) / 2) * 0.01
    for view in range(12):
        g = ConeGeometry(2, 2, nz, size, np.array([0.3 + 0.5 * view]), P, xi, D)
        R = np.zeros(g.sino_shape, np.float32)
        R[:, ::2] = 1.0
        got = ConePlan(g).bp(torch.from_numpy(R).cuda()).cpu().numpy()
        assert rel_l2(got, oracle.cone_bp(R, g.beta, g.P, g.xi, size, D, (nz, 2, 2))) <= 2.0 ** -22


# Threads whose z lie about the mid-plane of a volume of tall voxels close to the source, where the chord is no quadratic
# in z: 4, 8 and 32 slices per thread against the reference's FP64 arithmetic
@pytest.mark.gpu
@pytest.mark.parametrize("nt,nz,rz", [(3, 20, 2.0), (3, 4, 0.7), (200, 48, 3.0), (130, 40, 1.5), (3, 32, 0.3)])
def test_cone_backprojection_about_the_mid_plane(oracle, nt, nz, rz):
    import torch
    from ctgb.device import ConePlan
    from ctgb.geometry import ConeGeometry
    views, cols, rows = 5, 80, 90
    size, D = (float(nt), float(nt), nz * rz), 1.2 * nt
    P = (np.arange(cols) - (cols - 1) / 2) * (4.0 * nt / cols)
    xi = (np.arange(rows) - (rows - 1) / 2) * (9.0 * nz * rz / rows)
    g = ConeGeometry(nt, nt, nz, size, np.arange(1, views + 1) * (2 * np.pi / views), P, xi, D)
    R = np.random.default_rng(nz).random(g.sino_shape).astype(np.float32)
    got = ConePlan(g).bp(torch.from_numpy(R).cuda()).cpu().numpy()
    assert rel_l2(got, oracle.cone_bp(R, g.beta, g.P, g.xi, size, D, (nz, nt, nt))) <= 1e-6
