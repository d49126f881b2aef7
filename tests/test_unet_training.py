"""The training step's sums are fixed: the weight gradients' partial sums and the channel sums take the same terms in
the same order on every route, and a second step starts from the same weights.  Adam divides a gradient by its own
size, so another order of an FP32 sum shows as whole bf16 steps of a few weights, and those as 1e-3 of the next
gradients."""
import pytest

pytestmark = pytest.mark.gpu


def _tensors(cins, cout, nb, nz, ny, nx, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    xs = [torch.relu(torch.randn((nb, nz, ny, nx, c), device="cuda", generator=g)).to(torch.bfloat16) for c in cins]
    return xs, torch.randn((nb, nz, ny, nx, cout), device="cuda", generator=g).to(torch.bfloat16)


def _channel_major(xs, dy, taps, kper):
    """The weight gradient through the channel-major copies."""
    import torch
    from ctgb import _lib, unet
    n, z, y, x, cout = dy.shape
    cin = sum(t.shape[-1] for t in xs)
    dw = torch.zeros((cout, taps, cin), device="cuda")
    xm, x0, xp = unet.shift_copies(xs, taps)
    _, dyt, _ = unet.shift_copies([dy], 1)
    _lib.call("ct_unet_conv3d_wgrad", unet._p(xm), unet._tptr(x0), unet._p(xp), cin, unet._tptr(dyt), cout, n, z, y, x,
              taps, kper, unet._tptr(dw), unet._stream())
    return dw


# One partial sum over all voxels (one addition to dw): the same bits as the channel-major kernel's.  Rows of 16, 32, 48
# (one segment), 64, 128 (two), 192, 240 (three of 80) and 256 voxels (four); several planes and samples per sum.
@pytest.mark.parametrize("cins,cout,taps,nb,nz,ny,nx", [
    ((32,), 32, 27, 1, 3, 5, 64), ((32, 32), 64, 27, 2, 2, 4, 128), ((64,), 128, 27, 1, 4, 8, 32),
    ((32,), 256, 27, 1, 3, 16, 16), ((32,), 32, 27, 1, 2, 8, 48), ((32,), 32, 27, 1, 2, 3, 256),
    ((32,), 64, 27, 1, 2, 4, 192), ((32,), 32, 27, 1, 1, 4, 240), ((32,), 32, 1, 1, 3, 4, 64), ((64, 64), 64, 1, 2, 2, 4, 48),
    ((32,), 32, 27, 1, 4, 1, 64), ((64,), 128, 27, 1, 2, 2, 512), ((128,), 256, 1, 1, 2, 8, 16)])
def test_weight_gradient_sum_is_the_channel_major_one(cins, cout, taps, nb, nz, ny, nx):
    import torch
    from ctgb import unet
    xs, dy = _tensors(cins, cout, nb, nz, ny, nx, nx + cout)
    kper = nb * nz * ny * nx // 64 + 1
    assert unet._wgrad_cl(cins, cout, ny, nx, taps)
    got = unet.conv3d_wgrad(xs, dy, taps, kper=kper)
    assert unet.status() == 0
    assert torch.equal(got, _channel_major(xs, dy, taps, kper))


# Many partial sums, some of which start or end inside a row (64 voxels in rows of 48, 96 or 128) or a plane, or are cut
# short: their own bits are compared through sums of integers of at most 2^24, which every order adds exactly
@pytest.mark.parametrize("kper", [1, 2, 3, 7])
@pytest.mark.parametrize("cin,cout,taps,nz,ny,nx", [(32, 32, 27, 3, 4, 48), (32, 64, 27, 2, 6, 96), (64, 32, 27, 2, 5, 128),
                                                    (64, 128, 27, 3, 8, 32), (64, 32, 1, 3, 4, 48)])
def test_weight_gradient_partial_sums(cin, cout, taps, nz, ny, nx, kper):
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(nx + kper)
    x = torch.randint(-8, 9, (1, nz, ny, nx, cin), device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randint(-8, 9, (1, nz, ny, nx, cout), device="cuda", generator=g).to(torch.bfloat16)
    got = unet.conv3d_wgrad([x], dy, taps, kper=kper)
    assert unet.status() == 0
    assert torch.equal(got, _channel_major([x], dy, taps, kper))


# 32-channel chunks of the input that do not fill the rows of an instruction, one by one: integers again, in FP64
@pytest.mark.parametrize("cin,cout", [(96, 128), (160, 32)])
def test_one_tap_weight_gradient_chunks(cin, cout):
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(cin)
    x = torch.randint(-8, 9, (1, 2, 8, 16, cin), device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randint(-8, 9, (1, 2, 8, 16, cout), device="cuda", generator=g).to(torch.bfloat16)
    ref = dy.double().reshape(-1, cout).t() @ x.double().reshape(-1, cin)
    assert torch.equal(unet.conv3d_wgrad([x], dy, 1, kper=3)[:, 0].double(), ref)


# One block of the channel sums: its voxels added one after the other, in FP32
@pytest.mark.parametrize("c", [8, 32, 64, 128])
def test_channel_sums_keep_their_order(c):
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(c)
    x = torch.randn((256 // c, c), device="cuda", generator=g).to(torch.bfloat16)
    db = torch.zeros(c, device="cuda")
    unet.colsum(x, db)
    ref = torch.zeros(c, device="cuda")
    for row in x.float():
        ref = ref + row
    assert torch.equal(db, ref)


# Two training steps against the same network on the channel-major weight gradients, torch's Adam expressions and torch's
# sum of the skip gradients.  Each side's FP32 atomics add its partial sums in any order, a few 2^-24 of a gradient: 2e-6.
# One of 4 million weights may come out a bf16 step away for that; the second step starts from the same ones.
@pytest.mark.parametrize("shape", [(64, 64, 64), (32, 64, 128)])
def test_two_training_steps_repeat(shape, monkeypatch):
    import torch
    from ctgb import unet, warmstart
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(shape, device="cuda", generator=g)
    y = torch.rand(shape, device="cuda", generator=g)
    nets = warmstart.load(), warmstart.load()
    for _ in range(2):
        grads = []
        for net, plain in zip(nets, (True, False)):
            with monkeypatch.context() as m:
                if plain:
                    m.setattr(unet, "_wgrad_cl", lambda *a: False)
                out = net.forward(x, keep=True)
                grads.append(net.backward((2.0 / out.numel()) * (out - y)))
            # strided gradients take torch's expressions
            net.adam_step({k: torch.stack((v, v), -1)[..., 0] for k, v in grads[-1].items()} if plain else grads[-1], lr=1e-5)
        for k, v in grads[0].items():
            assert float((grads[1][k] - v).norm()) <= 2e-6 * float(v.norm()), k
        assert sum(int((nets[0].wb[k] != nets[1].wb[k]).sum()) for k in nets[0].wb) <= 8
        for net in nets:
            net.load_state_dict({k: v.clone() for k, v in nets[0].params.items()})


# The fused Adam pass is bit for bit torch's expressions
def test_adam_bits():
    import torch
    from ctgb import unet
    g = torch.Generator(device="cuda").manual_seed(11)
    net, twin = unet.UNet3D(), unet.UNet3D()
    net.params = {"a.w": 0.05 * torch.randn(1 << 20, device="cuda", generator=g)}
    twin.params = {k: v.clone() for k, v in net.params.items()}
    for _ in range(3):
        gr = {"a.w": torch.randn(1 << 20, device="cuda", generator=g) * torch.rand(1 << 20, device="cuda", generator=g) ** 8}
        net.adam_step(gr, lr=1e-5)
        twin.adam_step({k: torch.stack((v, v), -1)[..., 0] for k, v in gr.items()}, lr=1e-5)
        assert torch.equal(net.params["a.w"], twin.params["a.w"])
        assert torch.equal(net.wb["a"], twin.wb["a"])
