"""The training step keeps its bits: Adam divides a gradient by its own size, so another rounding or order of an FP32 sum
shows as whole bf16 steps of a few weights, and those as 1e-3 of the next gradients."""
import pytest

pytestmark = pytest.mark.gpu


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
