"""The network's parameters are FP32 masters with BF16 copies whatever torch's
default type is (a program in double precision sets it to float64)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_parameters_are_fp32_under_a_float64_default():
    from pic_b200 import unet
    torch.set_default_dtype(torch.float64)
    try:
        net = unet.UNet(seed=3)
        net._ensure(1, 16, 16)
        net.a["x0"].normal_(generator=torch.Generator(device="cuda").manual_seed(1))
        z = net.forward().clone()
    finally:
        torch.set_default_dtype(torch.float32)
    for v in net.params.values():
        assert {k: t.dtype for k, t in v.items()} == {"p": torch.float32, "bf": torch.bfloat16, "g": torch.float32,
                                                      "m": torch.float32, "v": torch.float32}
    # the same weights loaded into a network made under the usual default
    other = unet.UNet(seed=0)
    other.load_state(net.state())
    other._ensure(1, 16, 16)
    other.a["x0"].copy_(net.a["x0"])
    torch.cuda.synchronize()
    assert torch.equal(other.forward(), z) and bool(z.any())
