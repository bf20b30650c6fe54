"""The U-Net's flat parameter vectors: a pass takes addresses in them, so one
that does not hold every parameter is refused before anything is launched."""
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", ["w", "wb", "g"])
@pytest.mark.parametrize("change", [lambda t: t[:100], lambda t: t[:0], lambda t: t.view(2, -1)])
def test_vectors_that_hold_too_little(name, change):
    from seispie_b200.unet import UNet
    net = UNet("cpu")
    setattr(net, name, change(getattr(net, name)))
    with pytest.raises(RuntimeError, match="UNet." + name):
        if name == "g":
            net.acts, net.shape = {}, (1, 8, 8)
            net.backward(torch.zeros(1, 8, 8))
        else:
            net.forward(torch.zeros(1, 3, 8, 8))
