"""The network's launches set up beside the ones before them and read their
weights before they wait: a forward call right behind a change of the
weights gives, bit for bit, what a network made with those weights gives."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,batch", [(8, 16, 1), (24, 48, 3), (64, 384, 2)])
def test_forward_behind_new_weights(H, W, batch):
    import torch
    from vdropimpact_b200 import learned

    g = torch.Generator(device="cuda").manual_seed(H + W)
    x, t = (torch.randn(batch, H, W, device="cuda", generator=g) for _ in range(2))
    net, fresh = learned.UNet(H, W, batch=batch, seed=3), learned.UNet(H, W, batch=batch, seed=4)
    p = fresh.get_params()
    want = fresh.forward(x).clone()
    for _ in range(3):
        net.forward(x)
        net.set_params(p)
        assert torch.equal(net.forward(x), want)
        for k in range(3):
            net.train_step(x, t, 1e-2)
            got = net.forward(x).clone()
        fresh.set_params(net.get_params())
        assert torch.equal(got, fresh.forward(x))
        fresh.set_params(p)
