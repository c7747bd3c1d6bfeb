"""Arrays that are not plain model-shaped ones take NumPy's way to the network's
images: what it accepts (broadcast channels, masks with a leading axis, flat or of
one value) is accepted, with its values, and what it refuses is refused. A
stand-in without a GPU: any call into the library fails."""
import numpy as np
import pytest

H, W = 32, 5


@pytest.fixture
def net(fw):
    torch = pytest.importorskip("torch")
    from fwiflow_gb300.precond import N_OUT, CnnPreconditioner

    n = CnnPreconditioner.__new__(CnnPreconditioner)
    n.Hz, n.Wx, n.npix, n.dev, n.lib = H, W, H * W, torch.device("cpu"), None
    n.x0 = torch.zeros((n.npix, 16), dtype=torch.bfloat16)
    n.target, n.mask = torch.zeros((n.npix, N_OUT)), torch.zeros(n.npix)
    n.forward = lambda: torch.ones((n.npix, 16))
    return n


def _image(a, c_pad):
    out = np.zeros((W, H, c_pad), dtype=np.float32)
    out[:, :, :a.shape[0]] = np.transpose(a, (2, 1, 0))
    return out.reshape(-1, c_pad)


RNG = np.random.default_rng(0)
F = RNG.standard_normal((5, 1, W))  # broadcast along z


@pytest.mark.parametrize("mask", [RNG.uniform(size=(1, H, W)), RNG.uniform(size=H * W), np.full((1, 1), 0.5)])
def test_accepted(mask, net):
    import torch

    net.stage(F, F[:3], mask)
    assert torch.equal(net.x0, torch.from_numpy(_image(F, 16)).to(torch.bfloat16))
    assert np.array_equal(net.target.numpy(), _image(F[:3], 3))
    assert np.array_equal(net.mask.numpy(), np.broadcast_to(mask.T.reshape(-1).astype(np.float32), H * W))
    net.stage(np.empty((0, H, W)))
    assert not net.x0.any()
    assert np.array_equal(net.to_image(F, 16, torch.float32).numpy(), _image(F, 16))


@pytest.mark.parametrize("feats,mask", [(F[:, 0], None), (np.ones((5, H + 1, W)), None), (np.ones((17, 1, 1)), None),
                                        (F, np.ones(W)), (F, np.ones((H, W - 1)))])
def test_refused(feats, mask, net):
    with pytest.raises((ValueError, RuntimeError)):
        net.stage(feats, mask=mask)


def test_precondition(net):
    from fwiflow_gb300 import precond

    g = list(RNG.standard_normal((3, 1, W)))
    illum, mask = RNG.uniform(size=(1, W)), np.ones((1, W))
    got = net.precondition(*g, illum, mask)
    assert np.allclose(got, np.stack(g) * np.exp(1.0) * np.ones((H, W)), rtol=1e-15)
    assert np.array_equal(net.x0.float().numpy(),
                          net.to_image(precond.features(*g, illum, mask), 16, net.x0.dtype).float().numpy())
    full = list(RNG.standard_normal((3, H, W)))
    with pytest.raises(Exception):  # (an illumination that is no array)
        net.precondition(*full, 1.0, np.ones((H, W)))
