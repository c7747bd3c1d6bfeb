"""The kernels between model-shaped arrays and network images against their
NumPy forms. Packing rounds double to FP32 (and BF16) as NumPy and torch do:
equal bits. The features and the gains take a few double operations whose last
bits may differ from NumPy's, rounded to FP32 / BF16 or kept in double: one
unit of the rounding of the largest value, 2^-8 in BF16, and 1e-13 in double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(32, 1), (64, 33), (96, 70)]


def _old_image(a, c_pad):
    out = np.zeros((a.shape[2], a.shape[1], c_pad), dtype=np.float32)
    out[:, :, :a.shape[0]] = np.transpose(a, (2, 1, 0))
    return out.reshape(-1, c_pad)


@pytest.mark.parametrize("nz,nx", SHAPES)
def test_packed_images_are_the_transposed_arrays(nz, nx, gpu_lib, fw):
    import torch
    from fwiflow_gb300.precond import CnnPreconditioner

    net = CnnPreconditioner(nz, nx)
    rng = np.random.default_rng(nz)
    for c, c_pad, dtype in ((5, 16, torch.bfloat16), (3, 3, torch.float32), (1, 1, torch.float32), (16, 16, torch.float32)):
        a = rng.standard_normal((c, nz, nx))
        ref = torch.from_numpy(_old_image(a, c_pad)).to(dtype)
        assert torch.equal(net.to_image(a, c_pad, dtype).cpu(), ref)
    f, t, m = rng.standard_normal((5, nz, nx)), rng.standard_normal((3, nz, nx)), rng.uniform(0, 1, (nz, nx))
    net.stage(f, t, m)
    assert torch.equal(net.x0.cpu(), torch.from_numpy(_old_image(f, 16)).to(torch.bfloat16))
    assert torch.equal(net.target.cpu(), torch.from_numpy(_old_image(t, 3)))
    assert torch.equal(net.mask.cpu(), torch.from_numpy(m.T.reshape(-1).astype(np.float32)))
    with pytest.raises(ValueError):
        net.stage(rng.standard_normal((5, nz + 1, nx)))


@pytest.mark.parametrize("nz,nx", SHAPES)
@pytest.mark.parametrize("kind", ["plain", "empty mask", "dark"])
def test_precondition_matches_numpy(nz, nx, kind, gpu_lib, fw):
    import torch
    from fwiflow_gb300 import precond

    net = precond.CnnPreconditioner(nz, nx, seed=2)
    rng = np.random.default_rng(nx)
    g = [s * rng.standard_normal((nz, nx)) for s in (1e-3, 1.0, 40.0)]
    illum = np.zeros((nz, nx)) if kind == "dark" else rng.uniform(0.0, 3.0, (nz, nx)) ** 4
    mask = np.zeros((nz, nx)) if kind == "empty mask" else (rng.uniform(-1.0, 1.0, (nz, nx))).clip(0.0)
    got = net.precondition(*g, illum, mask)
    x = precond.features(*g, illum, mask)
    ref = torch.from_numpy(_old_image(x, 16)).to(torch.bfloat16).float()
    assert float((net.x0.cpu().float() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    out = net.from_image(net.out, 3)
    want = np.stack(g) * np.exp(np.clip(out, -30.0, 5.0)) * mask
    assert got.shape == want.shape and got.dtype == np.float64
    assert np.abs(got - want).max() <= 1e-13 * max(np.abs(want).max(), 1e-300)
