"""Vp models and gradients formed on the device (fwigb_set_model_vp,
fwigb_fetch_vp_gradient) against the NumPy forms of inversion.py. The chain
rule is ~15 double operations per cell, each within an ulp or two of NumPy's:
1e-13 relative. The models agree to the last bit of a double before they are
rounded to FP32, so the misfits agree to FP32 rounding of single cells: 1e-6."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,nPml", [(20, 13, 6), (37, 70, 9), (64, 40, 16)])
@pytest.mark.parametrize("masked", [True, False])
def test_vp_model_and_gradient(nz, nx, nPml, masked, gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import inversion, synthetic

    w = synthetic.tiny(nz=nz, nx=nx, nPml=nPml, nSteps=80, n_shots=2, seed=8)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    obs = ctx.obs(*w.moduli(w.vp_obs), w.stf, [0, 1], write_files=False)
    rng = np.random.default_rng(1)
    mask = rng.uniform(-0.2, 1.2, w.vp.shape).clip(0.0, 1.0) if masked else None
    vmin, vmax = np.quantile(w.vp, [0.1, 0.8])
    v = np.clip(w.vp_obs * (1 - mask) + w.vp * mask, vmin, vmax) if masked else w.vp
    J0, gl, gm, gd, _ = ctx.misfit_grad(*inversion.moduli_of_vp(v), w.stf, [0, 1], obs=obs)
    with pytest.raises(fw.FwiError):
        ctx.vp_gradient()
    ctx.stage_shots(w.stf, [0, 1], obs=obs)
    ctx.set_model_vp(w.vp, *((w.vp_obs, mask, vmin, vmax) if masked else ()))
    ctx.run(1)
    J, al, am, ad, _ = ctx.fetch(grads=True, n_shots=2)
    assert abs(J - J0) <= 1e-6 * J0
    for a, b in ((al, gl), (am, gm), (ad, gd)):
        assert rel(a, b) < 1e-5
    ref = inversion.chain_to_vp(v, al, am, ad) * (mask if masked else 1.0)
    assert rel(ctx.vp_gradient(), ref) < 1e-13
    with pytest.raises(fw.FwiError):  # the Courant number of a model twice as fast
        ctx.set_model_vp(3.0 * w.vp)
    ctx.close()
