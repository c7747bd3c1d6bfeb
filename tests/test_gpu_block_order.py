"""The sweeps' block orders (tile by tile over the shots, and back over the
columns and packs), which calls of a few million cells take, against the same
shots one by one, which are too small for them.

Each shot's operations are the same: gathers to 1e-6 relative L2; the shots'
images are summed in another order: misfit and gradients to 1e-5."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

CASES = {
    "by_tile": dict(nz=900, nx=930, nPml=16, nSteps=40, n_shots=3),
    "two_packs": dict(nz=300, nx=520, nPml=16, nSteps=30, n_shots=17),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("rows", [1, 2])
def test_block_order(name, rows, gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(seed=9, **CASES[name])
    para = w.write_files(str(tmp_path))
    ids = list(range(len(w.shots)))
    out = []
    for groups in ([ids], [[k] for k in ids]):
        ctx = fw.FwiContext(para, 0)
        ctx.set_tile_config([8] * 4)
        ctx.set_tile_rows([rows] * 4)
        obs, J, grads = [], 0.0, None
        for g in groups:
            obs += ctx.obs(*w.moduli(w.vp_obs), w.stf, g, write_files=True)
            r = ctx.misfit_grad(*w.moduli(), w.stf, g)
            J += r[0]
            grads = [a.copy() for a in r[1:4]] if grads is None else [a + b for a, b in zip(grads, r[1:4])]
        out.append((obs, J, grads))
        ctx.close()
    (oa, Ja, ga), (ob, Jb, gb) = out
    for a, b in zip(oa, ob):
        assert np.linalg.norm(a) > 0 and rel(a, b) < 1e-6
    assert abs(Ja - Jb) <= 1e-5 * abs(Jb)
    for a, b in zip(ga, gb):
        assert rel(a, b) < 1e-5
