"""The sweeps' edge tiles at sizes where they can go wrong: tiles that hold
CPML, ring and interior cells together, tiles of CPML cells only, a last row
alone in its pair, columns past the stencil domain, a source and receivers in
the CPML; for every tile shape, against the oracle.

Tolerances as in the other parity tests (gathers and misfit 1e-4 relative L2,
gradients 1e-3); the illumination, which the oracle does not have, against the
marching kernels, whose operations are the same, at 1e-5."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

CASES = {
    # CPML thinner than a tile, odd height and width
    "thin": (dict(nz=37, nx=45, nPml=5, nSteps=90, n_shots=2), 3),
    # CPML that fills tiles of 32 and of 64 rows
    "thick": (dict(nz=70, nx=61, nPml=33, nSteps=80, n_shots=1), 4),
    # a height that is no multiple of 32 and the source in the CPML
    "ragged": (dict(nz=51, nx=70, nPml=32, nSteps=80, n_shots=2), 7),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_edge_tiles(name, gpu_lib, fw, orc, tmp_path):
    from fwiflow_gb300 import synthetic

    kw, pad = CASES[name]
    w = synthetic.tiny(seed=5, **kw)
    w.nPad = pad
    w.vp, w.vp_obs = (np.ascontiguousarray(v[:w.nz_pad]) for v in (w.vp, w.vp_obs))
    if name == "ragged":
        w.shots[0].update(z_src=-20, x_src=-9)
        w.shots[0]["z_rec"][3], w.shots[0]["x_rec"][3] = -12, 20
    para = w.write_files(str(tmp_path))
    ids = list(range(len(w.shots)))
    lo, mo, ro = w.moduli(w.vp_obs)
    ref = orc.cufd(2, lo, mo, ro, w.stf, ids, para, write_files=True, want_gathers=True)["gathers"]
    lam, mu, rho = w.moduli()
    g = orc.cufd(1, lam, mu, rho, w.stf, ids, para)
    J0 = orc.cufd(0, lam, mu, rho, w.stf, ids, para)["misfit"]
    ctx = fw.FwiContext(para, 0)
    ctx.set_illumination(True)
    ctx.misfit_grad(lam, mu, rho, w.stf, ids)
    ill = ctx.illumination()
    for width in (4, 8, 16):
        for rows in (1, 2):
            ctx.set_tile_config([width] * 4)
            ctx.set_tile_rows([rows] * 4)
            for a, b in zip(ctx.obs(lo, mo, ro, w.stf, ids, write_files=False), ref):
                assert rel(a, b) < 1e-4, (width, rows)
            r = ctx.misfit_grad(lam, mu, rho, w.stf, ids)
            assert abs(r[0] - J0) <= 1e-4 * abs(J0)
            for a, k in zip(r[1:5], ("g_lambda", "g_mu", "g_den", "g_stf")):
                assert rel(a, g[k]) < 1e-3, (width, rows, k, rel(a, g[k]))
            assert rel(ctx.illumination(), ill) < 1e-5


def test_sweep_time_refuses_backward_sweeps_without_a_ring(gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nSteps=20)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    ctx.obs(*w.moduli(), w.stf, [0, 1], write_files=False)
    assert ctx.sweep_time(0, 2) > 0
    for kind in (2, 3):
        with pytest.raises(Exception, match="backward"):
            ctx.sweep_time(kind, 2)
