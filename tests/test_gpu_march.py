"""The marching kernels (small calls: one launch per pass over time) against
the oracle and against the tile sweeps, which a fixed tile shape selects.

Tolerances: the oracle's as in the other parity tests (gathers and misfit
1e-4 relative L2, gradients 1e-3); against the tile sweeps, whose operations
are the same up to the order of a few FP32 sums, a tenth of those."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

CASES = {
    # strips of 2 and 3 columns, one 32-depth chunk and a remainder
    "narrow": dict(nz=20, nx=13, nPml=6, nSteps=90, n_shots=1),
    # a padded height that is no multiple of 32
    "ragged": dict(nz=37, nx=71, nPml=9, nSteps=120, n_shots=3),
    # chunks and strips without any CPML cell
    "interior": dict(nz=110, nx=150, nPml=12, nSteps=150, n_shots=2),
    # several rounds of a block's warps, strips of different widths in the two passes
    "rounds": dict(nz=177, nx=233, nPml=16, nSteps=70, n_shots=2),
    # as many shots as a pack holds
    "sixteen": dict(nz=40, nx=48, nPml=10, nSteps=80, n_shots=16),
}


def _workload(name):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(seed=21, **CASES[name])
    if name == "ragged":
        w.nPad = 5
        rows = w.nz_pad
        w.vp, w.vp_obs = (np.ascontiguousarray(v[:rows]) for v in (w.vp, w.vp_obs))
        for s in w.shots:  # scattered receivers, two on one cell
            s["z_rec"] = [(7 * r) % (w.nz - 1) for r in range(len(s["x_rec"]))]
            s["x_rec"][1], s["z_rec"][1] = s["x_rec"][0], s["z_rec"][0]
        w.shots[1].update(nSteps=75, win_x0=0, win_x1=59)
        w.shots[1]["z_rec"], w.shots[1]["x_rec"] = [2] * 60, list(range(60))
        w.shots[1]["x_src"] = 30
    return w


@pytest.mark.parametrize("name", sorted(CASES))
def test_marching_matches_oracle_and_tiles(name, gpu_lib, fw, orc, tmp_path):
    w = _workload(name)
    para = w.write_files(str(tmp_path))
    ids = list(range(len(w.shots)))
    lo, mo, ro = w.moduli(w.vp_obs)
    ref = orc.cufd(2, lo, mo, ro, w.stf, ids, para, write_files=True, want_gathers=True)["gathers"]
    lam, mu, rho = w.moduli()
    g = orc.cufd(1, lam, mu, rho, w.stf, ids, para)
    J0 = orc.cufd(0, lam, mu, rho, w.stf, ids, para)["misfit"]
    march, tiles = fw.FwiContext(para, 0), fw.FwiContext(para, 0)
    tiles.set_tile_config([8] * 4)
    tiles.set_tile_rows([1] * 4)
    for a, b, c in zip(march.obs(lo, mo, ro, w.stf, ids, write_files=False), ref,
                       tiles.obs(lo, mo, ro, w.stf, ids, write_files=False)):
        assert rel(a, b) < 1e-4 and rel(a, c) < 1e-5
    out = []
    for ctx in (march, tiles):
        ctx.set_illumination(True)
        r = ctx.misfit_grad(lam, mu, rho, w.stf, ids)
        out.append((*r, ctx.illumination(), ctx.last_launch_count()))
    m, t = out
    assert m[-1] < t[-1]  # the two took different paths
    assert abs(m[0] - J0) <= 1e-4 * abs(J0) and abs(m[0] - t[0]) <= 1e-5 * abs(J0)
    for a, b, k in zip(m[1:5], t[1:5], ("g_lambda", "g_mu", "g_den", "g_stf")):
        assert rel(a, g[k]) < 1e-3 and rel(a, b) < 1e-4, (k, rel(a, g[k]), rel(a, b))
    assert rel(m[5], t[5]) < 1e-5
    again = march.misfit_grad(lam, mu, rho, w.stf, ids)
    assert again[0] == m[0] and all(np.array_equal(a, b) for a, b in zip(again[1:], m[1:5]))
    march.close()
    tiles.close()
