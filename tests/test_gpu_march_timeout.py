"""The marching kernels' bounded wait (between neighbouring strips) runs out
under the test hook, and ends the call with a status; in an aperture window, one
shot and several, with and without a graph."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("window,n_shots", [(True, 1), (False, 1), (False, 3)])
def test_wait_for_a_strip_runs_out(window, n_shots, graphs, gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nz=40, nx=60, nPml=10, nSteps=60, n_shots=3, seed=31)
    if window:
        w.shots[0].update(win_x0=0, win_x1=27, x_src=9, z_rec=[2] * 8, x_rec=list(range(8)))
    ids = list(range(n_shots))
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    ctx.set_graphs(graphs)
    ctx.set_model(*w.moduli())
    ctx.stage_shots(w.stf, ids, obs=[np.zeros((len(s["x_rec"]), w.nSteps), np.float32) for s in w.shots[:n_shots]])
    ctx.run(1)
    ref = ctx.fetch(grads=True, n_shots=n_shots)
    assert ctx.last_launch_count() < w.nSteps  # (it marches)
    ctx.test_inject_wait_timeout(True)
    for kind in (1, 0):
        ctx.synchronize()
        t = time.perf_counter()
        ctx.run(kind)
        with pytest.raises(fw.FwiError) as e:
            ctx.fetch()
        assert e.value.status == 7 and "bounded wait" in str(e.value)
        assert 0.02 <= time.perf_counter() - t < 1.0  # the hook's wait of 20 ms ended, and nobody else waited long
    ctx.test_inject_wait_timeout(False)
    ctx.run(1)
    got = ctx.fetch(grads=True, n_shots=n_shots)
    assert got[0] == ref[0] and all(np.array_equal(a, b) for a, b in zip(got[1:], ref[1:]))
    ctx.close()
