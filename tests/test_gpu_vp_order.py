"""The Vp gradient belongs to the last run and the Vp model it was made under:
calls in any other order, and after a wait that gave up, are refused."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.fixture
def case(gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nz=37, nx=45, nPml=9, nSteps=80, n_shots=2, seed=8)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    ctx.stage_shots(w.stf, [0, 1], obs=ctx.obs(*w.moduli(w.vp_obs), w.stf, [0, 1], write_files=False))
    yield ctx, w
    ctx.close()


def _refused(ctx, fw, status):
    with pytest.raises(fw.FwiError) as e:
        ctx.vp_gradient()
    assert e.value.status == status


def _agrees(ctx, vp):
    from fwiflow_gb300 import inversion

    grads = ctx.fetch(grads=True, n_shots=2)[1:4]
    assert rel(ctx.vp_gradient(), inversion.chain_to_vp(vp, *grads)) < 1e-13  # (as in test_gpu_vp_model.py)


@pytest.mark.parametrize("first", ["vp", "moduli"])
def test_gradient_of_another_model_is_refused(first, case, fw):
    ctx, w = case
    if first == "vp":
        ctx.set_model_vp(w.vp)
    else:
        ctx.set_model(*w.moduli())
    ctx.run(1)
    ctx.set_model_vp(w.vp_obs)
    _refused(ctx, fw, 1)
    ctx.run(1)
    _agrees(ctx, w.vp_obs)
    ctx.set_model(*w.moduli())
    _refused(ctx, fw, 1)


def test_gradient_needs_the_last_run(case, fw):
    ctx, w = case
    ctx.set_model_vp(w.vp)
    _refused(ctx, fw, 1)
    ctx.run(1)
    ctx.run(0)
    _refused(ctx, fw, 1)
    ctx.run(1)
    _agrees(ctx, w.vp)


@pytest.mark.parametrize("fetch_first", [False, True])
def test_gradient_after_a_wait_that_gave_up_is_refused(fetch_first, case, fw):
    ctx, w = case
    ctx.set_model_vp(w.vp)
    ctx.test_inject_wait_timeout(True)
    ctx.run(1)
    if fetch_first:
        with pytest.raises(fw.FwiError):
            ctx.fetch()
    else:
        _refused(ctx, fw, 7)
    _refused(ctx, fw, 1)
    ctx.test_inject_wait_timeout(False)
    ctx.run(1)
    _agrees(ctx, w.vp)
