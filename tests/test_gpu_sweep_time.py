"""fwigb_sweep_time launches the sweeps of the last run on its buffers: refused
where there are none, or none any more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _refused(ctx, fw, kinds=range(4)):
    for kind in kinds:
        with pytest.raises(fw.FwiError) as e:
            ctx.sweep_time(kind, 2)
        assert e.value.status == 1


def test_after_a_failed_run_and_new_shots(gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nSteps=40)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    obs = ctx.obs(*w.moduli(w.vp_obs), w.stf, [0, 1], write_files=False)
    _refused(ctx, fw, (2, 3))
    ctx.set_batching(0, 1024)
    with pytest.raises(fw.FwiError):  # not even one shot's wavefields
        ctx.misfit_grad(*w.moduli(), w.stf, [0, 1], obs=obs)
    _refused(ctx, fw)
    ctx.set_batching(0, 0)
    ctx.misfit_grad(*w.moduli(), w.stf, [0, 1], obs=obs)
    assert all(ctx.sweep_time(kind, 2) > 0 for kind in range(4))
    ctx.stage_shots(w.stf, [1], obs=obs[1:])
    _refused(ctx, fw)
    ctx.run(1)
    assert all(ctx.sweep_time(kind, 2) > 0 for kind in range(4))
    ctx.close()


def test_record_of_one_step(gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nSteps=1)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    ctx.set_model(*w.moduli())
    ctx.stage_shots(w.stf, [0, 1], obs=[np.zeros((w.nx, 1), np.float32)] * 2)
    ctx.run(1)
    assert ctx.fetch()[0] == 0.0
    _refused(ctx, fw, (2, 3))  # (there is no step to take back)
    ctx.close()
