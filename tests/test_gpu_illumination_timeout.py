"""The illumination of a run whose wait gave up is refused, as its other results are."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fetch_first", [False, True])
def test_illumination_after_a_wait_that_gave_up(fetch_first, gpu_lib, fw, tmp_path):
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nSteps=60)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    ctx.set_illumination(True)
    ctx.set_model(*w.moduli())
    ctx.stage_shots(w.stf, [0, 1], with_obs=False)
    ctx.test_inject_wait_timeout(True)
    ctx.run(2)
    for status in (7, 1):
        with pytest.raises(fw.FwiError) as e:
            ctx.fetch(misfit=False) if fetch_first and status == 7 else ctx.illumination()
        assert e.value.status == status
    ctx.test_inject_wait_timeout(False)
    ctx.run(2)
    assert ctx.illumination().max() > 0
    ctx.close()
