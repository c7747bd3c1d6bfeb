"""The group state keeps to mem_budget_bytes: a budget of one shot's 18
wavefields, 3 gradient arrays and boundary store (4 with the illumination) runs
shot by shot within it, with the results of an unlimited call; a byte less is
refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state_bytes(w, illum):
    """One shot's state with three gradient arrays (and the illumination)."""
    array = -(-w.nz_pad // 32) * 32 * w.nx_pad * 4
    ring = 10 * (w.nx + 4) + 10 * (w.nz + 4 - 10)  # cells of the boundary ring: 5 deep on each side
    return (18 + 3 + illum) * array + w.nSteps * 5 * ring * 4, array


@pytest.mark.parametrize("illum", [False, True])
@pytest.mark.parametrize("nz,nx", [(1000, 1500), (37, 45)])
def test_state_keeps_to_the_budget(nz, nx, illum, gpu_lib, fw, tmp_path):
    import torch
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nz=nz, nx=nx, nPml=12, nSteps=40, n_shots=2, seed=5)
    para = w.write_files(str(tmp_path))
    budget, array = _state_bytes(w, illum)
    out = []
    for limit in (0, budget):
        ctx = fw.FwiContext(para, 0)
        ctx.set_tile_config([8] * 4)
        ctx.set_tile_rows([1] * 4)
        ctx.set_illumination(illum)
        ctx.set_batching(1, limit)
        ctx.set_model(*w.moduli())
        ctx.stage_shots(w.stf, [0, 1], obs=[np.ones((w.nx, w.nSteps), np.float32)] * 2)
        free = torch.cuda.mem_get_info()[0]
        ctx.run(1)
        r = ctx.fetch(grads=True, n_shots=2)
        used = free - torch.cuda.mem_get_info()[0]
        assert ctx.last_group_count() == 2
        out.append((r, ctx.illumination() if illum else None))
        if limit and nz > 500:  # (allocations are in pieces of 2 MB)
            assert used <= limit + array
        if limit:
            ctx.set_batching(1, limit - 1)
            with pytest.raises(fw.FwiError) as e:
                ctx.run(1)
            assert e.value.status == 5
        ctx.close()
    (a, ia), (b, ib) = out
    assert a[0] == b[0] and all(np.array_equal(x, y) and np.abs(x).max() > 0 for x, y in zip(a[1:], b[1:]))
    assert ia is None or np.array_equal(ia, ib)


def test_small_call_in_a_tight_budget(gpu_lib, fw, tmp_path):
    """A call that would march, at the limit: the tile sweeps, to FP32 rounding of the sums."""
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nz=37, nx=45, nPml=12, nSteps=120, n_shots=1, seed=5)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    ctx.obs(*w.moduli(w.vp_obs), w.stf, [0], write_files=True)
    a = ctx.misfit_grad(*w.moduli(), w.stf, [0])
    ctx.set_batching(0, _state_bytes(w, False)[0])
    b = ctx.misfit_grad(*w.moduli(), w.stf, [0])
    assert abs(a[0] - b[0]) <= 1e-5 * a[0]
    for x, y in zip(a[1:], b[1:]):
        assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(y)  # (as in test_gpu_march.py)
    ctx.close()
