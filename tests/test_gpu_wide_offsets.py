"""The sweeps' form for arrays of 4 GB and more, forced on small grids: edge
tiles, sources and receivers inside fast tiles and windows against the oracle
(through the tests of the usual form), the block orders, graph replay against
eager launches, and what the autotuner picks."""
import numpy as np
import pytest

import test_gpu_batching as batching
import test_gpu_block_order as block_order
import test_gpu_edge_tiles as edge_tiles
import test_gpu_parity as parity

pytestmark = pytest.mark.gpu


@pytest.fixture
def wide(fw):
    class Package:
        FwiError = fw.FwiError

        @staticmethod
        def FwiContext(*args):
            ctx = fw.FwiContext(*args)
            ctx.test_wide_offsets(True)
            return ctx

    return Package


@pytest.mark.parametrize("name", sorted(edge_tiles.CASES))
def test_edge_tiles(name, gpu_lib, wide, orc, tmp_path):
    edge_tiles.test_edge_tiles(name, gpu_lib, wide, orc, tmp_path)


@pytest.mark.parametrize("test", [parity.test_every_tile_shape_with_deep_source_and_receivers,
                                  batching.test_windows_and_record_lengths_match_oracle,
                                  batching.test_batched_graph_replay_is_identical,
                                  batching.test_illumination_matches_oracle])
def test_interior_and_windows(test, gpu_lib, wide, orc, tmp_path):
    test(gpu_lib, wide, orc, tmp_path)


@pytest.mark.parametrize("name", sorted(block_order.CASES))
def test_block_order(name, gpu_lib, wide, tmp_path):
    block_order.test_block_order(name, 1, gpu_lib, wide, tmp_path)


def test_shapes_and_graph(gpu_lib, fw, tmp_path):
    """The autotuner takes the one shape that there is; a graph of one form is not replayed for the other."""
    from fwiflow_gb300 import synthetic

    w = synthetic.tiny(nz=64, nx=96, nPml=12, nSteps=60, n_shots=2)
    ctx = fw.FwiContext(w.write_files(str(tmp_path)), 0)
    obs = ctx.obs(*w.moduli(w.vp_obs), w.stf, [0, 1], write_files=False)
    ctx.test_wide_offsets(True)
    a = ctx.misfit_grad(*w.moduli(), w.stf, [0, 1], obs=obs)
    assert ctx.last_launch_count() > w.nSteps  # (not marching)
    for shape, one in ((ctx.tile_config(), 8), (ctx.tile_rows(), 1)):
        assert [shape[k] for k in (0, 1, 3)] == [one] * 3
    ctx.set_tile_config([16] * 4)
    ctx.set_tile_rows([2] * 4)
    for enable in (False, True, False):
        ctx.test_wide_offsets(enable)
        b = ctx.misfit_grad(*w.moduli(), w.stf, [0, 1], obs=obs)
        assert abs(a[0] - b[0]) <= 1e-6 * a[0]
        for x, y in zip(a[1:], b[1:]):
            assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)
    ctx.close()
