"""Small calls march; here the checks that were written for the sweeps' tiles run
on these, with a fixed tile shape: golden fixtures, odd sizes, determinism, graph
replay, the bounded wait, windows and uneven records, groups, illumination."""
import pytest

import test_gpu_batching as batching
import test_gpu_failures as failures
import test_gpu_parity as parity

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 2])
def tiles(request, fw):
    """The package, with contexts whose tile shape is fixed (one or two depths a thread)."""
    class Package:
        FwiError = fw.FwiError

        @staticmethod
        def FwiContext(*args):
            ctx = fw.FwiContext(*args)
            ctx.set_tile_config([8] * 4)
            ctx.set_tile_rows([request.param] * 4)
            return ctx

    return Package


@pytest.mark.parametrize("name", ["tiny_elastic", "tiny_acoustic", "tiny_window", "tiny_filter", "tiny_srcupd",
                                  "tiny_srcupd_filter"])
def test_golden(name, gpu_lib, tiles, orc, tmp_path):
    parity.test_cuda_matches_reference_golden(name, gpu_lib, tiles, orc, tmp_path)


@pytest.mark.parametrize("case", [dict(nz=20, nx=33, nPml=6, nSteps=120, n_shots=1, seed=3),
                                  dict(nz=37, nx=70, nPml=9, nSteps=160, n_shots=3, seed=4)])
def test_irregular(case, gpu_lib, tiles, orc, tmp_path):
    parity.test_cuda_matches_oracle_irregular(case, gpu_lib, tiles, orc, tmp_path)


@pytest.mark.parametrize("test", [parity.test_cuda_repeatable_and_deterministic,
                                  parity.test_cuda_graph_replay_is_identical,
                                  batching.test_memory_budget_splits_groups])
def test_without_oracle(test, gpu_lib, tiles, tmp_path):
    test(gpu_lib, tiles, tmp_path)


@pytest.mark.parametrize("test", [batching.test_windows_and_record_lengths_match_oracle,
                                  batching.test_batched_graph_replay_is_identical,
                                  batching.test_illumination_matches_oracle])
def test_with_oracle(test, gpu_lib, tiles, orc, tmp_path):
    test(gpu_lib, tiles, orc, tmp_path)


@pytest.mark.parametrize("n_shots", [1, 2])
def test_wait_timeout(n_shots, gpu_lib, tiles, tmp_path):
    failures.test_wait_timeout_is_reported_and_the_context_recovers(n_shots, gpu_lib, tiles, tmp_path)
