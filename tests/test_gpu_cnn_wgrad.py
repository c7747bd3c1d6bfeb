"""The weight gradient where its blocks take several tiles each (more tiles than
blocks), against the sum of a partial per tile and against PyTorch; FP32 sums over
192,000 pixels in another order: 1e-4 relative L2, as in test_gpu_cnn.py."""
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cip,cop", [(16, 32), (32, 32), (32, 16)])
def test_weight_gradient_over_many_tiles(cip, cop, gpu_lib, fw):
    import torch
    from fwiflow_gb300.precond import CnnPreconditioner

    Hz, Wx = 96, 2000
    net = CnnPreconditioner(Hz, Wx)
    tiles, blocks = gpu_lib.fwigb_cnn_tile_count(Hz, Wx), gpu_lib.fwigb_cnn_wgrad_blocks(Hz, Wx)
    assert 1 < blocks < tiles and net.part.numel() == blocks * 9 * 32 * 32
    torch.manual_seed(cip + cop)
    x = torch.randn(Hz * Wx, cip, device="cuda").to(torch.bfloat16)
    dz = torch.randn(Hz * Wx, cop, device="cuda").to(torch.bfloat16)
    n = 9 * cip * cop
    part, a, b = (torch.full((k,), float("nan"), device="cuda") for k in (tiles * n, n, n))
    s = torch.cuda.current_stream().cuda_stream
    args = x.data_ptr(), dz.data_ptr(), Hz, Wx, cip, cop
    assert gpu_lib.fwigb_cnn_wgrad_partials(*args, part.data_ptr(), s) == 0
    assert gpu_lib.fwigb_cnn_reduce_partials(part.data_ptr(), tiles, n, a.data_ptr(), s) == 0
    assert gpu_lib.fwigb_cnn_wgrad(*args, net.part.data_ptr(), b.data_ptr(), s) == 0
    img = [t.float().reshape(Wx, Hz, -1).permute(2, 1, 0)[None] for t in (x, dz)]
    ref = torch.nn.grad.conv2d_weight(img[0], (cop, cip, 3, 3), img[1], padding=1)
    ref = ref.permute(2, 3, 1, 0).reshape(-1).cpu()  # [tap][ci][co]
    assert rel(a.cpu(), ref) < 1e-4 and rel(b.cpu(), ref) < 1e-4 and rel(b.cpu(), a.cpu()) < 1e-4
