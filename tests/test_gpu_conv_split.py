"""Forward convolutions of narrow images with their output channels split over
CTAs: channel counts that do not divide evenly, one pixel tile to more tiles
than SMs.  FP32 references on the CPU, tolerances as for the kernels' other
tests (2e-3 of the largest, 1e-4 relative L2)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1, 16, 16), (1, 4, 4, 48, 40), (1, 8, 8, 256, 256), (1, 16, 32, 80, 384),
                                   (2, 5, 40, 64, 112), (1, 3, 100, 16, 300), (1, 20, 96, 32, 48), (3, 8, 16, 128, 80),
                                   (5, 64, 64, 64, 64), (4, 127, 60, 16, 96)])
def test_split_channels(cuda_ctx, shape):
    from pupiloptixlab_gb300 import denoiser as dnm
    n, h, w, cin, cout = shape
    g = torch.Generator().manual_seed(h * w + cout)
    x = torch.randn(n, h, w, cin, generator=g).to(torch.bfloat16)
    wt = (0.1 * torch.randn(cout, 9, cin, generator=g)).to(torch.bfloat16)
    b = torch.randn(cout, generator=g)
    pad = torch.zeros((cout + 15) // 16 * 16, 9, cin, dtype=torch.bfloat16)
    pad[:cout] = wt
    y = dnm.conv3x3_forward(x.cuda(), pad.cuda(), b.cuda(), cout, out_f32=True).cpu()
    ref = F.conv2d(x.float().permute(0, 3, 1, 2), wt.float().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2), b, padding=1)
    ref = ref.permute(0, 2, 3, 1)
    assert float((y - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
    assert float((y - ref).norm()) <= 1e-4 * float(ref.norm())
