"""Convolution kernels at the edges of their tiles: rows per halo tile with one
to many chunks, channel counts whose weights stay resident or stream, image
heights and widths around the tiles; the weight gradient's 32 x 4 and 16 x 8
tiles, chunk widths 16, 32 and 64 with a partial last chunk, and its bias sums.
References in FP32 on the CPU; tolerances as for the kernels' other tests:
products of BF16 values summed in FP32 (2e-3 of the largest, 1e-4 relative L2)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf16(shape, g, scale=1.0):
    return (torch.randn(shape, generator=g) * scale).to(torch.bfloat16)


def _rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("rows", ["", "1", "2", "3", "4"])
@pytest.mark.parametrize("shape", [(1, 5, 129, 16, 32), (1, 9, 131, 48, 48), (2, 6, 256, 112, 48), (1, 4, 140, 192, 64),
                                   (1, 7, 128, 128, 128), (1, 3, 130, 32, 3)])
def test_forward_halo_tiles(cuda_ctx, monkeypatch, rows, shape):
    from pupiloptixlab_gb300 import denoiser as dnm
    if rows:
        monkeypatch.setenv("PT_CONV_HALO_ROWS", rows)
    n, h, w, cin, cout = shape
    g = torch.Generator().manual_seed(h * w + cin)
    x, wt, b = _bf16((n, h, w, cin), g), _bf16((cout, 9, cin), g, 0.1), torch.randn(cout, generator=g)
    pad = torch.zeros((cout + 15) // 16 * 16, 9, cin, dtype=torch.bfloat16)
    pad[:cout] = wt
    y = dnm.conv3x3_forward(x.cuda(), pad.cuda(), b.cuda(), cout, out_f32=True).cpu()
    ref = F.conv2d(x.float().permute(0, 3, 1, 2), wt.float().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2), b, padding=1)
    ref = ref.permute(0, 2, 3, 1)
    assert float((y - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
    assert _rel(y, ref) <= 1e-4


@pytest.mark.parametrize("shape", [(1, 3, 16, 16, 16), (2, 9, 48, 48, 32), (1, 5, 32, 80, 32), (1, 7, 160, 112, 48),
                                   (1, 2, 137, 32, 16), (2, 4, 64, 64, 96), (1, 6, 32, 128, 256), (1, 4, 16, 16, 128)])
def test_weight_gradient_tiles(cuda_ctx, shape):
    from pupiloptixlab_gb300 import denoiser as dnm
    n, h, w, cin, cout = shape
    g = torch.Generator().manual_seed(h * w + cout)
    x, dy = _bf16((n, h, w, cin), g), _bf16((n, h, w, cout), g)
    dw, db = (t.cpu() for t in dnm.conv3x3_backward_weights(x.cuda(), dy.cuda()))
    wr, br = torch.zeros(cout, cin, 3, 3, requires_grad=True), torch.zeros(cout, requires_grad=True)
    F.conv2d(x.float().permute(0, 3, 1, 2), wr, br, padding=1).backward(dy.float().permute(0, 3, 1, 2))
    ref = wr.grad.permute(0, 2, 3, 1).reshape(cout, 9, cin)
    assert float((dw - ref).abs().max()) <= 2e-3 * float(ref.abs().max())
    assert _rel(dw, ref) <= 1e-4 and _rel(db, br.grad) <= 1e-4


@pytest.mark.parametrize("rows", ["2", "3", "4"])
@pytest.mark.parametrize("shape", [(2, 7, 130, 16, 32), (1, 9, 256, 32, 64), (1, 6, 140, 48, 48)])
def test_bf16_rows_agree(cuda_ctx, monkeypatch, rows, shape):
    """BF16 outputs with ReLU and masked data gradients of halo tiles with several
    rows: bit for bit those of one-row tiles."""
    from pupiloptixlab_gb300 import denoiser as dnm
    n, h, w, cin, cout = shape
    g = torch.Generator().manual_seed(h + w)
    x, wt, b = _bf16((n, h, w, cin), g).cuda(), _bf16((cout, 9, cin), g, 0.1).cuda(), torch.randn(cout, generator=g).cuda()
    dy, mask = _bf16((n, h, w, cout), g).cuda(), _bf16((n, h, w, cin), g).cuda()
    outs = []
    for r in ("1", rows):
        monkeypatch.setenv("PT_CONV_HALO_ROWS", r)
        outs.append((dnm.conv3x3_forward(x, wt, b, cout, relu=True), dnm.conv3x3_backward_data(dy, wt, cin, mask)))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


def test_many_halo_tiles_a_cta(cuda_ctx, monkeypatch):
    """More than three tiles a CTA at any number of rows (both accumulators, the ring across tiles)."""
    from pupiloptixlab_gb300 import denoiser as dnm
    n, h, w, cin, cout = 1, 1021, 600, 16, 32
    g = torch.Generator().manual_seed(17)
    x, wt, b = _bf16((n, h, w, cin), g), _bf16((cout, 9, cin), g, 0.1), torch.randn(cout, generator=g)
    ref = F.conv2d(x.float().permute(0, 3, 1, 2), wt.float().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2), b, padding=1)
    ref = ref.permute(0, 2, 3, 1)
    for rows in ("1", "2", "4"):
        monkeypatch.setenv("PT_CONV_HALO_ROWS", rows)
        y = dnm.conv3x3_forward(x.cuda(), wt.cuda(), b.cuda(), cout, out_f32=True).cpu()
        assert float((y - ref).abs().max()) <= 2e-3 * float(ref.abs().max()) and _rel(y, ref) <= 1e-4, rows
