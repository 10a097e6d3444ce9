"""Material binning: counts and prefix over the blocks in one kernel, queue pushes
by whole blocks.  Queues of one pixel to several stretches per block, one and
several waves, all materials and only misses, against shading in queue order."""
import pytest
import torch

from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,spp,wave_spp", [((1, 1), 1, 0), ((3, 5), 2, 1), ((64, 4), 1, 0), ((257, 1), 3, 2),
                                               ((640, 487), 1, 0), ((700, 467), 5, 3)])
@pytest.mark.parametrize("misses", [False, True])
def test_binned_equals_queue_order(cuda_ctx, size, spp, wave_spp, misses):
    sc = scenes.material_spheres(*size)
    if misses:
        sc.camera = scenes.camera(30.0, size[0] / size[1], scenes.look_at_to_world((0.0, 50.0, 0.0), (1.0, 99.0, 0.0)))
    g = GpuScene(cuda_ctx, sc)
    want = g.render(spp, seed=3, wave_spp=wave_spp, flags=abi.RENDER_NO_MATERIAL_SORT | abi.RENDER_NO_GRAPH)
    for _ in range(2):
        got = g.render(spp, seed=3, wave_spp=wave_spp)
        assert all(torch.equal(got[k].view(torch.int32), want[k].view(torch.int32)) for k in want)
