"""Shadow rays beside the next bounce's extension rays, per-bounce counter sets
and unbinned one-material and last bounces: the captured render against the
serial one (no graph) and against binning in place, over depths and wave sizes."""
import pytest
import torch

from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene, render_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [scenes.cornell_box, scenes.material_spheres], ids=["one material type", "seven"])
@pytest.mark.parametrize("depth", [1, 2, 3, 9])
def test_graph_equals_serial_launches(cuda_ctx, make, depth):
    g = GpuScene(cuda_ctx, make(61, 45))
    for wave_spp in (0, 2):  # 5 spp: one wave, and three
        want = g.render(5, seed=4, max_depth=depth, wave_spp=wave_spp, flags=abi.RENDER_NO_GRAPH)
        want = {k: v.clone() for k, v in want.items()}
        for flags in (0, abi.RENDER_NO_MATERIAL_SORT, 0):
            got = g.render(5, seed=4, max_depth=depth, wave_spp=wave_spp, flags=flags)
            assert all(torch.equal(got[k].view(torch.int32), want[k].view(torch.int32)) for k in want)


def test_batch_with_scene_depths(cuda_ctx):
    gs = [GpuScene(cuda_ctx, scenes.material_spheres(31, 17, max_depth=d)) for d in (1, 5, 2)]
    serial = [g.render(3, seed=8)["accum"].clone() for g in gs]
    for _ in range(2):
        batched = render_batch(cuda_ctx, gs, 3, seed=8)
        assert all(torch.equal(a, b["accum"]) for a, b in zip(serial, batched))
