"""The batch's scene lookup by stretches of 4,096 pixels: scenes that end on a
stretch's border, one pixel before and after it, many in one stretch and one over
many, against the scenes rendered alone."""
import pytest
import torch

from pupiloptixlab_gb300 import scenes
from pupiloptixlab_gb300.api import GpuScene, render_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(64, 64), (1, 1), (64, 64)], [(65, 63), (1, 1), (64, 64), (3, 3)], [(17, 241), (64, 64)],
                                   [(1, 1)] * 40 + [(129, 127)], [(200, 150), (1, 7), (90, 91)], [(4096, 1)],
                                   [(8, 8)] * 128])
def test_batch_equals_serial(cuda_ctx, sizes):
    shapes = {s: GpuScene(cuda_ctx, scenes.cornell_box(*s)) for s in set(sizes)}
    gs, seen = [], set()
    for s in sizes:
        gs.append(shapes[s] if s not in seen else GpuScene(cuda_ctx, scenes.cornell_box(*s)))
        seen.add(s)
    for g, b in zip(gs, render_batch(cuda_ctx, gs, 2, seed=9)):
        assert torch.equal(g.render(2, seed=9)["accum"], b["accum"])
