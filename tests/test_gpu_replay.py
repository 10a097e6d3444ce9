"""A render whose launches equal the last call's is replayed: seed, sample count,
buffers and flags that only the call block holds must still reach the kernels, and
everything else (camera, depth, samples, statistics, another scene of the
workspace) must lead to a new capture.  Each call is compared with the same call
as serial launches."""
import pytest
import torch

from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene, render_batch

pytestmark = pytest.mark.gpu


def equal(a, b):
    return a.keys() == b.keys() and all(torch.equal(a[k].view(torch.int32), b[k].view(torch.int32)) for k in a)


@pytest.mark.parametrize("make", [scenes.cornell_box, scenes.material_spheres], ids=["one material type", "seven"])
def test_replayed_calls(cuda_ctx, make):
    g = GpuScene(cuda_ctx, make(53, 37))
    calls = [dict(seed=1), dict(seed=2), dict(seed=2, sample_cnt=3), dict(seed=2, accumulate=False),
             dict(seed=2, rng=1), dict(seed=2), dict(seed=3, max_depth=2), dict(seed=3, max_depth=2, wave_spp=1),
             dict(seed=4), dict(seed=4, flags=abi.RENDER_DROP_NONFINITE), dict(seed=5, sample_cnt=7)]
    other = torch.cuda.Stream()
    for i, kw in enumerate(calls + calls):
        aovs = i % 3 != 1
        mine, ref = (g.alloc_buffers(aovs) for _ in range(2))
        mine["accum"].fill_(0.25 * i)  # sample counts above 0 blend with what is there
        ref["accum"].fill_(0.25 * i)
        if i in (5, 16):
            g.set_camera(scenes.camera(40.0, 53 / 37, scenes.look_at_to_world((0.05 * i, 1.2, 3.5), (0.0, 0.9, 0.0))))
        torch.cuda.synchronize()
        g.render(4, buffers=mine, stream=other if i % 2 else None, **kw)
        kw = dict(kw, flags=kw.get("flags", 0) | abi.RENDER_NO_GRAPH)
        g.render(4, buffers=ref, **kw)
        assert equal(mine, ref), (i, kw)


def test_replayed_batches(cuda_ctx):
    gs = [GpuScene(cuda_ctx, scenes.cornell_box(w, 21)) for w in (33, 19, 40)]
    for seed, pick in ((1, (0, 1, 2)), (2, (0, 1, 2)), (2, (2, 0, 1)), (2, (0, 1, 2)), (3, (1,)), (3, (2,))):
        batched = render_batch(cuda_ctx, [gs[i] for i in pick], 3, seed=seed)
        for i, b in zip(pick, batched):
            assert equal(b, gs[i].render(3, seed=seed, flags=abi.RENDER_NO_GRAPH)), (seed, pick, i)
