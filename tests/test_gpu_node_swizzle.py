"""Swizzled node records and near / far planes picked by octant: every width,
nodes from global memory and staged in shared memory, merged at offsets that
change the swizzle, and rays of every octant with zero components of either
sign, against brute force and against the scenes alone."""
import numpy as np
import pytest
import torch

import oracle
from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene, render_batch

pytestmark = pytest.mark.gpu


def cloud(n, width=9, height=7):
    sc = scenes.Scene(width, height, 3)
    mat = sc.add_material(scenes.diffuse(0.5))
    r = np.random.default_rng(n)
    p = r.uniform(-1, 1, (n, 1, 3)) + r.normal(0, 0.2, (n, 3, 3))
    sc.add_instance(abi.SHAPE_MESH, sc.add_mesh(scenes.Mesh(p.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3))), mat)
    sc.env = (1.0, 1.0, 1.0)
    sc.camera = scenes.camera(40.0, 1.0, scenes.look_at_to_world((0, 0, 5), (0, 0, 0)))
    return sc


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("staged", [0, 1, 13, 400])
def test_octants(cuda_ctx, width, staged):
    sc = cloud(300)
    r = np.random.default_rng(3)
    d = r.normal(size=(640, 3)).astype(np.float32)
    d[np.abs(d) < 0.6] *= np.float32(0.0)  # many zeros, of both signs
    d[np.all(d == 0, axis=1)] = (0.0, -1.0, -0.0)
    rays = np.zeros((640, 8), np.float32)
    rays[:, 0:3] = r.uniform(-1, 1, (640, 3)) - 2.0 * d
    rays[:, 3], rays[:, 4:7], rays[:, 7] = 0.001, d, 1e16
    assert np.signbit(d[d == 0]).any() and not np.signbit(d[d == 0]).all()
    ref = oracle.OracleScene(sc, bvh=False).trace(rays, brute_force=True)
    g = GpuScene(cuda_ctx, sc, bvh_width=width, max_leaf=2, smem_nodes=staged)
    dev = torch.from_numpy(rays).cuda()
    assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32))
    occluded = g.trace(dev, anyhit=True).cpu().numpy()[:, 0]
    assert np.array_equal(occluded, (ref[:, 1].view(np.int32) >= 0).astype(np.float32))


@pytest.mark.parametrize("width", [2, 4, 8])
def test_merged_offsets(cuda_ctx, width):
    gs = [GpuScene(cuda_ctx, cloud(n), bvh_width=width, max_leaf=1) for n in (1, 2, 23, 1, 90, 7, 300, 5)]
    batched = render_batch(cuda_ctx, gs, 2, seed=6)
    for g, b in zip(gs, batched):
        assert torch.equal(g.render(2, seed=6)["accum"], b["accum"])
