"""Nodes that hold their children as traversal items: leaves of 1 to 15
primitives as a root and below one, empty slots, origins far outside the
scene (the unfused slab form), every width, against brute force."""
import numpy as np
import pytest
import torch

import oracle
from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene

pytestmark = pytest.mark.gpu


def cloud(n):
    sc = scenes.Scene(8, 8, 4)
    mat = sc.add_material(scenes.diffuse(0.5))
    r = np.random.default_rng(n)
    p = r.uniform(-1, 1, (n, 1, 3)) + r.normal(0, 0.2, (n, 3, 3))
    sc.add_instance(abi.SHAPE_MESH, sc.add_mesh(scenes.Mesh(p.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3))), mat)
    sc.env = (1.0, 1.0, 1.0)
    sc.camera = scenes.camera(40.0, 1.0, scenes.look_at_to_world((0, 0, 5), (0, 0, 0)))
    return sc


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("n,leaf", [(1, 1), (2, 1), (15, 15), (16, 15), (17, 1), (700, 3)])
def test_hits_equal_brute_force(cuda_ctx, width, n, leaf):
    sc = cloud(n)
    r = np.random.default_rng(7)
    rays = np.zeros((512, 8), np.float32)
    d = r.normal(size=(512, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:24] = np.tile(np.concatenate([np.eye(3), -np.eye(3)]), (4, 1))  # along the axes
    back = np.where(np.arange(512) % 2, 3.0, 3e4)[:, None]
    rays[:, 0:3] = r.uniform(-0.5, 0.5, (512, 3)) - back * d
    rays[:, 3], rays[:, 4:7], rays[:, 7] = 0.001, d, 1e16
    ref = oracle.OracleScene(sc, bvh=False).trace(rays, brute_force=True)
    g = GpuScene(cuda_ctx, sc, bvh_width=width, max_leaf=leaf)
    dev = torch.from_numpy(rays).cuda()
    for _ in range(2):  # as built, then refit
        assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32))
        occluded = g.trace(dev, anyhit=True).cpu().numpy()[:, 0]
        assert np.array_equal(occluded, (ref[:, 1].view(np.int32) >= 0).astype(np.float32))
        g.refit()
