"""Refit, K lanes a node and the short levels at the top in one launch: after
vertices move, a refit tree finds exactly the hits of brute force, for one
primitive to several levels, every width, both builders and repeated refits,
and its SAH cost does not depend on the run."""
import numpy as np
import pytest
import torch

import oracle
from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene

pytestmark = pytest.mark.gpu


def cloud(p):
    sc = scenes.Scene(8, 8, 4)
    mat = sc.add_material(scenes.diffuse(0.5))
    sc.add_instance(abi.SHAPE_MESH, sc.add_mesh(scenes.Mesh(p.reshape(-1, 3), np.arange(p.size // 3).reshape(-1, 3))), mat)
    sc.env = (1.0, 1.0, 1.0)
    sc.camera = scenes.camera(40.0, 1.0, scenes.look_at_to_world((0, 0, 5), (0, 0, 0)))
    return sc


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("n,leaf,flags", [(1, 1, 0), (2, 1, 0), (9, 1, 0), (33, 15, 0), (700, 1, abi.BVH_FAST_BUILD),
                                          (5000, 4, 0)])
def test_moved_vertices(cuda_ctx, width, n, leaf, flags):
    r = np.random.default_rng(n)
    rays = np.zeros((400, 8), np.float32)
    d = r.normal(size=(400, 3))
    rays[:, 0:3] = r.uniform(-1, 1, (400, 3)) - 3.0 * d
    rays[:, 3], rays[:, 4:7], rays[:, 7] = 0.001, d, 1e16
    dev = torch.from_numpy(rays).cuda()
    start = (r.uniform(-1, 1, (n, 1, 3)) + r.normal(0, 0.2, (n, 3, 3))).astype(np.float32)
    g = GpuScene(cuda_ctx, cloud(start), bvh_width=width, max_leaf=leaf, bvh_flags=flags)
    for step in range(3):
        moved = (start[r.permutation(n)] * (1.0 + step)).astype(np.float32)
        if step % 2:
            g.update_all_vertices(torch.from_numpy(moved.reshape(-1, 3)).cuda())
        else:
            g.update_vertices(0, moved.reshape(-1, 3))
        costs = set()
        ref = oracle.OracleScene(cloud(moved), bvh=False).trace(rays, brute_force=True)
        for _ in range(3):
            g.refit()
            costs.add(np.float32(g.bvh_stats().sah_cost))
            assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32))
        # the cost is a sum in double precision in some order, rounded once
        assert max(costs) - min(costs) <= 2 * np.spacing(max(costs))
