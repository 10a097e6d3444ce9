"""The BVH build around its tile sizes (sort tiles of 4096, clustering tiles of
1024 with halos, the one-block tail of 2048) and with coincident boxes: every
primitive is found, and the cost the collapse sums is the one refit computes
from the nodes."""
import numpy as np
import pytest
import torch

import oracle
from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene

pytestmark = pytest.mark.gpu


def triangles(n, kind, seed=1):
    """n small triangles: scattered, on few distinct places (equal codes), or along a line."""
    r = np.random.default_rng([n, seed])
    if kind == "scattered":
        c = r.uniform(-1, 1, (n, 1, 3))
    elif kind == "repeated":
        c = r.uniform(-1, 1, (7, 1, 3))[r.integers(0, 7, n)]
    else:
        c = np.linspace(-1, 1, n)[:, None, None] * np.array([1.0, 0.0, 0.0])
    p = c + r.normal(0, 0.03, (n, 3, 3))
    sc = scenes.Scene(8, 8, 4)
    mat = sc.add_material(scenes.diffuse(0.5))
    sc.add_instance(abi.SHAPE_MESH, sc.add_mesh(scenes.Mesh(p.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3))), mat)
    sc.env = (1.0, 1.0, 1.0)
    sc.camera = scenes.camera(40.0, 1.0, scenes.look_at_to_world((0, 0, 5), (0, 0, 0)))
    return sc, p


@pytest.mark.parametrize("flags", [0, abi.BVH_FAST_BUILD], ids=["ploc", "radix"])
@pytest.mark.parametrize("n,kind", [(2, "scattered"), (33, "scattered"), (1025, "line"), (2047, "scattered"),
                                    (2048, "repeated"), (2049, "scattered"), (4096, "line"), (4097, "repeated"),
                                    (9001, "scattered")])
def test_every_primitive_is_found(cuda_ctx, n, kind, flags):
    sc, p = triangles(n, kind)
    r = np.random.default_rng(3)
    pick = r.integers(0, n, 1500)
    target = p[pick].mean(axis=1)
    d = r.normal(size=target.shape)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((len(pick), 8), np.float32)
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = target - 2.0 * d, 0.001, d, 1e16
    ref = oracle.OracleScene(sc, bvh=False).trace(rays, brute_force=True)
    dev = torch.from_numpy(rays).cuda()
    g = GpuScene(cuda_ctx, sc, build=False)
    for width in (2, 4, 8):
        st = g.build_bvh(width=width, flags=flags)
        assert st.num_prims == n
        if kind == "scattered":
            assert st.builder == (abi.BVH_BUILDER_RADIX if flags else abi.BVH_BUILDER_PLOC)
        assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32)), (n, kind, width)
        # refit pads a parent again over its padded children: at most 2.6e-6 (4e-7 of the scene's and the
        # box's extent, 1e-6 of the box's) a side and level, 12 levels, against boxes of 0.05 and more:
        # 4 * 2.6e-6 * 12 / 0.05 = 2.5e-3 of an area
        assert g.refit().sah_cost == pytest.approx(st.sah_cost, rel=5e-3)


@pytest.mark.parametrize("flags", [0, abi.BVH_FAST_BUILD], ids=["ploc", "radix"])
@pytest.mark.parametrize("n", [40, 3000])
def test_box_area_overflows(cuda_ctx, n, flags):
    """A triangle whose box has no finite area (2.4e19 on two axes) among n small
    ones: its ancestors' costs are infinite and every primitive is still found.
    The triangle is a strip that passes 1.5e18 from the origin, so that the
    intersection test itself stays finite; rays run along y, across it."""
    sc, p = triangles(n, "scattered")
    strip = np.array([[-1.2, 0, -1.0], [1.2, 0, 1.4], [1.2, 0, 1.3]]) * 1e19 + np.array([0.0, -3.0, 0.0])
    sc.add_instance(abi.SHAPE_MESH, sc.add_mesh(scenes.Mesh(strip, np.array([[0, 1, 2]]))), sc.add_material(scenes.diffuse(0.5)))
    r = np.random.default_rng(5)
    pick = np.arange(1000) % n
    o = np.concatenate([p[pick].mean(axis=1), np.tile([0.0, -1.0, 1.75e18], (3, 1))])
    d = np.concatenate([r.normal(size=(1000, 3)) * [0.2, 0, 0.2] + [0, 1, 0], np.tile([1e-3, -1.0, 1e-3], (3, 1))])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o[:1000] -= 4.0 * d[:1000]
    rays = np.zeros((len(o), 8), np.float32)
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = o, 0.001, d, 1e16
    ref = oracle.OracleScene(sc, bvh=False).trace(rays, brute_force=True)
    hit = ref.view(np.int32)[:, 1] >= 0
    assert hit[1000:].all() and hit[:1000].mean() > 0.9
    dev = torch.from_numpy(rays).cuda()
    g = GpuScene(cuda_ctx, sc, build=False)
    for width in (2, 4, 8):
        assert g.build_bvh(width=width, flags=flags).num_prims == n + 1
        assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32)), (n, width)
        g.refit()
        assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32)), (n, width, "refit")


@pytest.mark.parametrize("width", [2, 4, 8])
def test_many_clusters(cuda_ctx, width):
    """Enough primitives that clustering searches for four positions a thread
    (300,000 clusters, tiles of 1,120), with a part of a last tile."""
    n = 301_001
    sc, p = triangles(n, "scattered", seed=4)
    r = np.random.default_rng(6)
    pick = np.concatenate([r.integers(0, n, 1500), [0, n - 1]])
    d = r.normal(size=(len(pick), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((len(pick), 8), np.float32)
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = p[pick].mean(axis=1) - 1e-2 * d, 0.001, d, 1e16
    ref = oracle.OracleScene(sc).trace(rays)
    g = GpuScene(cuda_ctx, sc, build=False)
    st = g.build_bvh(width=width)
    assert st.num_prims == n and st.builder == abi.BVH_BUILDER_PLOC
    dev = torch.from_numpy(rays).cuda()
    assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32))
    g.refit()
    assert np.array_equal(g.trace(dev).cpu().numpy().view(np.uint32), ref.view(np.uint32))
