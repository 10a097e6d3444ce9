"""Path slots in tile order, frame-minor: film sizes around the 4-row bands and
one- and many-frame waves, against the CPU oracle and against each other."""
import numpy as np
import pytest
import torch

import oracle
from pupiloptixlab_gb300 import abi, scenes
from pupiloptixlab_gb300.api import GpuScene, render_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (5, 3), (7, 4), (1, 9), (33, 6), (40, 5)])
def test_film_sizes_match_the_oracle_for_every_wave_size(cuda_ctx, size):
    sc = scenes.material_spheres(*size)
    spp = 9  # not a multiple of the eight frames accumulated at a time
    ref = oracle.OracleScene(sc).render(abi.RenderParams(spp=spp, seed=3, accumulate=1, rng=abi.RNG_PCG32))
    g = GpuScene(cuda_ctx, sc)
    for wave_spp in (0, 1, 4):
        out = g.render(spp, seed=3, rng=abi.RNG_PCG32, wave_spp=wave_spp)
        for k in ("accum", "albedo", "normal"):
            got = out[k].cpu().numpy()
            want = ref[k].reshape(got.shape)
            assert np.array_equal(got[:, :3], want[:, :3]), (k, size, wave_spp)


def test_batch_of_odd_films_equals_serial_renders(cuda_ctx):
    gs = [GpuScene(cuda_ctx, scenes.material_spheres(w, h)) for w, h in [(5, 3), (33, 6), (1, 9)]]
    serial = [g.render(9, seed=2)["accum"].clone() for g in gs]
    batched = render_batch(cuda_ctx, gs, 9, seed=2)
    assert all(torch.equal(a, b["accum"]) for a, b in zip(serial, batched))
