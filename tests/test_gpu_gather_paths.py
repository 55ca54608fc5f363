"""The grid step's gather and static-cloud kernels at the sizes where their splits change: few
particles per warp, the last warp partly filled, either side of the line between the warp-wide and
the per-thread walk, cells that hold more occupants than the entry's count, folded grids.  Bit
for bit against the oracle."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api, scenes
from oracle import cpu

pytestmark = pytest.mark.gpu

STATE = ("pos", "quat", "vel", "angvel")


def _check(ctx, sc, steps=3, cloud=None, **kw):
    gs = api.GpuScene(ctx, sc, **kw)
    if cloud is not None:
        gs.set_static_cloud(*(torch.from_numpy(a).cuda() for a in cloud))
    gs.step(steps)
    ctx.check()
    got = gs.download()
    gs.close()
    ref = cpu.step(sc, steps, cloud=cloud)
    for k in STATE:
        assert np.array_equal(got[k], ref[k]), k


# 27, 135, 1,000 (not a multiple of 32), 4,096, 13,824 and 15,625 particles
@pytest.mark.parametrize("side,k", [(1, 3), (5, 1), (5, 2), (8, 2), (8, 3), (25, 1)])
def test_gather_sizes(ctx, side, k):
    _check(ctx, scenes.small_scene(side, nb_side=side, k=k, r=1.0 / (2.5 * side * max(k, 2)),
                                   packed=True))


@pytest.mark.parametrize("side", [4, 9])  # the warp-wide and the per-thread walk
def test_gather_crowded_cells_and_folded_grid(ctx, side):
    sc = scenes.small_scene(3, nb_side=side, k=3, r=1.0 / 256, packed=True)
    sc.body_pos[:, :3] = 0.5 + (sc.body_pos[:, :3] - 0.5) * np.float32(0.4)  # bodies overlap
    sc.spring = 500.0
    _check(ctx, sc)
    folded = scenes.small_scene(4, nb_side=side, k=3, r=1.0 / 256, packed=True)
    folded.grid_log2 = (2, 3, 2)  # every cell holds many far particles
    _check(ctx, folded)


@pytest.mark.parametrize("side,k,points", [(1, 1, 1), (3, 2, 33), (12, 2, 20000), (25, 2, 20000)])
def test_cloud_sizes(ctx, side, k, points):
    rng = np.random.default_rng(points)
    sc = scenes.small_scene(side, nb_side=side, k=k, r=1.0 / (4 * side * k))
    cloud = np.zeros((2, points, 4), np.float32)
    cloud[0, :, :3] = sc.world_positions()[rng.integers(0, sc.num_particles, points), :3]
    cloud[0, :, :3] += rng.normal(0.0, sc.radius, (points, 3))
    n = rng.normal(size=(points, 3))
    cloud[1, :, :3] = n / np.linalg.norm(n, axis=1, keepdims=True)
    _check(ctx, sc, cloud=tuple(np.ascontiguousarray(c) for c in cloud))
