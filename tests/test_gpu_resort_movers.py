"""The re-sort from the previous order when whole runs of tiles hold movers only: every particle of the
scene, those on one side of it, a slab in the middle, and a few that stay, over one tile, a few and
more than 32 tiles (of 512 positions).  The step's state against the oracle's, bit for bit."""
import numpy as np
import pytest

from diploma_thesis_b200 import api, scenes
from oracle import cpu

pytestmark = pytest.mark.gpu

STATE = ("pos", "quat", "vel", "angvel")


@pytest.mark.parametrize("broadphase", ["grid", "bvh"])
@pytest.mark.parametrize("move", ["all", "low", "high", "slab", "all but two"])
@pytest.mark.parametrize("side", [3, 7, 14])  # 729, 9,261 and 74,088 particles: 2, 19, 145 tiles
def test_runs_of_movers(ctx, side, move, broadphase):
    sc = scenes.config0(side, lattice=side)
    rng = np.random.default_rng(side)
    v = rng.normal(size=(sc.num_bodies, 3))
    v *= 3 * 2 * sc.radius / sc.dt / np.linalg.norm(v, axis=1, keepdims=True)  # three cells a step
    z = sc.body_pos[:, 2]
    still = {"all": z > 2, "low": z > 0.6, "high": z < 0.4, "slab": abs(z - 0.5) > 0.3,
             "all but two": np.isin(np.arange(sc.num_bodies), [1, sc.num_bodies - 2])}[move]
    v[still] = 0
    sc.body_vel = sc.body_vel.copy()
    sc.body_vel[:, :3] = v
    gs = api.GpuScene(ctx, sc, broadphase=broadphase)
    gs.step(3)
    ctx.check()
    got = gs.download()
    gs.close()
    ref = cpu.step(sc, 3, broadphase=broadphase)
    for k in STATE:
        assert np.array_equal(got[k], ref[k]), k
