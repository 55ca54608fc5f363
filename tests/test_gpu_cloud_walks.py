"""The static cloud where its kernel's two walks meet: clouds all over the box with a few points per
cell (each lane walks its own particle), sheets (the warp walks), both in one scene, rows of cells
that wrap, points on cell borders, empty cells inside a row, and a batch in which one scene has no
cloud.  Bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api, scenes
from oracle import cpu

pytestmark = pytest.mark.gpu

STATE = ("pos", "quat", "vel", "angvel")


def _scene(side, log2=None):
    sc = scenes.small_scene(side, nb_side=side, k=3, r=1.0 / (8 * side), packed=True)
    if log2:
        sc.grid_log2 = log2
    return sc


def _cloud(sc, points, shape, seed):
    rng = np.random.default_rng(seed)
    p = sc.world_positions()[:, :3]
    lo, hi = p.min(0) - 0.02, p.max(0) + 0.02
    cloud = np.zeros((2, points, 4), np.float32)
    cloud[0, :, :3] = rng.uniform(lo, hi, (points, 3))
    if shape != "volume":  # all of them, or every other one
        cloud[0, :: 1 if shape == "sheet" else 2, 1] = 0.5 * (lo[1] + hi[1])
    if shape == "borders":  # multiples of the contact distance
        d = np.float32(2 * sc.radius)
        cloud[0, :, :3] = np.round(cloud[0, :, :3] / d) * d
    n = rng.normal(size=(points, 3))
    cloud[1, :, :3] = n / np.linalg.norm(n, axis=1, keepdims=True)
    return cloud


@pytest.mark.parametrize("side,points,shape,log2", [
    (4, 300, "volume", None), (4, 40000, "volume", None), (12, 4000, "volume", None),
    (12, 60000, "volume", None), (12, 60000, "sheet", None), (12, 60000, "both", None),
    (12, 30000, "borders", None), (12, 60000, "volume", (4, 3, 2)), (12, 30000, "both", (2, 2, 5)),
    (22, 30000, "volume", None)])
def test_cloud_walks(ctx, side, points, shape, log2):
    sc = _scene(side, log2)
    cloud = _cloud(sc, points, shape, points)
    gs = api.GpuScene(ctx, sc)
    gs.set_static_cloud(*(torch.from_numpy(c).cuda() for c in cloud))
    gs.step(2)
    ctx.check()
    got = gs.download()
    gs.close()
    ref = cpu.step(sc, 2, cloud=tuple(cloud))
    for k in STATE:
        assert np.array_equal(got[k], ref[k]), k


def test_cloud_walks_in_a_batch(ctx):
    many = [_scene(s) for s in (3, 12, 5)]
    clouds = [_cloud(many[0], 500, "both", 1), _cloud(many[1], 50000, "volume", 2), None]
    gs = [api.GpuScene(ctx, sc) for sc in many]
    for g, c in zip(gs, clouds):
        if c is not None:
            g.set_static_cloud(*(torch.from_numpy(a).cuda() for a in c))
    batch = api.Batch(ctx, gs)
    batch.step(2)
    ctx.check()
    for g, sc, c in zip(gs, many, clouds):
        got, ref = g.download(), cpu.step(sc, 2, cloud=None if c is None else tuple(c))
        for k in STATE:
            assert np.array_equal(got[k], ref[k]), k
    batch.close()
    [g.close() for g in gs]
