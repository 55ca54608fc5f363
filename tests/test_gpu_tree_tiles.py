"""Trees at the sizes where their tiles, groups of tiles and levels begin and end, with equal
codes (the index tie-break), one-particle scenes and long chains: the fused step's tree against
the oracle's nodes and boxes, and whole steps against the oracle."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api, scenes
from diploma_thesis_b200._lib import ArError
from oracle import cpu

pytestmark = pytest.mark.gpu

STATE = ("pos", "quat", "vel", "angvel")


def _points(n: int, layout: str, seed: int = 0) -> scenes.Scene:
    """n bodies of one particle: spread over the box, clustered in one Morton cell (equal codes),
    or on a line whose codes halve their distance to its end (deep, one-sided trees)."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    lattice = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    if layout == "spread":
        c = (lattice + rng.uniform(0.2, 0.8, (n, 3))) / side
        r = 0.1 / side
    elif layout == "cluster":
        c = 0.5 + 1e-5 + lattice * (0.9e-3 / side)
        r = 1e-7
    else:
        c = np.zeros((n, 3))
        c[:, 0] = 0.5 ** (1 + np.arange(n) % 10) + rng.uniform(0.0, 1e-4, n)
        c[:, 1:] = rng.uniform(0.0, 0.9, (n, 2)) * (np.arange(n) % 3 == 0)[:, None]
        r = 1e-8
    return scenes._assemble([np.zeros((1, 3))] * n, c, scenes.random_quaternions(rng, n),
                            rng.normal(0.0, 0.1, (n, 3)), r, (0, 0, 0), (1, 1, 1))


def _view(gs):
    v = gs.step_view()
    n = v.num_particles
    get = lambda a, m, t=torch.int32: api.device_view(a, m, t).cpu().numpy()  # noqa: E731
    nodes = get(v.tree_nodes16, 16 * max(n - 1, 1), torch.float32).reshape(-1, 16)
    return (n, get(v.sorted_keys, n).view(np.uint32), get(v.tree_left, 2 * n),
            get(v.tree_right, 2 * n), get(v.tree_parent, 2 * n), nodes,
            get(v.sorted_pos4, 4 * n, torch.float32).reshape(n, 4))


def _check(ctx, gs, ref):
    """The states equal the oracle's; two particles that coincide (some lines have such) make the
    state NaN in both, and the context says so."""
    if all(np.isfinite(ref[k]).all() for k in STATE):
        ctx.check()
    else:
        with pytest.raises(ArError, match="AR_ERR_NAN"):
            ctx.check()
    got = gs.download()
    for k in STATE:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k


@pytest.mark.parametrize("layout", ["spread", "cluster", "line"])
@pytest.mark.parametrize("n", [2, 255, 256, 257, 511, 4096, 4097, 65537])
def test_step_tree(ctx, n, layout):
    sc = _points(n, layout, n)
    gs = api.GpuScene(ctx, sc, broadphase="bvh")
    gs.step(1)
    _check(ctx, gs, cpu.step(sc, 1, broadphase="bvh"))
    n, keys, left, right, parent, nodes, pos = _view(gs)
    t = cpu.radix_tree(keys.copy())
    inner = slice(n, 2 * n - 1)
    assert np.array_equal(left[inner], t["left"][inner])
    assert np.array_equal(right[inner], t["right"][inner])
    t["parent"][n] = -1
    assert np.array_equal(parent[:2 * n - 1], t["parent"][:2 * n - 1])
    box = np.zeros((2 * n - 1, 8), np.float32)
    r = np.float32(sc.radius)
    box[:n, :3], box[:n, 3:6] = pos[:, :3] - r, pos[:, :3] + r
    box = cpu.refit(t, box)
    for side, child in ((nodes[:, :8], left[inner]), (nodes[:, 8:], right[inner])):
        assert np.array_equal(side[:, :6], box[child, :6])
        assert np.array_equal(side[:, 6].copy().view(np.int32), child)
    gs.step(2)
    _check(ctx, gs, cpu.step(sc, 3, broadphase="bvh"))
    gs.close()


@pytest.mark.parametrize("sizes", [(1, 1), (1, 300, 1, 255), (1, 2, 700, 1, 256, 1, 4100)])
def test_step_tree_of_a_batch(ctx, sizes):
    group = [_points(n, "spread", i) for i, n in enumerate(sizes)]
    scs = [api.GpuScene(ctx, sc, broadphase="bvh") for sc in group]
    batch = api.Batch(ctx, scs)
    batch.step(5)
    ctx.check()
    for gs, sc in zip(scs, group):
        got, ref = gs.download(), cpu.step(sc, 5, broadphase="bvh")
        for k in STATE:
            assert np.array_equal(got[k], ref[k]), k
    batch.close()
    for gs in scs:
        gs.close()
