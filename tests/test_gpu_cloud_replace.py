"""A scene's static cloud replaced by one of the same, a smaller and a larger size, detached and
attached again, alone and in a batch, between steps of the same graphs: every state as the oracle's."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api, scenes
from oracle import cpu

pytestmark = pytest.mark.gpu

STATE = ("pos", "quat", "vel", "angvel")


@pytest.mark.parametrize("batched", [False, True])
def test_cloud_replaced(ctx, batched):
    sc = scenes.small_scene(5, nb_side=4, r=1 / 128)
    gs = api.GpuScene(ctx, sc)
    batch = api.Batch(ctx, [gs]) if batched else None
    ref = {k: getattr(sc, "body_" + k) for k in STATE}
    for i, m in enumerate((5000, 5000, 700, 9000, 0, 8000, 9001)):
        rng = np.random.default_rng(i)
        cloud = np.zeros((2, m, 4), np.float32)
        cloud[0, :, :3] = rng.uniform(0.2, 0.8, (m, 3))
        n = rng.normal(size=(m, 3))
        cloud[1, :, :3] = n / np.linalg.norm(n, axis=1, keepdims=True)
        if m:
            gs.set_static_cloud(*(torch.from_numpy(c).cuda() for c in cloud))
        else:
            gs.set_static_cloud(None, None)
        (batch or gs).step(9)
        ctx.check()
        ref = cpu.step(sc, 9, cloud=tuple(cloud) if m else None, state={k: ref[k] for k in STATE})
        got = gs.download()
        for k in STATE:
            assert np.array_equal(got[k], ref[k]), (i, k)
    if batch:
        batch.close()
    gs.close()
