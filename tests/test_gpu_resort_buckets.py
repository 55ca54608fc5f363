"""The re-sort's buckets (csrc/ar_resort.cuh) where their movers come in bunches: the bodies of a
stepped scene are drawn together, so that every particle changes key and single buckets hold a
warp's share of movers, a block's, and more than a block stages in shared memory.  The next step
must match the first step of a fresh scene with the same state (radix sort), bit for bit."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api, scenes

pytestmark = pytest.mark.gpu

BLOCK = 2048  # movers a block stages; the last case has 287,496 particles, in larger tiles


def _sorted(gs):
    v = gs.step_view()
    n = v.num_particles
    return [api.device_view(p, m * n, torch.int32).cpu().numpy().copy()
            for p, m in ((v.sorted_keys, 1), (v.sorted_idx, 1), (v.particle_force4, 4))], v


def _biggest(ka, kb, va, vb, key_bits):
    """Movers of the fullest bucket between two orders (about 256 particles per bucket)."""
    old, new = np.empty_like(ka), np.empty_like(kb)
    old[va], new[vb] = ka, kb
    moved = new[old != new].view(np.uint32)
    bits = min(12, max(5, (len(ka) - 1).bit_length() - 8))
    return np.bincount(moved >> max(0, key_bits - bits)).max()


@pytest.mark.parametrize("broadphase", ["grid", "bvh"])
@pytest.mark.parametrize("side,draw,least", [(2, 0.9, 1), (4, 0.9, 1), (6, 0.9, 1), (9, 0.5, 1),
                                             (12, 0.1, BLOCK + 1), (22, 0.9, 1)])
def test_bunched_movers(ctx, broadphase, side, draw, least):
    sc = scenes.small_scene(5, nb_side=side, packed=True, r=1 / 128 if side < 20 else 1 / 256)
    a = api.GpuScene(ctx, sc, broadphase=broadphase)
    a.step(3)
    (k0, i0, _), _ = _sorted(a)
    state = a.download_state()
    centre = state[0, :, :3].mean(axis=0)
    state[0, :, :3] = centre + np.float32(draw) * (state[0, :, :3] - centre)
    a.upload_state(state)
    b = api.GpuScene(ctx, sc, broadphase=broadphase)
    b.upload_state(state)
    a.step(1)
    b.step(1)
    ctx.check()
    (ka, ia, fa), v = _sorted(a)
    (kb, ib, fb), _ = _sorted(b)
    assert _biggest(k0, ka, i0, ia, v.key_bits) >= least
    assert np.array_equal(ka, kb) and np.array_equal(ia, ib)
    assert np.array_equal(fa, fb)
    assert np.array_equal(a.download_state(), b.download_state())
    a.close()
    b.close()
