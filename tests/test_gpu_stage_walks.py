"""The stage entry points' searches at their limits: trees deeper than the walk's stack, particles
with more contacts than a thread's list, wrapped grids."""
import ctypes as C

import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api, scenes
from diploma_thesis_b200._lib import call
from oracle import cpu

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("levels", [1, 31, 33, 62])
def test_walk_deeper_than_its_stack(ctx, levels):
    """Pairs of keys 2^k, 2^k + 1: every level's right subtree waits while the left one is walked.
    All points touch one another, so every pair of them is found."""
    codes = np.array([v for k in range(1, levels + 1) for v in (1 << k, (1 << k) + 1)], np.uint64)
    n, s = len(codes), api.stream_handle()
    m = 2 * n - 1
    rng = np.random.default_rng(levels)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, 0.1, (n, 3))
    z = lambda k, t=torch.int32: torch.zeros(k, dtype=t, device="cuda")  # noqa: E731
    leaf, left, right, parent, lo, hi = z(m, torch.uint8), z(m), z(m), z(m), z(m), z(m)
    cms, bounds, radii = z(4 * n, torch.float32), z(8 * m, torch.float32), z(n, torch.float32)
    P, h, idx = api.ptr, ctx.handle, _dev(np.arange(n, dtype=np.int32))
    call("ar_lbvh_build64", h, P(_dev(codes.view(np.int64))), n, P(leaf), P(left), P(right),
         P(parent), P(lo), P(hi), s)
    call("ar_lbvh_leaves", h, n, P(idx), P(_dev(pos)), C.c_float(1.0), P(leaf), P(lo), P(hi),
         P(cms), P(bounds), P(radii), s)
    call("ar_lbvh_refit", h, n, P(left), P(right), P(parent), P(bounds), s)
    cap = n * n
    pairs, count = z(2 * cap), z(1)
    call("ar_pairs_bvh", h, C.c_float(1.0), P(idx), P(leaf), P(left), P(right), P(parent), P(cms),
         P(bounds), P(idx), n, P(pairs), cap, P(count), s)
    ctx.check()
    k = int(count.item())
    got = pairs.cpu().numpy().reshape(-1, 2)[:k]
    want = np.stack(np.triu_indices(n, 1), 1)
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)


@pytest.mark.parametrize("n,spread,dims", [(1, 1.0, 8), (129, 0.25, 8), (2000, 0.3, 8),
                                           (2000, 0.9, 2)])
def test_grid_forces_and_contacts(ctx, n, spread, dims):
    """Particles of three to a body, crowded enough for dozens of contacts each."""
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, spread, (n, 3))
    vel = rng.normal(0, 1, (n, 4)).astype(np.float32)
    rel = rng.normal(0, 0.1, (n, 4)).astype(np.float32)
    rb = (np.arange(n) // 3).astype(np.int32)
    r = 0.05
    prm = api.sim_params(r, (0.0, 0.0, 0.0), 2 * r, (dims,) * 3)
    P, h, s = api.ptr, ctx.handle, api.stream_handle()
    z = lambda shape, t=torch.float32: torch.zeros(shape, dtype=t, device="cuda")  # noqa: E731
    i32, pp, d = torch.int32, C.byref(prm), {k: _dev(v) for k, v in
                                             (("pos", pos), ("vel", vel), ("rel", rel), ("rb", rb))}
    hsh, idx, sh, si = (z(n, i32) for _ in range(4))
    cells = dims ** 3
    cs, ce, sp, sv = z(cells, i32), z(cells, i32), z((n, 4)), z((n, 4))
    call("ar_calc_hash", h, pp, P(d["pos"]), n, P(hsh), P(idx), s)
    call("ar_radix_sort_pairs_u32", h, P(hsh), P(idx), P(sh), P(si), n, 0, 32, s)
    call("ar_reorder_cells", h, P(sh), P(si), P(d["pos"]), P(d["vel"]), n, cells, P(cs), P(ce),
         P(sp), P(sv), s)
    f, t = z((n, 4)), z((n, 4))
    call("ar_collide_grid_dem", h, pp, P(d["rb"]), P(sp), P(sv), P(d["rel"]), P(si), P(cs), P(ce),
         n, P(f), P(t), s)
    cd, cb, cp = z(n), z(n, i32), z(n, i32)
    call("ar_find_contacts_grid", h, pp, P(d["rb"]), P(sp), P(si), P(cs), P(ce), n, P(cd), P(cb),
         P(cp), s)
    ctx.check()
    host = lambda x: x.cpu().numpy()  # noqa: E731
    origin, cell, dd = np.zeros(3, np.float32), np.full(3, 2 * r, np.float32), (dims,) * 3
    law = [prm.spring, prm.damping, prm.shear, prm.attraction, r]
    rf, rt = cpu.collide_grid_dem(origin, cell, dd, law, rb, host(sp), host(sv), rel,
                                  host(si).view(np.uint32), host(cs).view(np.uint32),
                                  host(ce).view(np.uint32))
    assert np.array_equal(host(f), rf) and np.array_equal(host(t), rt)
    rd, rbody, rpart = cpu.find_contacts_grid(origin, cell, dd, r, rb, host(sp),
                                              host(si).view(np.uint32), host(cs).view(np.uint32),
                                              host(ce).view(np.uint32), np.zeros(n, np.float32))
    assert np.array_equal(host(cd), rd)
    hit = rd > 0
    assert np.array_equal(host(cb)[hit], rbody[hit]) and np.array_equal(host(cp)[hit], rpart[hit])
