"""ar_lbvh_refit where its two forms meet (2^20 leaves), with a partly filled last tile, equal codes,
and internal nodes numbered at random (then nothing merges inside a tile)."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api
from diploma_thesis_b200._lib import call
from oracle import cpu

pytestmark = pytest.mark.gpu


def _renumbered(t, n, rng):
    """The same tree with its internal nodes, but the root, numbered at random."""
    new = np.arange(2 * n - 1, dtype=np.int32)
    new[n + 1:] = n + 1 + rng.permutation(n - 2)
    old = np.argsort(new)
    out = {k: new[t[k][old]] for k in ("left", "right")}
    parent = t["parent"][old]
    out["parent"] = np.where(parent >= 0, new[parent], -1).astype(np.int32)
    out["left"][:n] = out["right"][:n] = -1
    return out


@pytest.mark.parametrize("n,codes,renumber", [
    (2, "spread", False), (257, "spread", True), ((1 << 20) - 1, "spread", False),
    (1 << 20, "equal", False), ((1 << 20) + 1, "spread", False), ((1 << 20) + 130, "spread", True)])
def test_refit_forms(ctx, n, codes, renumber):
    rng = np.random.default_rng(n)
    keys = np.sort(rng.integers(0, 1 << 30, n)).astype(np.uint32)
    t = cpu.radix_tree(keys * np.uint32(codes == "spread"))
    t["parent"][n] = -1
    if renumber:
        t |= _renumbered(t, n, rng)
    box = np.zeros((2 * n - 1, 8), np.float32)
    c = rng.normal(size=(n, 3)).astype(np.float32)
    box[:n, :3], box[:n, 3:6] = c - np.float32(0.1), c + np.float32(0.1)
    dev = {k: torch.from_numpy(t[k]).cuda() for k in ("left", "right", "parent")}
    d = torch.from_numpy(box).cuda()
    call("ar_lbvh_refit", ctx.handle, n, *(api.ptr(dev[k]) for k in ("left", "right", "parent")),
         api.ptr(d), api.stream_handle())
    ctx.check()
    # a box is the smallest around its leaves, whatever the order of the merges
    want = box.copy()
    lo, hi = want[:, :3], want[:, 3:6]
    levels = [np.array([n])]
    while len(levels[-1]):
        kids = np.concatenate([t["left"][levels[-1]], t["right"][levels[-1]]])
        levels.append(kids[kids >= n])
    for nodes in reversed(levels):
        a, b = t["left"][nodes], t["right"][nodes]
        lo[nodes] = np.minimum(lo[a], lo[b])
        hi[nodes] = np.maximum(hi[a], hi[b])
    assert np.array_equal(d.cpu().numpy()[:, :6], want[:, :6])
