"""ar_lbvh_build / ar_lbvh_build64 on both sides of the size from which the nodes are built in
tiles, and around the tiles: ranges that end at, cross
and span tiles, equal codes, and codes whose ranges nest one inside the other."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api
from diploma_thesis_b200._lib import call
from oracle import cpu

pytestmark = pytest.mark.gpu

TILES = 1 << 17  # leaves from which the tiles are used (1,024 nodes each)


def _codes(kind, n, bits, rng):
    if kind == "spread":
        c = rng.integers(0, 1 << bits, n, dtype=np.uint64)
    elif kind == "few":  # long runs of equal codes
        c = rng.integers(0, 7, n, dtype=np.uint64) << np.uint64(bits - 5)
    elif kind == "equal":
        c = np.full(n, 5, np.uint64)
    else:  # nested: leaf after leaf leaves the range from one side, then from the other
        c = np.uint64(1) << (np.arange(n, dtype=np.uint64) * np.uint64(bits) // np.uint64(n))
        c[n // 2:] = np.uint64((1 << bits) - 1) - c[n // 2:]
    return np.sort(c)


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("kind", ["spread", "few", "equal", "nested"])
@pytest.mark.parametrize("n", [2, 3, TILES - 1, TILES, TILES + 1, TILES + 2, TILES + 1023, TILES + 1025,
                               3 * TILES + 77])
def test_build_tiles(ctx, n, kind, bits):
    c = _codes(kind, n, bits, np.random.default_rng(n + bits))
    if bits == 30:
        c = c.astype(np.uint32)
    want = cpu.radix_tree(c)
    d = torch.from_numpy(c.view(np.int32 if bits == 30 else np.int64)).cuda()
    out = {"is_leaf": torch.full((2 * n - 1,), 9, dtype=torch.uint8, device="cuda")}
    for k in ("left", "right", "parent", "min_r", "max_r"):
        out[k] = torch.full((2 * n - 1,), -7, dtype=torch.int32, device="cuda")
    call("ar_lbvh_build" if bits == 30 else "ar_lbvh_build64", ctx.handle, api.ptr(d), n,
         *(api.ptr(t) for t in out.values()), api.stream_handle())
    ctx.check()
    got = {k: t.cpu().numpy() for k, t in out.items()}
    assert np.array_equal(got["left"][n:], want["left"][n:])
    assert np.array_equal(got["right"][n:], want["right"][n:])
    assert got["parent"][n] == -1 and np.all(got["is_leaf"][n:] == 0)
    inner = np.arange(2 * n - 1) != n
    assert np.array_equal(got["parent"][inner], want["parent"][inner])
    assert np.array_equal(got["min_r"][n:], want["min_r"][n:])
    assert np.array_equal(got["max_r"][n:], want["max_r"][n:])
