"""ar_scene_aabb at the edges of its blocks, its load batches and its last block's fold."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api
from diploma_thesis_b200._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 257, 1023, 256 * 257, 1024 * 256 + 1, 1024 * 1024 + 3])
def test_aabb_sizes(ctx, n):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 4)).astype(np.float32)
    p[n // 2, 1] = np.nan  # never a bound
    d = torch.from_numpy(p).cuda()
    lo, hi = torch.zeros(4, device="cuda"), torch.zeros(4, device="cuda")
    call("ar_scene_aabb", ctx.handle, api.ptr(d), n, api.ptr(lo), api.ptr(hi),
         api.stream_handle())
    ctx.check()
    if n > 1:
        assert np.array_equal(lo.cpu().numpy(), np.nanmin(p, 0))
        assert np.array_equal(hi.cpu().numpy(), np.nanmax(p, 0))
    else:  # no finite value in the second component: the bounds stay at their start values
        assert lo[1].item() == 2139095040.0 and hi[1].item() == -2139095040.0
        assert np.array_equal(lo.cpu().numpy()[[0, 2, 3]], p[0, [0, 2, 3]])
