"""The radix sort at the edges of its tiles and where the tile shapes change (2^19 keys, 8- and
9-bit digits, 32- and 64-bit keys), against numpy's stable sort."""
import numpy as np
import pytest
import torch

from diploma_thesis_b200 import api
from diploma_thesis_b200._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,bits", [(32, 24), (32, 25), (64, 34), (64, 63)])
@pytest.mark.parametrize("n", [1, 2047, 2049, 4097, (1 << 19) - 1, 1 << 19, (1 << 19) + 4097,
                               (1 << 20) + 1])
def test_sort_tiles(ctx, width, bits, n):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64) >> np.uint64(rng.integers(0, bits))
    keys = keys.astype(np.uint32 if width == 32 else np.uint64)
    dt = torch.int32 if width == 32 else torch.int64
    k = torch.from_numpy(keys.view(np.int32 if width == 32 else np.int64)).cuda()
    ko, vo = torch.zeros(n, dtype=dt, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    call(f"ar_radix_sort_pairs_u{width}", ctx.handle, api.ptr(k), None, api.ptr(ko), api.ptr(vo),
         n, 0, bits, api.stream_handle())
    ctx.check()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(vo.cpu().numpy(), order.astype(np.int32))
    assert np.array_equal(ko.cpu().numpy().view(keys.dtype), keys[order])
