"""A radix sort whose look-back gives up (AR_SORT_TEST_MUTE_FIRST_TILE: tile 0 of every digit pass
publishes nothing) reports AR_ERR_TIMEOUT and still returns the sorted pairs: what follows a sort
indexes with its order.  Both tile shapes, 8- and 9-bit digits, both rankings, a last tile of one
key, keys that share one digit."""
import numpy as np
import pytest

from test_gpu_sort_paths import AR_SORT_RANK_MATCH, AR_SORT_TEST_MUTE_FIRST_TILE
from diploma_thesis_b200._lib import lib
from gpu_util import P, S, dev, empty, host

import torch

pytestmark = pytest.mark.gpu

AR_ERR_TIMEOUT = 3


@pytest.mark.parametrize("flags", [0, AR_SORT_RANK_MATCH])
@pytest.mark.parametrize("n,bits", [(2049, 8), (30_001, 24), (30_001, 25), ((1 << 19) - 1, 16),
                                    ((1 << 19) + 1, 24), (700_000, 27), (100_000, 0)])
def test_order_is_right_after_a_timeout(ctx, n, bits, flags):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n).astype(np.uint32)
    vals = rng.integers(0, 1 << 31, n).astype(np.uint32)
    ko, vo = empty(n, torch.int32), empty(n, torch.int32)
    assert lib.ar_radix_sort_pairs_u32_ex(ctx.handle, P(dev(keys)), P(dev(vals)), P(ko), P(vo), n,
                                          0, max(bits, 8), flags | AR_SORT_TEST_MUTE_FIRST_TILE,
                                          S()) == 0
    assert ctx.status() == AR_ERR_TIMEOUT
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(host(ko, np.uint32), keys[order])
    assert np.array_equal(host(vo, np.uint32), vals[order])
