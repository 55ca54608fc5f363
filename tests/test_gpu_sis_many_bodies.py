"""The sequential-impulse solver beyond the body counts whose state fits shared memory: velocities in
global memory (from 7,041 bodies on), the level walk's too (from 25,601 on), with plain and odd
contacts, runs cut at chunks, and few contacts per body.  Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_sis import _synthetic_contacts
from test_gpu_sis_odd import _list
from test_gpu_sis_schedule import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.0, 0.1])
@pytest.mark.parametrize("nb,count", [(7040, 9000), (7041, 9000), (8000, 3000), (25600, 5000),
                                      (25601, 5000), (30000, 20000)])
def test_many_bodies(ctx, nb, count, share):
    rng = np.random.default_rng(nb + count)
    pairs = _list(nb, count, share, rng)
    pairs[::2] = [(a, b) if b < 0 else (b, a) for a, b in pairs[::2]]  # runs of one and two
    _check(ctx, *_synthetic_contacts(rng, nb, pairs), 3)
