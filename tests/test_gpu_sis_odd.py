"""The sequential-impulse sweeps on lists with odd contacts (one body, one body twice, divisors outside
the reciprocal division's range) among plain ones: warps with none, with some, only odd ones, odd
ones in the last half-filled warp and beyond a block's first round, frictions carried over more than
32 sweeps, zero and tiny dividends.  Bit for bit against the oracle's sequential loop."""
import numpy as np
import pytest

from test_gpu_sis import _synthetic_contacts
from test_gpu_sis_schedule import _check

pytestmark = pytest.mark.gpu


def _list(nb, count, share, rng):
    """Contacts sorted by first body, `share` of them with one body."""
    b1 = np.sort(rng.integers(0, nb, count))
    b2 = (b1 + rng.integers(1, max(2, min(nb, 40)), count)) % nb
    b2[rng.random(count) < share] = -1
    return [(int(a), int(b)) for a, b in zip(b1, b2)]


@pytest.mark.parametrize("share", [0.003, 0.1, 1.0])
@pytest.mark.parametrize("nb,count,iterations", [(2, 33, 40), (60, 900, 40), (700, 2100, 18),
                                                 (1100, 6000, 18)])
def test_shares_of_one_body_contacts(ctx, nb, count, iterations, share):
    rng = np.random.default_rng(nb)
    _check(ctx, *_synthetic_contacts(rng, nb, _list(nb, count, share, rng)), iterations)


@pytest.mark.parametrize("form", ["self", "masses", "heavy inertia", "dividends", "rest"])
def test_odd_forms_with_one_body_contacts(ctx, form):
    rng = np.random.default_rng(len(form))
    pairs = _list(80, 1200, 0.1, rng)
    if form == "self":
        pairs[::40] = [(a, a) for a, _ in pairs[::40]]
    contacts, cms, vel, ang, ib, mass = _synthetic_contacts(rng, 80, pairs)
    if form == "masses":  # 1 / mass out of range, and with it mc, k1 and k2
        mass[::5] = np.float32(2.0 ** 45)
        mass[1::5] = np.float32(2.0 ** -45)
    elif form == "heavy inertia":  # k1 and k2 out of range, mc mostly set to 1
        mass[::3] = np.float32(2.0 ** 60)
        ib[::3] *= np.float32(2.0 ** -60)
    elif form == "dividends":
        vel *= np.float32(2.0 ** -80)
        ang *= np.float32(2.0 ** -80)
        contacts["bias"] *= np.float32(2.0 ** -80)
    elif form == "rest":
        vel[:], ang[:] = 0, 0
        contacts["bias"][::2] = 0
    _check(ctx, contacts, cms, vel, ang, ib, mass, 18)
