"""The sequential-impulse sweeps where their block, schedules and forms change: either block size,
more contacts in a step than lane pairs, more sweeps than one schedule holds, a body paired with
itself, divisors and dividends outside the reciprocal division's range, bodies at rest.  Bit for bit
against the oracle's sequential loop."""
import numpy as np
import pytest

from oracle import cpu
from test_gpu_sis import _solve_gpu, _synthetic_contacts

pytestmark = pytest.mark.gpu


def _check(ctx, contacts, cms, vel, ang, ib, mass, iterations):
    gv, gw, gacc = _solve_gpu(ctx, contacts, cms, vel, ang, ib, mass, iterations)
    rv, rw, *racc = cpu.sequential_impulse(contacts, cms, vel, ang, ib, mass,
                                           iterations=iterations)
    assert np.array_equal(gv, rv) and np.array_equal(gw, rw)
    for got, want in zip(gacc, racc):
        assert np.array_equal(got, want)


def _pairs(rng, nb, count):
    b1 = np.sort(rng.integers(0, nb, count))
    return [(int(a), int((a + d) % nb)) for a, d in zip(b1, rng.integers(1, min(nb, 40), count))]


@pytest.mark.parametrize("nb,count,iterations", [(2, 1, 33), (40, 500, 70), (1023, 9000, 18),
                                                 (1024, 9000, 18), (4000, 3000, 2)])
def test_schedules(ctx, nb, count, iterations):
    rng = np.random.default_rng(nb)
    _check(ctx, *_synthetic_contacts(rng, nb, _pairs(rng, nb, count)), iterations)


@pytest.mark.parametrize("form", ["self", "masses", "dividends", "rest"])
def test_forms(ctx, form):
    rng = np.random.default_rng(len(form))
    pairs = _pairs(rng, 60, 900)
    if form == "self":
        pairs[::50] = [(a, a) for a, _ in pairs[::50]]
    contacts, cms, vel, ang, ib, mass = _synthetic_contacts(rng, 60, pairs)
    if form == "masses":
        mass[::7] = np.float32(2.0 ** 45)
    elif form == "dividends":  # impulses below the range: tiny velocities and biases
        vel *= np.float32(2.0 ** -80)
        ang *= np.float32(2.0 ** -80)
        contacts["bias"] *= np.float32(2.0 ** -80)
    elif form == "rest":
        vel[:], ang[:] = 0, 0
        contacts["bias"][::2] = 0
    _check(ctx, contacts, cms, vel, ang, ib, mass, 18)
