"""ar_sequential_impulse in an arena that holds no more than 272 bytes per contact slot and 8 per
body, reserved before, and inside a stream capture after a call of one sweep: it allocates nothing,
cuts its sweeps into as many schedules as it needs and gives the oracle's results bit for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

from diploma_thesis_b200 import _lib, api
from gpu_util import P, call, dev, empty, host
from oracle import cpu
from test_gpu_sis import _synthetic_contacts

pytestmark = pytest.mark.gpu


class _List:
    """A contact list on the device, with room for `capacity` contacts."""

    def __init__(self, nb, count, capacity):
        rng = np.random.default_rng(count)
        b1 = np.sort(rng.integers(0, nb, count))
        b2 = (b1 + rng.integers(1, 30, count)) % nb
        b2[::37] = -1
        self.args = _synthetic_contacts(rng, nb, list(zip(b1.tolist(), b2.tolist())))
        contacts, cms, vel, ang, ib, mass = self.args
        self.nb, self.count, self.capacity = nb, count, capacity

        def room(a):
            t = empty((capacity, *a.shape[1:]), torch.int32 if a.dtype == np.int32 else torch.float32)
            t[:count] = dev(a)
            return t
        self.t = [room(contacts[k]) for k in ("normal", "point", "body1", "body2", "bias")]
        self.acc = [empty(capacity) for _ in range(3)]
        self.bodies = [dev(a) for a in (cms, vel, ang, ib, mass)]
        self.first = [t.clone() for t in self.bodies]
        self.n = dev(np.array([count], np.int32))
        self.prm = api.sim_params(0.01, (0, 0, 0), 0.02, (4, 4, 4))
        self.prm.ar_friction, self.prm.rb_friction = 0.3, 0.1

    def reset(self):
        for t, f in zip(self.bodies, self.first):
            t.copy_(f)
        for a in self.acc:
            a.zero_()

    def solve(self, ctx, iterations):
        cms, vel, ang, ib, mass = self.bodies
        call("ar_sequential_impulse", ctx.handle, C.byref(self.prm), P(self.n), self.capacity,
             *(P(t) for t in self.t), *(P(a) for a in self.acc), self.nb, P(cms), P(vel), P(ang),
             P(ib), P(mass), iterations, C.c_void_p(torch.cuda.current_stream().cuda_stream))

    def check(self, iterations):
        rv, rw, *racc = cpu.sequential_impulse(*self.args, iterations=iterations)
        assert np.array_equal(host(self.bodies[1]), rv) and np.array_equal(host(self.bodies[2]), rw)
        for got, want in zip(self.acc, racc):
            assert np.array_equal(host(got)[:self.count], want)


@pytest.fixture()
def own_ctx():
    c = api.Context(0)
    yield c
    _lib.lib.ar_test_fail_allocations(-1)
    c.close()


@pytest.mark.parametrize("nb,count,capacity,iterations", [
    (700, 30_000, 30_000, 18), (1500, 30_000, 70_000, 18), (50, 400, 400_000, 33)])
def test_reserved_arena_is_enough(own_ctx, nb, count, capacity, iterations):
    lst = _List(nb, count, capacity)
    call("ar_ctx_reserve", own_ctx.handle, 272 * capacity + 8 * nb + 24)
    _lib.lib.ar_test_fail_allocations(0)
    lst.solve(own_ctx, iterations)
    own_ctx.check()
    lst.check(iterations)


@pytest.mark.parametrize("reserve", [False, True])
def test_captured_after_a_call_of_one_sweep(own_ctx, reserve):
    lst = _List(600, 20_000, 20_000)
    if reserve:
        call("ar_ctx_reserve", own_ctx.handle, 272 * 20_000 + 8 * 600 + 24)
    lst.solve(own_ctx, 1)
    own_ctx.check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lst.solve(own_ctx, 18)
    for _ in range(2):
        lst.reset()
        graph.replay()
        own_ctx.check()
        lst.check(18)
