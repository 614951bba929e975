"""Lattices of different sizes alive at once.  The measurement kernels' blocks
follow the size of a group's lattices, and the shared-memory limit of a kernel
is one setting for the whole process: a group of small lattices must not lower
it under one of large lattices, in the same context, in another one or beside a
running server.  Results are those of each lattice alone, bit for bit."""
import time

import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64, Context, Job, Server
from msc_project_b200 import _capi as C

pytestmark = pytest.mark.gpu

LARGE, SMALL = (16, 16, 16, 16), (4, 6, 8, 10)  # the largest measurement blocks, and the smallest


def observe(lat):
    """Everything that launches the measurement kernels outside a captured graph, and one graph launch."""
    return [*lat.site_densities(), *lat.measure_flowed(), *lat.debug_fields(), *lat.measure(slices=True)]


def alone(shape, prec):
    with Context(0) as c, c.lattice(shape, prec) as lat:
        lat.generate(3)
        return observe(lat)


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b, strict=True))


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
@pytest.mark.parametrize("other_context", [False, True])
def test_a_small_lattice_leaves_a_large_one_its_launches(ctx, prec, other_context):
    large, small = alone(LARGE, prec), alone(SMALL, prec)
    with Context(0) as second, ctx.lattice(LARGE, prec) as a, ctx.lattice(LARGE, prec) as flowed, \
            (second if other_context else ctx).lattice(SMALL, prec) as b:
        for lat in (a, flowed, b):
            lat.generate(3)
        assert same(observe(a), large)
        flowed.flow(0.01, 0, 0, measure_at_t0=False)  # its kernels are set up, its measurement not captured yet
        assert same(observe(b), small)
        assert same(observe(a), large)
        assert same(flowed.measure(slices=True), large[-4:])
        assert same(observe(b), small)


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
def test_a_small_lattice_beside_a_server(ctx, prec):
    """The server's first measurement is captured after a small group was made elsewhere."""
    job = dict(shape=LARGE, precision=prec, seed=3, eps=0.01, nsteps=6000, meas_every=6000, measure_at_t0=False, slices=True)
    with ctx.lattice(LARGE, prec) as lat:
        lat.generate(3)
        ref = lat.flow(0.01, 6000, 6000, measure_at_t0=False, slices=True)
    with Context(0) as served, Context(0) as second, Server(served, 1 << 28, max_active=2) as srv:
        j = Job(**job)
        jid = srv.submit(j)
        deadline = time.monotonic() + 60
        while srv.poll(jid)[1].steps_done < 1 and time.monotonic() < deadline:
            pass
        with second.lattice(SMALL, prec) as b:
            b.generate(3)
            b.measure()
        st = srv.wait(jid, 120)
        assert st.state == C.LGF_JOB_DONE, st.error
    for k in ("E", "Q", "E_slice", "Q_slice"):
        assert np.array_equal(getattr(j.result, k), getattr(ref, k)), k
