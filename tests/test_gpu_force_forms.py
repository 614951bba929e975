"""The per-function force is the one that the flow takes.  The stage forms group
a link's six staples differently, which shows in the last bits: two lattices of
one field, the second the first repeated along x0, have the same force and flow
bit for bit where their forms sum alike, and neither where they do not."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64, Job
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
@pytest.mark.parametrize("shape, times", [((4, 4, 6, 6), 2), ((8, 8, 8, 8), 2), ((4, 6, 8, 10), 10), ((10, 10, 10, 10), 2),
                                          ((12, 12, 10, 10), 2)])
def test_the_debug_force_sums_as_the_flow_does(ctx, prec, shape, times):
    U = O.generate_G(shape, 29, 0.5)
    force, flowed = [], []
    for n in (1, times):
        with ctx.lattice((n * shape[0], *shape[1:]), prec) as lat:
            lat.upload(np.tile(U, n))
            force.append(lat.debug_gradient()[:U.size])
            lat.flow(0.01, 1, 0, measure_at_t0=False)
            flowed.append(lat.download()[:U.size])
    assert np.max(np.abs(force[0] - force[1])) < (1e-13 if prec == FP64 else 3e-5)  # twice 6 projections of 40 roundings
    assert np.array_equal(*force) == np.array_equal(*flowed)


# FP32 on both sides of each line of its forms (split, staple, plaquette), a partial last tile among them
@pytest.mark.parametrize("shape", [(4, 4, 4, 74), (4, 4, 6, 50), (8, 8, 8, 16), (4, 4, 6, 148), (4, 4, 4, 224), (6, 10, 14, 18)])
def test_fp32_lines_alone_and_batched(ctx, shape):
    """Force against FP64 (six projections of products of unit-size matrices, 40 roundings each: 1.5e-5); bits alone and batched."""
    U = O.generate_G(shape, 31, 0.5).astype(np.float32).astype(np.float64)
    with ctx.lattice(shape, FP64) as lat:
        lat.upload(U)
        want = lat.debug_gradient()
    with ctx.lattice(shape, FP32MIXED) as lat:
        lat.upload(U)
        assert np.max(np.abs(lat.debug_gradient() - want)) < 1.5e-5
        r = lat.flow(0.01, 6, 2, reunit_every=3, slices=True)
        links = lat.download()
    jobs = [Job(s, FP32MIXED, links=U if s == shape else None, seed=5, nsteps=6, meas_every=2, reunit_every=3, slices=True, want_links=True)
            for s in (shape, (8, 8, 8, 8), (4, 6, 8, 10), (4, 4, 6, 148), (6, 10, 14, 18))]
    ctx.batch_run(jobs)
    assert np.array_equal(jobs[0].links_out, links)
    assert all(np.array_equal(getattr(jobs[0].result, k), getattr(r, k)) for k in ("E", "Q", "E_slice", "Q_slice"))
