"""The stage's forms -- split (lattices of up to 148 tiles of 32 sites), plaquettes
(FP32 from 8192 sites on, FP64 from 18432 to 200000), staples -- at tile edges:
slices and volumes that are no multiple of 32 sites, extents of 4 (every neighbour wraps), volumes on both sides of the
rule's line.

Tolerance: a force coordinate sums six projections of products of unit-size
matrices, each about 40 roundings: 6 * 40 * 2^-24 = 1.5e-5.  The reference is
the FP64 force of the same (float) links, itself checked against the oracle."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64
from msc_project_b200.lgf import Job
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4, 6), (4, 6, 8, 10), (8, 8, 8, 8), (4, 4, 4, 74), (4, 4, 4, 76), (8, 8, 8, 14), (8, 8, 8, 16), (4, 4, 4, 130), (10, 14, 10, 6), (6, 10, 14, 18), (4, 50, 6, 10)]


@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_force_matches_fp64(ctx, shape):
    U = O.generate_G(shape, 17, 0.5).astype(np.float32).astype(np.float64)
    with ctx.lattice(shape, FP64) as lat:
        lat.upload(U)
        want = lat.debug_gradient()
    with ctx.lattice(shape, FP32MIXED) as lat:
        lat.upload(U)
        got = lat.debug_gradient()
        assert np.array_equal(lat.download(), U)
        lat.flow(0.01, 1, 0, measure_at_t0=False)  # one step, both forms against FP64
        step = lat.download()
    with ctx.lattice(shape, FP64) as lat:
        lat.upload(U)
        lat.flow(0.01, 1, 0, measure_at_t0=False)
        step64 = lat.download()
    assert np.max(np.abs(got - want)) < 1.5e-5
    # three exponentials of eps times such a force, three products: 9 * 2^-24 * ~8 roundings
    assert np.max(np.abs(step - step64)) < 5e-6


@pytest.mark.parametrize("shape", [(4, 4, 4, 4), (4, 6, 8, 10), (8, 8, 8, 8), (4, 4, 4, 74), (4, 4, 4, 76), (12, 12, 8, 14),
                                   (12, 12, 8, 16), (10, 14, 10, 14), (4, 4, 4, 290), (20, 20, 20, 24), (20, 20, 20, 26)])
def test_fp64_steps_match_the_oracle(ctx, shape):
    U = O.generate_G(shape, 23, 0.5)
    want = U
    for _ in range(2):
        want = O.rk3_step(want, shape, 0.01)
    with ctx.lattice(shape, FP64) as lat:
        lat.upload(U)
        lat.flow(0.01, 2, 0, measure_at_t0=False)
        assert np.max(np.abs(lat.download() - np.asarray(want).reshape(-1))) < 1e-13  # six stages of ~30 roundings


@pytest.mark.parametrize("prec, shapes", [
    (FP32MIXED, [(6, 10, 14, 18), (4, 4, 4, 4), (8, 8, 8, 14), (8, 8, 8, 16), (16, 16, 8, 10)]),
    (FP64, [(12, 12, 8, 14), (8, 8, 8, 8), (10, 14, 10, 14), (12, 12, 8, 16)]),
    # more small tiles than SMs: the batch takes the staple form with the split form's sums
    (FP32MIXED, [(8, 8, 8, 8), (4, 6, 8, 10), (6, 10, 14, 18), (4, 4, 4, 74)]),
    (FP64, [(8, 8, 8, 8), (4, 6, 8, 10), (12, 12, 8, 14), (4, 4, 4, 74)])])
def test_results_do_not_depend_on_the_batch(ctx, prec, shapes):
    """Small and large lattices in one batch take different forms and launches; each gives the bits it gives alone."""
    links = [O.generate_G(s, 40 + i, 0.5) for i, s in enumerate(shapes)]
    jobs = [Job(s, prec, links=u, nsteps=4 + 2 * (i % 2), meas_every=2, reunit_every=3, want_links=True, slices=True)
            for i, (s, u) in enumerate(zip(shapes, links))]
    ctx.batch_run(jobs)
    for j, u in zip(jobs, links):
        with ctx.lattice(j.shape, prec) as lat:
            lat.upload(u)
            r = lat.flow(j.eps, j.nsteps, 2, reunit_every=3, slices=True)
            assert np.array_equal(r.E, j.result.E) and np.array_equal(r.Q, j.result.Q)
            assert np.array_equal(r.E_slice, j.result.E_slice) and np.array_equal(r.Q_slice, j.result.Q_slice)
            assert np.array_equal(lat.download(), j.links_out)
