"""The measurement's loop and plane kernels at the edges of their tiles: slices
that are no multiple of 32 sites, the smallest extents (every shift wraps),
extents above a plane unit's sites (row tiles that recompute three rows before
their first output) and lattices of one and of many blocks, against the oracle.

Tolerances: a site's F coordinate is a sum of 24 products of at most eight
unit-size matrices, each product about 20 roundings: below 1e3 eps.  e(x) and
q(x) add some 50 products of such coordinates (|F| < 3): FP64 1e-12, FP32 1e-4
of the largest density."""
import numpy as np
import pytest
from conftest import q_err, rel_err

from msc_project_b200 import FP32MIXED, FP64
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4, 4), (4, 6, 8, 10), (6, 4, 10, 6), (10, 6, 6, 18), (100, 4, 4, 4), (4, 198, 4, 6), (6, 4, 102, 4),
          (4, 4, 4, 50), (12, 14, 16, 18)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
def test_site_densities_and_sums_match_the_oracle(ctx, shape, prec):
    U = O.generate_G(shape, 31, 0.5)
    if prec == FP32MIXED:  # the oracle measures the links the GPU holds
        U = U.astype(np.float32).astype(np.float64)
    eo, qo = O.site_densities(U, shape)
    with ctx.lattice(shape, prec) as lat:
        lat.upload(U)
        E, Q, es, qs = lat.measure(slices=True)
        e, q = lat.site_densities()
        assert np.array_equal(lat.download(), U)  # the pass leaves the links alone
        E2, Q2, es2, qs2 = lat.measure(slices=True)
    assert (E, Q) == (E2, Q2) and np.array_equal(es, es2) and np.array_equal(qs, qs2)
    tol = 1e-12 if prec == FP64 else 1e-4
    assert np.max(np.abs(e - eo)) < tol * np.max(np.abs(eo))
    assert np.max(np.abs(q - qo)) < tol * max(1.0, np.max(np.abs(qo)))
    # sums of the engine's own densities: double rounding only
    n0 = shape[0]
    assert rel_err(es, e.reshape(n0, -1).mean(1)) < 1e-13
    assert np.max(np.abs(qs - q.reshape(n0, -1).sum(1) / (4 * np.pi ** 2))) < 1e-13 * np.sum(np.abs(q))
    assert rel_err(E, e.mean()) < 1e-13 and q_err(Q, q.sum() / (4 * np.pi ** 2)) < 1e-12


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
def test_units_and_tiles_give_identical_results(ctx, prec):
    """Block sizes of both kernels (chosen by lattice size and measurement split) change no bit."""
    shape = (12, 14, 16, 18)
    U = O.generate_G(shape, 5, 0.5)
    got = []
    for split in (1, 2):
        ctx.set_tiles(prec, shape, meas_split=split)
        with ctx.lattice(shape, prec) as lat:
            lat.upload(U)
            got.append(lat.measure(slices=True))
    small = ctx.batch_run  # the same lattice in a group sized for more sites
    from msc_project_b200.lgf import Job
    jobs = [Job(s, prec, links=O.generate_G(s, 5, 0.5), nsteps=0, meas_every=0, slices=True)
            for s in (shape, (4, 4, 4, 4), (4, 100, 4, 6))]
    small(jobs)
    r = jobs[0].result
    got.append((r.E[0], r.Q[0], r.E_slice[0], r.Q_slice[0]))
    for g in got[1:]:
        assert g[0] == got[0][0] and g[1] == got[0][1]
        assert np.array_equal(g[2], got[0][2]) and np.array_equal(g[3], got[0][3])
