"""A batch's results come back whole whatever their size: jobs that share an
area, a job larger than it (16 MiB) between them, jobs without measurements and
jobs without a place for them."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64, Context, Job

pytestmark = pytest.mark.gpu


def test_large_and_empty_results():
    shape = (64, 4, 4, 4)  # 1040 bytes per measurement
    jobs = [Job((4, 6, 8, 10), FP64, seed=1, nsteps=4, meas_every=2, slices=True),
            Job((4, 4, 4, 6), FP64, seed=2, nsteps=3, meas_every=0, measure_at_t0=False, want_links=True),
            Job(shape, FP32MIXED, seed=3, nsteps=16200, meas_every=1, eps=1e-4, slices=True),
            Job((6, 4, 4, 4), FP32MIXED, seed=4, nsteps=5, meas_every=1, want_links=True)]
    with Context(0) as c:
        c.batch_run(jobs)
        for j in jobs:
            with c.lattice(j.shape, j.precision) as lat:
                lat.generate(j.seed, 0.5)
                r = lat.flow(j.eps, j.nsteps, j.meas_every, 0.0, j.measure_at_t0, 0, slices=j.slices)
                for k in ("t", "E", "Q") + (("E_slice", "Q_slice") if j.slices else ()):
                    assert np.array_equal(getattr(j.result, k), getattr(r, k)), (j.shape, k)
                assert len(j.result.E) == 0 or np.all(j.result.E != 0)
                if j.want_links:
                    assert np.array_equal(lat.download(), j.links_out)
