"""The per-function force is the one that the flow takes.  The stage forms group
a link's six staples differently, which shows in the last bits: two lattices of
one field, the second the first repeated along x0, have the same force and flow
bit for bit where their forms sum alike, and neither where they do not."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64
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
