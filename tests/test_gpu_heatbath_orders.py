"""Short calls sweep the links in site order, longer ones in parity order, with
register caps by the number of blocks: the same sweeps give the same links and
rejections, bit for bit, however they are divided into calls."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64

pytestmark = pytest.mark.gpu


# one and several waves of blocks with each cap; halves that are no multiple of a block or of 32 sites
@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
@pytest.mark.parametrize("shape", [(4, 4, 4, 4), (4, 6, 8, 10), (18, 20, 18, 18), (20, 20, 20, 20), (20, 20, 20, 24), (24, 24, 20, 24)])
def test_calls_divide_without_a_trace(ctx, shape, prec):
    got = []
    for calls in ([(6, 1)], [(1, 1)] * 6, [(2, 1), (3, 1), (1, 1)]):
        with ctx.lattice(shape, prec) as lat:
            lat.generate(5, 0.5)
            rejected = sum(lat.heatbath(5.9, n, over, 11) for n, over in calls)
            for n in ([5] if len(calls) == 1 else [1, 2, 1, 1]):
                lat.overrelax(n)
            rejected += sum(lat.heatbath(5.9, n, 0, 11) for n in ([3] if len(calls) == 1 else [1, 1, 1]))
            got.append((rejected, lat.download()))
    assert all(r == got[0][0] and np.array_equal(u, got[0][1]) for r, u in got[1:])
