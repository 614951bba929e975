"""The first call on a small lattice sets up its kernels' lists without another
chunk of device memory from the driver (mapping one takes longer than the call),
and gives everything back with the lattice."""
import pytest

from msc_project_b200 import FP32MIXED, FP64, Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
def test_the_first_measurement_maps_no_memory(prec):
    import torch
    free = lambda: torch.cuda.mem_get_info(0)[0]  # noqa: E731
    with Context(0) as c:
        for warm in (True, False):  # kernels are loaded, and graphs first captured, in the first round
            start = free()
            with c.lattice((8, 8, 8, 8), prec) as lat:
                lat.generate(3)
                lat.unitarity()
                before = free()
                lat.measure()
                lat.flow(0.01, 2, 1)
                lat.site_densities()
                assert warm or free() == before
        assert free() == start
