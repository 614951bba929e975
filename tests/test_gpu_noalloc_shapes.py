"""lgf_measure_noalloc at tile edges: slices that end inside a 32-site tile (its
idle lanes still take part in the paired link loads), odd numbers of 32-site
tiles, extents of 4, and a largest case near its scratch's slice bound, against
lgf_measure on the same links.  Both sum the same terms in FP64: 1e-12."""
import ctypes

import numpy as np
import pytest
from conftest import q_err, rel_err

from msc_project_b200 import FP64
from msc_project_b200 import _capi as C
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 4, 4, 4), (4, 6, 6, 6), (6, 4, 6, 10), (256, 4, 4, 4), (8, 10, 14, 18)])
def test_noalloc_matches_measure(ctx, shape):
    import torch
    U = O.generate_G(shape, 13, 0.5)
    with ctx.lattice(shape, FP64) as lat:
        lat.upload(U)
        E, Q, es, qs = lat.measure(slices=True)
    dev = torch.from_numpy(U).to("cuda:0")
    out = torch.full((2 + 2 * shape[0],), float("nan"), dtype=torch.float64, device="cuda:0")
    ptr = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))  # noqa: E731
    rc = ctx.lib.lgf_measure_noalloc(ptr(dev), (ctypes.c_int * 4)(*shape), ptr(out),
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == C.LGF_OK
    got = out.cpu().numpy()
    assert rel_err(got[0], E) < 1e-12 and q_err(got[1], Q) < 1e-12
    assert rel_err(got[2:2 + shape[0]], es) < 1e-12
    assert np.max(np.abs(got[2 + shape[0]:] - qs)) < 1e-12


def test_noalloc_reads_the_links_as_given(ctx):
    """Links 1e-6 off SU(3): the result is that of the given matrices (full products), to rounding."""
    import torch
    shape = (4, 6, 4, 6)
    rng = np.random.default_rng(17)
    U = np.ascontiguousarray(O.generate_G(shape, 17, 0.5)).reshape(-1)
    U = U + 1e-6 * rng.standard_normal(U.size)
    dev = torch.from_numpy(U).to("cuda:0")
    out = torch.empty(2 + 2 * shape[0], dtype=torch.float64, device="cuda:0")
    ptr = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))  # noqa: E731
    assert ctx.lib.lgf_measure_noalloc(ptr(dev), (ctypes.c_int * 4)(*shape), ptr(out),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == C.LGF_OK
    got = out.cpu().numpy()
    assert rel_err(got[0], O.energy_density(U, shape)) < 1e-12 and q_err(got[1], O.topological_charge(U, shape)) < 1e-12
