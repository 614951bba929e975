"""Sweeps on parity-ordered links at the edges of the order: rows of two sites
of each parity, every extent different, volumes whose halves are no multiple of
32 sites, and one of more than 444 blocks (the kernel of four blocks per SM).

Overrelaxation leaves the Wilson action unchanged only if every link meets its
own staple, so a wrong neighbour shows at once: 30 sweeps of FP64 rounding stay
below 1e-12, of FP32 (three 2x2 rotations of unit rows per link and sweep)
below 30 * 12 * 2^-24 = 2e-5."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
@pytest.mark.parametrize("shape", [(4, 4, 4, 4), (4, 6, 8, 10), (6, 10, 4, 6), (10, 4, 6, 8), (18, 20, 18, 18)])
def test_overrelaxation_keeps_the_action(ctx, shape, prec):
    with ctx.lattice(shape, prec) as lat:
        lat.generate(5, 0.5)
        p0 = lat.plaquette()
        before = lat.download()
        lat.overrelax(0)
        assert np.array_equal(lat.download(), before)
        lat.overrelax(30)
        p1 = lat.plaquette()
        after = lat.download()
        u, _ = lat.unitarity()
    tol = 1e-12 if prec == FP64 else 2e-5
    assert abs(p1 - p0) < tol and u < (1e-12 if prec == FP64 else 1e-4)
    assert np.all(np.max(np.abs(after - before).reshape(-1, 18), axis=1) > 1e-3)  # every link moved


@pytest.mark.parametrize("shape", [(4, 6, 8, 10), (6, 10, 4, 6)])
def test_plaquette_matches_host(ctx, shape):
    U = O.generate_G(shape, 3, 0.5)
    V = int(np.prod(shape))
    M = (U.reshape(V, 4, 18)[:, :, 0::2] + 1j * U.reshape(V, 4, 18)[:, :, 1::2]).reshape(*shape, 4, 3, 3)
    tot = 0.0
    for m in range(4):
        for n in range(m + 1, 4):
            a, b = M[..., m, :, :], np.roll(M[..., n, :, :], -1, axis=m)
            c, d = np.roll(M[..., m, :, :], -1, axis=n), M[..., n, :, :]
            tot += np.einsum("...ij,...jk,...lk,...il->...", a, b, c.conj(), d.conj()).real.sum()
    with ctx.lattice(shape, FP64) as lat:
        lat.upload(U)
        assert abs(lat.plaquette() - tot / (18 * V)) < 1e-13
