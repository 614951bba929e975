"""The autotuner times what a lattice's kernels read.  Lattices of the plaquette
and the split form leave the staple kernel's block size to the lattices that run
it, alone or in a batch; results never depend on it."""
import numpy as np
import pytest

from msc_project_b200 import FP32MIXED, FP64, Context, Job

pytestmark = pytest.mark.gpu


def jobs(spec, prec):
    return [Job(s, prec, seed=60 + i, nsteps=3, meas_every=3, want_links=True) for s, n in spec for i in range(n)]


@pytest.mark.parametrize("prec", [FP64, FP32MIXED])
@pytest.mark.parametrize("tuned, other", [((8, 8, 8, 8), (8, 8, 8, 14)), ((16, 16, 8, 10), (10, 10, 12, 10)),
                                          ((20, 20, 20, 24), (16, 24, 24, 24))])
def test_tuning_one_form_leaves_the_others_block_size(prec, tuned, other):
    with Context(0) as plain, Context(0) as c:
        keys = ("stage_threads", "stage_order", "stage_budget_kb")
        t = c.autotune_tiles(prec, tuned)
        assert c.get_tiles(prec, tuned) == t
        if not (prec == FP64 and tuned == (16, 16, 8, 10)):  # the one that runs the staple kernel itself
            assert [c.get_tiles(prec, other)[k] for k in keys] == [plain.get_tiles(prec, other)[k] for k in keys]
        c.set_tiles(prec, tuned, stage_threads=256)  # the caller's choice holds for the volume class
        assert c.get_tiles(prec, other)["stage_threads"] == 256


@pytest.mark.parametrize("spec, threads", [([((8, 8, 8, 8), 64)], 384), ([((8, 8, 8, 8), 7)], 128), ([((8, 8, 8, 8), 2)], 256),
                                           ([((6, 10, 10, 8), 2)], 384), ([((6, 10, 10, 8), 3)], 128),
                                           ([((8, 8, 8, 8), 16), ((12, 12, 12, 12), 1)], 384)])
def test_a_batch_sizes_its_blocks_by_the_staple_lattices(spec, threads):
    """FP64: 96-site tiles where the small lattices together fill the SMs with them, 64-site ones up to one per SM."""
    with Context(0) as c:
        js = jobs(spec, FP64)
        assert c.batch_run(js).block_threads == threads
        for j in (js[0], js[-1]):
            with c.lattice(j.shape, FP64) as lat:
                lat.generate(j.seed, 0.5)
                r = lat.flow(0.01, 3, 3)
                assert np.array_equal(r.Q, j.result.Q) and np.array_equal(lat.download(), j.links_out)


def test_one_lattice_timed_does_not_size_a_larger_batch():
    """A first batch of one lattice times its volume class; later batches of many take the size of their own launches."""
    shape = (6, 10, 10, 8)
    with Context(0) as c:
        c.batch_run(jobs([(shape, 1)], FP64))
        for n, threads in ((2, 384), (3, 128), (8, 384)):
            js = jobs([(shape, n)], FP64)
            assert c.batch_run(js).block_threads == threads
        c.set_tiles(FP64, shape, stage_threads=256)  # the caller's choice holds
        assert c.batch_run(jobs([(shape, 2)], FP64)).block_threads == 256
