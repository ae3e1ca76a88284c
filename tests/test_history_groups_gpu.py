"""The plain form runs the batches of a dose run together, as many as their
tallies fit, its histories taken from a counter by as many lanes of a warp as
hold them.  A history's stream depends on its index alone, so neither the
group, the lanes nor the block change the dose: the fixed-scratch run (groups
of three batches on 262,144 voxels, of ten on small phantoms) and blocks of
other sizes agree with run_beam up to the summation order of the FP64 tallies
(some thousand additions per voxel of relative rounding 1.1e-16 each: 1e-12)."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,histories,nbatch", [(64, 1003, 10), (64, 20, 2), (20, 7, 7), (20, 4001, 4), (40, 3000, 20)])
def test_dose_independent_of_groups_and_lanes(n, histories, nbatch):
    from ompmc_b200.engine import PLAIN_FP64, Engine
    ph = cases._phantom("water", n, 300.0 / n)
    tables = cases._tables(tuple(ph.media))
    call = dict(ncase=histories, nbatch=nbatch, seed=77, mono_energy=4.0, collimator=(-4.0, 4.0, -3.0, 3.0))
    ref = None
    for block in (0, 32, 96):
        eng = Engine(tables, ph, block=block)
        runs = [eng.run_beam(mode=PLAIN_FP64, **call), eng.run_beam_noalloc(**call)]
        eng.close()
        for dose, unc, st in runs:
            assert st["flags"] == 0 and st["histories"] == histories // nbatch * nbatch
            if ref is None:
                ref = dose, unc, st
                assert (dose > 0).sum() > 10
            np.testing.assert_allclose(dose, ref[0], rtol=1e-12)
            assert st["esrc"] == pytest.approx(ref[2]["esrc"], rel=1e-12)
