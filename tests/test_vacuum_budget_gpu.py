"""A particle that crosses vacuum voxels takes the same trajectory wherever its
events are cut: in cycles of any budget and in the drain, on uniform and
stretched grids.  The dose then agrees up to the summation order of the FP64
tallies (1e-9 per voxel), its uncertainty to 1e-6.  FP64: budgets only (its
drain is a kernel with roundings of its own)."""
import numpy as np
import pytest

from ompmc_b200 import assets
from perf import cases

pytestmark = pytest.mark.gpu


def _phantom(kind, stretched):
    """Half of the voxels are vacuum, so that most steps end at one."""
    p = cases._phantom(kind, 20, 5.0)
    rng = np.random.default_rng(11)
    med, rho = p.med.copy(), p.rho.copy()
    hole = rng.random(med.shape) < 0.5
    med[hole], rho[hole] = 0, 0.0
    bounds = [b.copy() for b in (p.xb, p.yb, p.zb)]
    if stretched:
        for b in bounds:
            b[1:-1] += rng.uniform(-0.3, 0.3, len(b) - 2) * (b[1] - b[0])
    return assets.Phantom(list(p.media), *bounds, med, rho, "holes")


CUTS = [dict(drain_particles=-1, electron_tsteps=1000), dict(drain_particles=-1, electron_tsteps=1, tail_boost=1), dict(),
        dict(electron_tsteps=3, drain_particles=1)]


@pytest.mark.parametrize("kind,stretched,source", [
    ("water", False, dict(mono_energy=6.0)), ("slab", True, dict(mono_energy=12.0)),
    ("slab", False, dict(mono_energy=8.0, charge=-1)), ("water", True, dict(mono_energy=4.0, charge=1))])
@pytest.mark.parametrize("form,nsplit", [("fp32", 1), ("fp32", 4), ("fp64", 1)])
def test_dose_independent_of_cuts_at_vacuum(kind, stretched, source, form, nsplit):
    from ompmc_b200.engine import EVENT_FP32, EVENT_FP64, Engine
    ph = _phantom(kind, stretched)
    tables = cases._tables(tuple(ph.media))
    ref = None
    for kw in CUTS if form == "fp32" else CUTS[:2]:
        eng = Engine(tables, ph, nsplit=nsplit, **kw)
        dose, unc, st = eng.run_beam(5000, 5, seed=21, mode=EVENT_FP32 if form == "fp32" else EVENT_FP64,
                                     collimator=(-2.0, 2.0, -3.0, 3.0), **source)
        eng.close()
        assert st["flags"] == 0
        if ref is None:
            ref = dose, unc
            assert (dose > 0).sum() > 50
        hit = ref[0] > 0
        assert np.array_equal(dose > 0, hit), kw
        np.testing.assert_allclose(dose, ref[0], rtol=1e-9, err_msg=str(kw))
        np.testing.assert_allclose(unc[hit], ref[1][hit], rtol=1e-6, atol=1e-9, err_msg=str(kw))
