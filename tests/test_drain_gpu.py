"""FP32 particles take the same trajectories wherever they run: in the transport
cycles (random numbers from shared memory, interactions in a kernel of their
own or in place), in the drain (an electron's turn out of line, work handed
between warps), cut into events of any budget, from one particle to more than
the drain has warps or lanes.  The dose then agrees up to the summation order
of the FP64 tallies (1e-9 per voxel, as tests/test_event_budget_gpu.py; here
with textbook physics data, so that it needs no physics files)."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu

FORMS = [dict(drain_particles=-1), dict(), dict(drain_particles=1 << 22), dict(drain_particles=1),
         dict(drain_particles=-1, electron_interact_kernel=0, electron_tsteps=3, tail_boost=1),
         dict(electron_tsteps=2, block=96, inflight=1 << 16)]


@pytest.mark.parametrize("kind,source,nsplit,histories", [
    ("slab", dict(mono_energy=6.0), 1, 20), ("slab", dict(mono_energy=6.0), 1, 2400),
    ("ct", dict(mono_energy=12.0), 1, 60_000), ("ct", dict(mono_energy=4.0, charge=1), 1, 3000),
    ("slab", dict(mono_energy=8.0, charge=-1), 1, 37), ("slab", dict(mono_energy=5.0), 5, 5000),
    ("ct", dict(mono_energy=10.0), 20, 500),
    # cascades of split rays deeper than a lane's stack (bremsstrahlung and
    # scattered photons of 18 MeV photons in water)
    ("water", dict(mono_energy=18.0), 64, 3000)])
def test_dose_independent_of_where_particles_run(kind, source, nsplit, histories):
    from ompmc_b200.engine import EVENT_FP32, Engine
    ph = cases._phantom(kind, 32, 5.0)
    tables = cases._tables(tuple(ph.media))
    ref = None
    for kw in FORMS:
        eng = Engine(tables, ph, nsplit=nsplit, **kw)
        dose, unc, st = eng.run_beam(histories, 2, seed=12345, mode=EVENT_FP32,
                                     collimator=(-2.0, 2.0, -3.0, 3.0), **source)
        eng.close()
        assert st["flags"] == 0
        if ref is None:
            ref = dose
            assert (dose > 0).sum() > 10
        assert np.array_equal(dose > 0, ref > 0), kw
        np.testing.assert_allclose(dose, ref, rtol=1e-9, err_msg=str(kw))
