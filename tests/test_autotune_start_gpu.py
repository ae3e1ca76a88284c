"""The autotuner starts from what the engine runs by default: a run launches
the same kernels as often, and its dose is the same (up to the summation
order of the FP64 tallies)."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


def test_tuner_starts_from_the_engines_defaults():
    from ompmc_b200 import autotune
    from ompmc_b200.engine import EVENT_FP32, Engine
    ph = cases._phantom("slab", 32, 5.0)
    tables = cases._tables(tuple(ph.media))
    assert all(v in autotune.SPACE[k] for k, v in autotune.DEFAULT.items())
    runs = []
    for cfg in ({}, autotune.DEFAULT):
        eng = Engine(tables, ph)
        eng.event_params(**cfg)
        runs.append([eng.run_beam(n, 10, seed=3, mode=EVENT_FP32, mono_energy=6.0, collimator=(-2.0, 2.0, -2.0, 2.0))
                     for n in (200_000, 3_000_000)])
        eng.close()
    for (d0, _, s0), (d1, _, s1) in zip(*runs):
        assert s0["launches"] == s1["launches"] and s0["flags"] == s1["flags"] == 0
        np.testing.assert_allclose(d1, d0, rtol=1e-9)
