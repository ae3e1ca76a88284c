"""A profiled engine counts every transport step, voxel crossing and deposit of
what it ran, wherever the particles ran: in cycles, interactions in a kernel
of their own or in place, or in the drain, in dose runs and on a server.
Trajectories do not depend on that, so the counts are equal to the last one
(deposits over both kinds: a secondary born below the cut-off is deposited
by the kernel that makes it, or by the drain's electron step)."""
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


def _engine(**kw):
    from ompmc_b200.engine import Engine
    ph = cases._phantom("ct", 32, 12.0)
    return Engine(cases._tables(tuple(ph.media)), ph, profile=True, **kw)


def _counts(eng):
    p = eng.profile_last()
    return [p[k][f] for k in ("photon", "electron") for f in ("steps", "cross")] + [p["photon"]["dep"] + p["electron"]["dep"]]


def test_dose_run_counts_its_drain():
    from ompmc_b200.engine import EVENT_FP32
    seen = []
    for kw in (dict(drain_particles=-1), dict(), dict(drain_particles=1 << 22), dict(electron_tsteps=1, tail_boost=1)):
        eng = _engine(**kw)
        _, _, st = eng.run_beam(20_000, 2, seed=4, mode=EVENT_FP32, mono_energy=6.0, collimator=(-3.0, 3.0, -3.0, 3.0))
        assert st["flags"] == 0
        seen.append(_counts(eng))
        eng.close()
    assert min(seen[0]) > 0
    assert all(s == seen[0] for s in seen)


def test_server_counts_its_drain():
    from ompmc_b200.engine import Server
    seen = []
    for kw in (dict(drain_particles=-1), dict(), dict(drain_particles=1 << 22)):
        eng = _engine(**kw)
        server = Server(eng, max_requests=4, seed=2)
        for k in range(6):
            server.submit_beam(4000 + 1000 * k, 4, mono_energy=3.0 + k, seed=50 + k, collimator=(-3.0, 3.0, -3.0, 3.0))
        while server.step(8) > 0:
            pass
        assert (server.stats()["drains"] > 0) == (kw.get("drain_particles") != -1)
        seen.append(_counts(eng))
        server.close()
        eng.close()
    assert min(seen[0]) > 0
    assert all(s == seen[0] for s in seen)
