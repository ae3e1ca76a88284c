"""Rays just split do not go to the drain, where a lane works off their
sub-photons one after the other, unless its warps hold them all at once: a
run or a load of more of them stays in cycles, each of which works off one
sub-photon of a ray, until the last ray injected is through."""
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsplit,histories,waits", [(64, 3000, True), (20, 3000, True), (20, 1000, False), (5, 3000, False)])
def test_split_rays_are_not_drained_at_once(nsplit, histories, waits):
    from ompmc_b200.engine import EVENT_FP32, Engine, Server
    ph = cases._phantom("water", 32, 10.0)
    tables = cases._tables(tuple(ph.media))
    eng = Engine(tables, ph, nsplit=nsplit, profile=True)
    _, _, st = eng.run_beam(histories, 2, seed=6, mode=EVENT_FP32, mono_energy=18.0)
    cycles = len(eng.profile_trace()) - 1
    eng.close()
    assert st["flags"] == 0
    assert (cycles >= nsplit) if waits else (cycles <= 2)
    eng = Engine(tables, ph, nsplit=nsplit)
    server = Server(eng, max_requests=1, seed=6)
    for load in range(2):
        before = server.stats()
        server.submit_beam(histories, 2, mono_energy=18.0, seed=6)
        while server.step(2) > 0:
            pass
        after = server.stats()
        assert after["drains"] == before["drains"] + 1
        assert (after["cycles"] - before["cycles"] >= nsplit) == waits
    server.close()
    eng.close()
