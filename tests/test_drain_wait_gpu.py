"""A block of the drain that gives up waiting may leave particles undone that
others hand over to it, so the run and the server step then fail with a
status; the engine stays usable, and the next run gives the dose as before.
The wait is cut short on the host (omc_drain_polls): every block leaves by
itself, none hangs."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


def test_abandoned_drain_is_an_error():
    from ompmc_b200.engine import EVENT_FP32, Engine, OmcError, Server, lib
    ph = cases._phantom("slab", 32, 5.0)
    eng = Engine(cases._tables(tuple(ph.media)), ph)
    call = dict(mono_energy=8.0, charge=-1, collimator=(-2.0, 2.0, -2.0, 2.0))
    ref, _, _ = eng.run_beam(400, 2, seed=3, mode=EVENT_FP32, **call)
    assert ref.max() > 0
    assert lib().omc_drain_polls(eng.h, 1) == 0
    with pytest.raises(OmcError) as err:
        eng.run_beam(400, 2, seed=3, mode=EVENT_FP32, **call)
    assert err.value.status == -12 and "gave up" in str(err.value)
    server = Server(eng, max_requests=2, seed=5)
    server.submit_beam(400, 2, seed=9, **call)
    with pytest.raises(OmcError) as err:
        while server.step(8) > 0:
            pass
    assert err.value.status == -12
    server.close()
    assert lib().omc_drain_polls(eng.h, 0) == 0
    assert lib().omc_drain_polls(eng.h, -1) == -1
    dose, _, st = eng.run_beam(400, 2, seed=3, mode=EVENT_FP32, **call)
    assert st["flags"] == 0
    np.testing.assert_allclose(dose, ref, rtol=1e-9)
    eng.close()
