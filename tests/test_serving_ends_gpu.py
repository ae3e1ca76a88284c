"""The end of a server's load: short loads that are injected and drained in one
step, also where the particles in flight do not hold them, and requests that
finish together, with columns shorter and longer than the server's pinned
buffers hold (78,643 entries) and whole doses between them.  A request's
result depends on its seed alone (up to the summation order of the FP64
tallies), so each is that of a server that runs it by itself in cycles."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


def _setup(n=40, **kw):
    from ompmc_b200.engine import Engine, bixel_grid
    ph = cases._phantom("water", n, 300.0 / n)
    eng = Engine(cases._tables(tuple(ph.media)), ph, **kw)
    # narrow and wide fields: short and long columns
    fields = []
    for bixel in (1.0, 16.0):
        bl = bixel_grid(ph, [20.0], bixel=bixel, field=(2 * bixel, bixel))
        bl.update(mono_energy=6.0)
        fields.append(bl)
    return eng, fields


def _submit(server, sets, what):
    kind, histories, seed = what
    if kind == "dose":
        return server.submit_beam(histories, 4, mono_energy=8.0, seed=seed, collimator=(-3.0, 3.0, -3.0, 3.0))
    return server.submit_beamlet(sets[kind // 2], kind % 2, histories, 4, 0.0, seed=seed)


def _result(server, what, rid):
    return server.result_dense(rid) if what[0] == "dose" else server.result_sparse(rid)


def _compare(a, b):
    if len(a) == 3:
        assert np.array_equal(a[0], b[0])
        np.testing.assert_allclose(a[1], b[1], rtol=1e-9)
        np.testing.assert_allclose(a[2], b[2], rtol=1e-6, atol=1e-30)
    else:
        np.testing.assert_allclose(a[0], b[0], rtol=1e-9)
        hit = b[0] > 0
        np.testing.assert_allclose(a[1][hit], b[1][hit], rtol=1e-6, atol=1e-9)


def _alone(what, n):
    from ompmc_b200.engine import Server
    eng, fields = _setup(n, drain_particles=-1)
    out = []
    for w in what:
        server = Server(eng, max_requests=1, seed=1)
        rid = _submit(server, [server.beamlet_set(f) for f in fields], w)
        while server.step(8) > 0:
            pass
        out.append(_result(server, w, rid))
        server.close()
    eng.close()
    return out


@pytest.mark.parametrize("kw", [dict(), dict(inflight=1 << 12), dict(nsplit=3), dict(drain_particles=3000)])
@pytest.mark.parametrize("n,what", [
    (40, [(0, 50_000, 7)]), (40, [(1, 4, 8), (0, 9_000, 9), ("dose", 20_000, 10)]),
    (70, [(2, 60_000, 11), (0, 8_000, 12), (3, 70_000, 13), ("dose", 30_000, 14), (1, 8_000, 15)])])
def test_requests_that_end_together(n, what, kw):
    from ompmc_b200.engine import Server
    if "nsplit" in kw:
        eng, fields = _setup(n, drain_particles=-1, **kw)
        server = Server(eng, max_requests=8, seed=1)
        ids = [_submit(server, [server.beamlet_set(f) for f in fields], w) for w in what]
        while server.step(8) > 0:
            pass
        ref = [_result(server, w, i) for w, i in zip(what, ids)]
        server.close()
        eng.close()
    else:
        ref = _alone(what, n)
    if n == 70:
        assert max(len(r[0]) for r in ref if len(r) == 3) > 78_643 > min(len(r[0]) for r in ref if len(r) == 3) > 100
    eng, fields = _setup(n, **kw)
    server = Server(eng, max_requests=8, seed=1)
    sets = [server.beamlet_set(f) for f in fields]
    for turn in range(2):   # the second load finds an idle server
        ids = [_submit(server, sets, w) for w in what]
        while server.step(8) > 0:
            pass
        assert sorted(server.completed()) == sorted(ids)
        for w, i, r in zip(what, ids, ref):
            _compare(_result(server, w, i), r)
            server.release(i)
    server.close()
    eng.close()


def test_a_drained_load_is_not_run_again():
    """Two cycles and one drain for a load that the drain holds, however often
    the server is asked; requests that arrive after the drain was queued run."""
    from ompmc_b200.engine import Server
    eng, fields = _setup()
    server = Server(eng, max_requests=4, seed=1)
    bset = server.beamlet_set(fields[0])
    ids = [server.submit_beamlet(bset, k, 20_000, 4, 1e-4, seed=5 + k) for k in range(2)]
    steps = 0
    while server.step(8) > 0:
        steps += 1
    st = server.stats()
    assert steps == 1 and st["finished"] == 2
    assert st["cycles"] == 2 and st["drains"] == 1 and st["launches"] == 2 * 5 + 1 + 2 * 4
    first = server.result_sparse(ids[0])

    server = Server(eng, max_requests=4, seed=1)
    bset = server.beamlet_set(fields[0])
    ids = [server.submit_beamlet(bset, 0, 20_000, 4, 1e-4, seed=5)]
    assert server.step(8) == 1
    ids.append(server.submit_beamlet(bset, 0, 20_000, 4, 1e-4, seed=5))
    while server.step(8) > 0:
        pass
    assert server.completed() == ids
    for i in ids:
        _compare(server.result_sparse(i), first)
    server.close()
    eng.close()
