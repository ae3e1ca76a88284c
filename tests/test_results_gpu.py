"""Results reach the caller's memory whole, whichever way they take: straight
below 8 MB and into pinned memory, through the engine's pinned buffers above,
at sizes on and off their chunks, into arrays that start anywhere.  The same
run has the same dose up to the summation order of the FP64 tallies."""
import numpy as np
import pytest

from ompmc_b200 import assets
from perf import cases

pytestmark = pytest.mark.gpu


def _water(nx, ny, nz):
    xb, yb, zb = (np.round(np.linspace(-10.0, 10.0, n + 1), 6) for n in (nx, ny, nz))
    return assets.Phantom(["H2O521ICRU"], xb, yb, zb + 10.0, np.ones((nz, ny, nx), np.int32), np.ones((nz, ny, nx)), "box")


# 8 MB less a voxel row, 8 MB, a voxel plane more, three chunks for four threads and some, an odd size
@pytest.mark.parametrize("shape", [(128, 64, 127), (128, 64, 128), (128, 64, 129), (93, 101, 137), (211, 103, 97)])
def test_results_take_any_way(shape):
    import torch
    from ompmc_b200.engine import EVENT_FP32, Engine
    ph = _water(*shape)
    eng = Engine(cases._tables(tuple(ph.media)), ph)
    n = ph.nvox
    call = dict(ncase=3000, nbatch=3, seed=8, mode=EVENT_FP32, mono_energy=6.0, collimator=(-8.0, 8.0, -8.0, 8.0))
    pinned = [torch.empty(n, dtype=torch.float64).pin_memory().numpy() for _ in range(2)]
    eng.run_beam(**call, out=tuple(pinned))
    dose, unc = (a.copy() for a in pinned)
    assert (dose > 0).sum() > 1000
    hit = dose > 0
    for offset in (0, 1):
        raw = [np.full(n + 3, -7.0) for _ in range(2)]
        eng.run_beam(**call, out=tuple(r[offset:offset + n] for r in raw))
        for r in raw:
            assert (r[:offset] == -7.0).all() and (r[offset + n:] == -7.0).all()
        got, gotu = (r[offset:offset + n] for r in raw)
        assert np.array_equal(got > 0, hit)
        np.testing.assert_allclose(got, dose, rtol=1e-9)
        np.testing.assert_allclose(gotu[hit], unc[hit], rtol=1e-6, atol=1e-9)
        assert np.array_equal(gotu[~hit], unc[~hit])
    eng.close()
