"""The plain form runs the batches of a call together, and one at a time on a
GPU that has no memory for that: dose runs and dose influence columns then
still give what they give with memory for all (up to the summation order of
the FP64 tallies: 1e-12, and 1e-6 for the uncertainty that differences of
sums make)."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu

BATCHES = 20   # of 8 MB each on the 100^3 voxels below
LEFT = 96 << 20


def _fill():
    """Device memory down to about LEFT bytes."""
    import torch
    held = []
    for _ in range(8):
        free = torch.cuda.mem_get_info()[0] - LEFT
        if free < 4 << 20:
            break
        held.append(torch.empty(free // (2 << 20) * (2 << 20), dtype=torch.uint8, device="cuda"))
    return held


def test_batches_run_one_at_a_time_without_memory():
    import torch
    from ompmc_b200.engine import PLAIN_FP64, Engine, bixel_grid
    ph = cases._phantom("water", 100, 3.0)
    tables = cases._tables(tuple(ph.media))
    bl = bixel_grid(ph, [0.0, 90.0], bixel=2.0, field=(2.0, 2.0))
    bl.update(mono_energy=4.0)

    def calls(eng, nbatch):
        dose, unc, st = eng.run_beam(2000, nbatch, seed=5, mode=PLAIN_FP64, mono_energy=4.0,
                                     collimator=(-4.0, 4.0, -3.0, 3.0))
        assert st["flags"] == 0
        return (dose, unc), eng.run_beamlets(bl, 2000, nbatch, 1e-3, seed=6, mode=PLAIN_FP64)

    eng = Engine(tables, ph)
    (dose, unc), (colptr, rows, vals, var, st) = calls(eng, BATCHES)
    eng.close()
    assert (dose > 0).sum() > 100 and colptr[-1] > 100 and len(colptr) == 3
    eng = Engine(tables, ph)
    calls(eng, 2)                        # its other buffers, and the kernels
    torch.cuda.empty_cache()
    held = _fill()
    try:
        assert torch.cuda.mem_get_info()[0] < 8 * ph.nvox * BATCHES
        (dose1, unc1), (colptr1, rows1, vals1, var1, st1) = calls(eng, BATCHES)
    finally:
        del held
        torch.cuda.empty_cache()
        eng.close()
    np.testing.assert_allclose(dose1, dose, rtol=1e-12)
    np.testing.assert_allclose(unc1[dose > 0], unc[dose > 0], rtol=1e-6, atol=1e-9)
    assert np.array_equal(colptr1, colptr) and np.array_equal(rows1, rows)
    np.testing.assert_allclose(vals1, vals, rtol=1e-12)
    np.testing.assert_allclose(var1, var, rtol=1e-6, atol=1e-30)
    # a launch and a fold each for all batches together or for every batch,
    # and five to finish a column
    assert st["launches"] == 2 * (2 + 5) and st1["launches"] == 2 * (2 * BATCHES + 5)


@pytest.mark.parametrize("n,histories,nbatch", [(64, 2000, 10), (61, 1501, 7), (20, 3000, 4)])
def test_batches_of_a_group_keep_apart(n, histories, nbatch):
    """The batch uncertainty, which a history tallied in another batch than its
    own would change: all batches in one launch, in launches of three (fixed
    scratch, 64^3 voxels) and of four or all (smaller grids)."""
    from ompmc_b200.engine import PLAIN_FP64, Engine
    ph = cases._phantom("water", n, 300.0 / n)
    eng = Engine(cases._tables(tuple(ph.media)), ph)
    call = dict(ncase=histories, nbatch=nbatch, seed=9, mono_energy=4.0, collimator=(-4.0, 4.0, -3.0, 3.0))
    dose, unc, _ = eng.run_beam(mode=PLAIN_FP64, **call)
    dose1, unc1, _ = eng.run_beam_noalloc(**call)
    eng.close()
    hit = dose > 0
    assert hit.sum() > 100 and 0 < unc[hit].min() < 0.9
    np.testing.assert_allclose(dose1, dose, rtol=1e-12)
    np.testing.assert_allclose(unc1[hit], unc[hit], rtol=1e-6, atol=1e-9)
