"""Waves of batches: however many batches share a drain, the Dij is the one that
batch-by-batch folds give.  The 48 columns of the 128^3 grid leave room for a
few quanta maps at a time (several waves of several batches), groups of three
columns for all of them at once (one wave, finalized in the fold); odd batch
counts leave a shorter last wave.  Integer quanta and ordered float64 folds:
exact equality."""

from __future__ import annotations

import numpy as np
import pytest

import pyradmc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_batches", [1, 2, 19, 23])
def test_waves_give_the_same_dij(gpu, n_batches):
    grid = P.VoxelGrid.uniform_water((128, 128, 128), (0.25, 0.25, 0.25))
    xs = P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material())
    src = P.BeamletGridSource(6.0, -1.0, (12.0, 20.0), (13.0, 19.0), 8, 6)
    args = (src, 40 * n_batches, n_batches, 20260711)
    whole = P.B200Engine(grid, xs, device=gpu).run_dij(*args, truncation=0.0)
    parts = P.B200Engine(grid, xs, device=gpu).run_dij(*args, truncation=0.0, beamlet_group_size=3)
    for name in ("indptr", "indices", "dose", "sigma"):
        assert np.array_equal(getattr(whole, name), getattr(parts, name)), name
    assert whole.indices.size > 0 and whole.energy_deposited == parts.energy_deposited


@pytest.mark.parametrize("shape,n_batches", [((3, 5, 7), 2), ((16, 16, 16), 10), ((61, 53, 87), 7)])
def test_waves_give_the_same_run(gpu, shape, n_batches):
    """Forward runs fold straight into the caller's dense maps: one column of a
    Dij with an untruncated CSC holds the same mean and sigma."""
    grid = P.VoxelGrid.uniform_water(shape, (0.5, 0.5, 0.5))
    xs = P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material())
    x, y = 0.5 * shape[0], 0.5 * shape[1]
    run = P.B200Engine(grid, xs, device=gpu).run(P.ParallelBeamSource(6.0, -1.0, (0.0, x), (0.0, y)),
                                                 500 * n_batches, n_batches, 3)
    dij = P.B200Engine(grid, xs, device=gpu).run_dij(P.BeamletGridSource(6.0, -1.0, (0.0, x), (0.0, y), 1, 1),
                                                     500 * n_batches, n_batches, 3, truncation=0.0)
    assert np.array_equal(dij.column_dense(0), run.dose) and np.array_equal(dij.sigma_dense(0), run.dose_sigma)


def test_progress_of_batches_that_complete_together_and_one_by_one(gpu):
    """One call a batch either way; batches above a wave's 64 primaries per resident
    thread are reported as each is done, not at the end."""
    grid = P.VoxelGrid.uniform_water((8, 8, 8), (0.5, 0.5, 0.5))
    engine = P.B200Engine(grid, P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material()), device=gpu)
    src = P.ParallelBeamSource(6.0, -1.0, (0.0, 4.0), (0.0, 4.0))
    events = []
    engine.run(src, 700, 7, 3, progress=events.append)
    assert [e.histories_done for e in events] == [100 * k for k in range(1, 8)]
    events.clear()
    engine.run(src, 48_000_000, 4, 3, progress=events.append)
    assert [e.histories_done for e in events] == [12_000_000 * k for k in range(1, 5)]
    elapsed = [e.elapsed_s for e in events]
    assert elapsed[0] < 0.7 * elapsed[-1] and elapsed[1] < 0.9 * elapsed[-1]
