"""Queue slots by the chunk: runs large enough for chunked pushes and 32-particle
claims (more than 512 input particles per transport block) against the same run
admitted in small windows (single slots, one particle a claim), at one block per
SM and at the default shape, for a photon source, a charged one (its primaries
enter the electron queue) and a fan that partly misses the grid (dead slots)."""

from __future__ import annotations

import numpy as np
import pytest

import pyradmc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("source", ["photons", "electrons", "missing"])
@pytest.mark.parametrize("blocks", [None, 1])
def test_chunked_queues_give_the_same_dose(gpu, source, blocks):
    grid = P.VoxelGrid.uniform_water((20, 17, 23), (0.5, 0.5, 0.5))
    xs = P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material())
    if source == "missing":
        src = P.SpectralBeamSource(P.ali_rogers_varian_6mv(), (5.0, 4.0, -100.0), (5.0, 4.0, 0.0), 18.0, 15.0)
    else:
        src = P.ParallelBeamSource(5.0, -1.0, (0.0, 10.0), (0.0, 8.5))
    n = 400_001 if source != "electrons" else 300_007
    kw = dict(n_histories=n, n_batches=1, seed=5, primary_kind="electron" if source == "electrons" else "photon")
    large = P.B200Engine(grid, xs, device=gpu, blocks_per_sm=blocks).run(src, **kw)
    small = P.B200Engine(grid, xs, device=gpu, chunk_size=50_001).run(src, **kw)
    assert np.array_equal(large.dose, small.dose) and large.energy_deposited == small.energy_deposited > 0
    assert large.energy_escaped == small.energy_escaped and large.energy_emitted == small.energy_emitted
