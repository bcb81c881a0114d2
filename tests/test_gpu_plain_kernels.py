"""The transport kernels of the usual run (dose to medium on the transport grid,
one deposit per half substep) against the general ones, which a deposit
resolution longer than any substep selects without changing a single number."""

from __future__ import annotations

import numpy as np
import pytest

import pyradmc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,spacing", [((1, 1, 1), 3.0), ((7, 3, 33), 0.4), ((40, 40, 40), 0.25)])
@pytest.mark.parametrize("kind,msc,electrons", [("photon", "gs", True), ("photon", "gs", False),
                                                ("electron", "gaussian", True)])
def test_plain_kernels_equal_the_general_ones(gpu, shape, spacing, kind, msc, electrons):
    rng = np.random.default_rng(3)
    grid = P.VoxelGrid(shape=shape, spacing=(spacing,) * 3, density=rng.uniform(0.2, 1.9, shape),
                       material=np.zeros(shape, np.int32))
    xs = P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material())
    src = P.ParallelBeamSource(6.0, -1.0, (0.0, shape[0] * spacing), (0.0, shape[1] * spacing))
    kw = dict(n_histories=20000, n_batches=4, seed=11, primary_kind=kind, msc_model=msc,
              transport_electrons=electrons)
    engine = P.B200Engine(grid, xs, device=gpu)
    plain = engine.run(src, **kw)
    general = engine.run(src, deposit_resolution_cm=1.0e6, **kw)
    assert np.array_equal(plain.dose, general.dose) and np.array_equal(plain.dose_sigma, general.dose_sigma)
    assert plain.energy_deposited == general.energy_deposited > 0
    assert plain.energy_escaped == general.energy_escaped
