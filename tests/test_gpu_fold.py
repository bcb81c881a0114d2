"""The fold's division by a reciprocal against numpy's: exact equality over masses
and history counts from the smallest to the largest an engine meets, quanta of one
to 2^52, ragged column lengths, several columns and batches."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from pyradmc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols,n_vox,n_batches", [(1, 1, 1), (3, 4095, 2), (2, 4097, 7), (5, 70_001, 3)])
def test_fold_equals_numpy(gpu, n_cols, n_vox, n_batches):
    rng = np.random.default_rng(n_vox)
    mass = 10.0 ** rng.uniform(-9.0, 6.0, n_vox)
    mass[rng.random(n_vox) < 0.01] = 0.0
    per_batch = np.floor(10.0 ** rng.uniform(0.0, 9.0, n_cols)).clip(1)
    q = np.floor(2.0 ** rng.uniform(0.0, 52.0, (n_batches, n_cols, n_vox))).astype(np.int64)
    q[rng.random(q.shape) < 0.3] = 0
    s1, s2 = np.zeros((n_cols, n_vox)), np.zeros((n_cols, n_vox))
    for b in range(n_batches):
        with np.errstate(divide="ignore", invalid="ignore"):
            d = np.where(mass > 0.0, (q[b] * 1.0e-9) / (mass[None, :] * per_batch[:, None]), 0.0)
        s1 += d
        s2 += d * d
    mean = s1 / n_batches
    var = np.maximum(0.0, s2 / n_batches - mean * mean)
    sigma = np.sqrt(var * n_batches / (n_batches - 1) / n_batches) if n_batches > 1 else np.zeros_like(mean)
    lib, e = _lib.load(), C.c_void_p()
    assert lib.pmc_create(C.byref(e), int(gpu.split(":")[1])) == 0
    got_mean, got_sigma, total = np.empty_like(mean), np.empty_like(mean), C.c_int64()
    try:
        assert lib.pmc_reduce_dense(e, _lib.ptr(q, C.c_int64), n_batches, n_cols, n_vox, _lib.ptr(mass, C.c_double),
                                    _lib.ptr(per_batch, C.c_double), _lib.ptr(got_mean, C.c_double),
                                    _lib.ptr(got_sigma, C.c_double), C.byref(total)) == 0
    finally:
        lib.pmc_destroy(e)
    assert np.array_equal(got_mean, mean) and np.array_equal(got_sigma, sigma)
    assert total.value == int(q.sum())


@pytest.mark.parametrize("mass", [np.inf, 1e300, 1e280, 1e-280, 1e-300, 3e-310, 5e-324, np.nan, -1.0])
@pytest.mark.parametrize("per_batch", [1.0, 1e9])
def test_masses_that_no_tissue_has_equal_numpy(gpu, mass, per_batch):
    """One voxel of such a mass among ordinary ones: an infinite mass takes no dose, a
    tiny one all that float64 holds, and the ordinary ones keep theirs."""
    masses = np.array([1.25, mass, 0.75, 0.0, 3e-4])
    q = np.array([[1, 2, 0, 5, 1 << 50], [3, 1 << 40, 7, 1, 0]], dtype=np.int64)
    with np.errstate(all="ignore"):
        d = np.where((masses > 0.0) & (q != 0), (q * 1.0e-9) / (masses * per_batch), 0.0)
        mean = d.sum(axis=0) / 2
        s2 = (d * d).sum(axis=0)
        sigma = np.sqrt(np.maximum(0.0, s2 / 2 - mean * mean) * 2 / 1 / 2)
    lib, e = _lib.load(), C.c_void_p()
    assert lib.pmc_create(C.byref(e), int(gpu.split(":")[1])) == 0
    got_mean, got_sigma, total, n = np.empty(5), np.empty(5), C.c_int64(), np.array([per_batch])
    try:
        assert lib.pmc_reduce_dense(e, _lib.ptr(q, C.c_int64), 2, 1, 5, _lib.ptr(masses, C.c_double),
                                    _lib.ptr(n, C.c_double), _lib.ptr(got_mean, C.c_double),
                                    _lib.ptr(got_sigma, C.c_double), C.byref(total)) == 0
    finally:
        lib.pmc_destroy(e)
    assert np.array_equal(got_mean, mean)
    finite = np.isfinite(s2)  # (squares of a tiny mass's doses overflow)
    assert np.array_equal(got_sigma[finite], sigma[finite]) and total.value == int(q.sum())


def test_a_scoring_grid_with_an_infinite_mass(gpu):
    """Through the engine: the voxel takes no dose, the others what they take beside an
    ordinary one, and a later run without the grid is an ordinary one again."""
    import pyradmc_b200 as P

    grid = P.VoxelGrid.uniform_water((6, 5, 7), (1.0, 1.0, 1.0))
    engine = P.B200Engine(grid, P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material()), device=gpu)
    source = P.ParallelBeamSource(6.0, -1.0, (0.0, 6.0), (0.0, 5.0))
    want = engine.run(source, 4_000, 4, 3)
    mass = np.array(P.ScoringGrid.for_grid(grid).voxel_mass)
    mass[2, 3, 4] = np.inf
    scoring = P.ScoringGrid(grid.shape, grid.spacing, grid.origin, mass)
    got = engine.run(source, 4_000, 4, 3, scoring_grid=scoring)
    assert want.dose[2, 3, 4] > 0 and got.dose[2, 3, 4] == 0
    keep = np.isfinite(mass)
    assert np.array_equal(got.dose[keep], want.dose[keep]) and np.array_equal(got.dose_sigma[keep], want.dose_sigma[keep])
    assert np.array_equal(engine.run(source, 4_000, 4, 3).dose, want.dose)
