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
