"""Truncation of dense columns tile by tile against numpy: column lengths around the
4096-voxel tile and its 256- and 512-entry steps, tiles wholly below the threshold,
empty columns, negative, infinite and NaN entries, no truncation at all."""

from __future__ import annotations

import numpy as np
import pytest

from pyradmc_b200 import denoise_dij

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_vox", [1, 31, 511, 4096, 4097, 8191, 3 * 4096 + 257])
@pytest.mark.parametrize("truncation", [0.0, 1e-3, 0.9])
@pytest.mark.parametrize("odd", [False, True])
def test_truncation_equals_numpy(gpu, n_vox, truncation, odd):
    import torch

    rng = np.random.default_rng(n_vox)
    mean = rng.random((7, n_vox)) ** 8
    mean[rng.random(mean.shape) < 0.5] = 0.0
    mean[1] = 0.0
    mean[2, : n_vox // 2] *= 1e-6
    if odd:
        mean[3] = -mean[3]
        mean[4, ::7] = -5.0
        mean[5, 0] = np.nan
        mean[6, -1] = np.inf
    sigma = rng.random(mean.shape)
    keep = []
    for col in mean:
        positive = col[col > 0.0]  # NaN compares false
        with np.errstate(invalid="ignore"):
            threshold = truncation * (positive.max() if positive.size else 0.0)
            keep.append(np.flatnonzero((col >= threshold) & (col > 0.0)))
    indptr, idx, dose, sig = denoise_dij.compact(torch.from_numpy(mean).to(gpu), torch.from_numpy(sigma).to(gpu),
                                                 truncation)
    assert np.array_equal(np.diff(indptr), [k.size for k in keep])
    assert np.array_equal(idx, np.concatenate(keep))
    assert np.array_equal(dose, np.concatenate([m[k] for m, k in zip(mean, keep)]))
    assert np.array_equal(sig, np.concatenate([s[k] for s, k in zip(sigma, keep)]))
