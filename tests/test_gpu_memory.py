"""Calls on a GPU that is nearly full.  Batches share waves where the device has room
for a wave's quanta maps and queues; where it has not, a call that fits batch by batch
runs batch by batch and gives the same numbers, also when the memory it needs is held
by maps that an earlier call of the engine left behind."""

from __future__ import annotations

import gc

import numpy as np
import pytest

import pyradmc_b200 as P

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _leave(gpu, nbytes):
    """Device memory held so that about `nbytes` are free."""
    import torch

    gc.collect()
    torch.cuda.synchronize(gpu)
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info(gpu)[0] - nbytes, dtype=torch.uint8, device=gpu)


def _release(held):
    import torch

    held.clear()
    torch.cuda.empty_cache()


def _engine(gpu, shape, **kw):
    grid = P.VoxelGrid.uniform_water(shape, (0.5, 0.5, 0.5))
    return P.B200Engine(grid, P.AnalyticWaterTables(geometry_densities=grid.max_density_by_material()), device=gpu, **kw)


def _same(a, b, names):
    for name in names:
        assert np.array_equal(getattr(a, name), getattr(b, name)), name


DIJ = ("indptr", "indices", "dose", "sigma")


def test_a_dij_without_room_for_its_waves_maps_runs_batch_by_batch(gpu):
    """100 columns of 64^3: 200 MB a map.  Two batches' maps and queues take 1.33 GB,
    one batch's 0.89; with 1.1 GB free the second map fits and the sums after it do not."""
    src = P.BeamletGridSource(6.0, -1.0, (11.0, 21.0), (11.0, 21.0), 10, 10)
    run = lambda e: e.run_dij(src, 1_000, 2, 20260711, beamlet_group_size=100)  # noqa: E731
    want = run(_engine(gpu, (64, 64, 64)))
    engine = _engine(gpu, (64, 64, 64))
    engine.run(P.PencilBeamSource(6.0, (16.0, 16.0, -1.0), (0.0, 0.0, 1.0)), 100, 2, 1)  # its small buffers
    held = [_leave(gpu, 1100 * MB)]
    try:
        got = run(engine)
    finally:
        _release(held)
    _same(got, want, DIJ)


def test_a_run_without_room_for_a_waves_queues_runs_batch_by_batch(gpu):
    """A wave's admission window of 1e6 primaries takes 4.4 GB of queues, a batch's 0.5."""
    src = P.ParallelBeamSource(6.0, -1.0, (0.0, 8.0), (0.0, 8.0))
    want = _engine(gpu, (16, 16, 16)).run(src, 1_000_000, 10, 3)
    engine = _engine(gpu, (16, 16, 16))
    engine.run(src, 100, 2, 1)
    held = [_leave(gpu, 1500 * MB)]
    ticks = []
    try:
        got = engine.run(src, 1_000_000, 10, 3, progress=ticks.append)
    finally:
        _release(held)
    _same(got, want, ("dose", "dose_sigma"))
    assert [t.histories_done for t in ticks] == [100_000 * k for k in range(1, 11)]


def test_maps_of_an_earlier_call_are_given_back_where_the_next_needs_the_room(gpu):
    """Twenty batches' maps of one 128^3 column (335 MB) stay with the engine; nine
    columns' sums (302 MB) then do not fit the 200 MB left unless those go first."""
    src = P.BeamletGridSource(6.0, -1.0, (25.0, 39.0), (25.0, 39.0), 3, 3)
    run = lambda e: e.run_dij(src, 100, 1, 20260711, beamlet_group_size=9)  # noqa: E731
    want = run(_engine(gpu, (128, 128, 128)))
    engine = _engine(gpu, (128, 128, 128))
    engine.run(P.PencilBeamSource(6.0, (32.0, 32.0, -1.0), (0.0, 0.0, 1.0)), 20_000, 20, 1)
    held = [_leave(gpu, 200 * MB)]
    try:
        got = run(engine)
    finally:
        _release(held)
    _same(got, want, DIJ)


def test_queues_sized_by_the_caller_are_not_refused_for_a_waves_window(gpu):
    """chunk_size above a batch and 70,000 slots a primary: one batch's 1,000 primaries
    can be numbered, a wave's 32,000 could not."""
    src = P.PencilBeamSource(6.0, (4.0, 4.0, -1.0), (0.0, 0.0, 1.0))
    want = _engine(gpu, (16, 16, 16)).run(src, 32_000, 32, 3)
    got = _engine(gpu, (16, 16, 16), chunk_size=1_000_000, queue_factor=70_000).run(src, 32_000, 32, 3)
    _same(got, want, ("dose", "dose_sigma"))
    with pytest.raises(ValueError, match="queue index range"):
        _engine(gpu, (16, 16, 16), chunk_size=1_000_000, queue_factor=70_000).run(src, 3_200_000, 32, 3)
