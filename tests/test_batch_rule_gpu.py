"""The batch's choice of tiles by the number of items, on both sides of its line.

States are compared for equality with the oracle (FP32) and with a
mixed-precision GridSolver (FP16): the tiles' shape does not enter a pixel's
arithmetic.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi, np_jacobi

pytestmark = pytest.mark.gpu

TILE_H, TILE_W = 32, 96  # the small regions' tiles


def _job(n, m, sweeps, seed):
    rng = np.random.default_rng(seed)
    mask = np.ones((n, m), np.int32)
    mask[0] = mask[-1] = 0
    mask[:, 0] = mask[:, -1] = 0
    t = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    g = rng.uniform(-20, 20, (n, m, 3)).astype(np.float32)
    g[mask == 0] = 0
    return mask, t, g, sweeps


def _tiles(n, m):
    # Tiles start at the crop's border and hold a masked pixel unless they
    # lie wholly in its last row or column.
    rows = sum(1 for r in range(0, n, TILE_H) if r < n - 1)
    return rows * sum(1 for c in range(0, m, TILE_W) if c < m - 1)


def _mix(over):
    import torch

    line = 2 * torch.cuda.get_device_properties(0).multi_processor_count // 3
    jobs, tiles = [], 0
    # Ragged and exact sizes: one tile, one pixel over, many tiles.
    for k, (n, m) in enumerate([(32, 96), (33, 97), (3, 3), (31, 200), (320, 100)] * 40):
        if tiles + _tiles(n, m) > line:
            break
        jobs.append(_job(n, m, 16 * k % 70 + 5, k))
        tiles += _tiles(n, m)
    while tiles < line:  # up to the line itself, one tile a job
        jobs.append(_job(20, 30, 33, 1000 + tiles))
        tiles += 1
    if over:
        jobs.append(_job(20, 30, 33, 5000))
    return jobs


@pytest.mark.parametrize("over,name", [(False, "p8w8k16"), (True, "p16w8k16")])
def test_choice_and_states_on_both_sides_of_the_line(over, name):
    from fpie_gb300.batch import BatchSolver

    jobs = _mix(over)
    b = BatchSolver(4e9)
    ids = [b.add(*j) for j in jobs]
    b.run(5)
    assert b.kernel == name
    b.run()
    for jid, (mask, t, g, sweeps) in zip(ids, jobs):
        o = cjacobi.CGrid(mask, t, g)
        o.sweep(sweeps)
        np.testing.assert_array_equal(b.state(jid), o.x)


def test_small_regions_mixed_equal_the_solver():
    from fpie_gb300 import backend
    from fpie_gb300.batch import BatchSolver

    jobs = [_job(32, 96, 130, 1), _job(97, 193, 64, 2), _job(3, 3, 7, 3), _job(150, 220, 300, 4)]
    b = BatchSolver(4e9, precision="fp16")
    ids = [b.add(*j) for j in jobs]
    b.run()
    assert b.kernel == "p8w8k16"
    for jid, (mask, t, g, sweeps) in zip(ids, jobs):
        s = backend.GridSolver(8, 8)
        s.set_precision("fp16")
        s.set_kernel("p16w8k16")
        s.reset(mask.size, mask, t, g)
        s.step(sweeps)
        np.testing.assert_array_equal(b.state(jid), s.state())


def _decaying(n, m):
    """Islands of 3x3 unknowns on black: values halve every two sweeps, through
    2^-60 and the subnormals to 0; beside them a solid part."""
    rng = np.random.default_rng(n)
    mask = np.zeros((n, m), np.int32)
    for r in range(2, n - 5, 7):
        for c in range(2, m // 2 - 5, 7):
            mask[r:r + 3, c:c + 3] = 1
    mask[3:n - 3, m // 2:m - 3] = 1
    mask[n // 2, m // 2 - 6:m // 2] = 1
    t = np.where(mask[..., None] != 0, rng.uniform(0, 255, (n, m, 3)), 0).astype(np.float32)
    g = np.zeros((n, m, 3), np.float32)
    g[:, m // 2:] = rng.uniform(-30, 30, (n, m - m // 2, 3))
    g[mask == 0] = 0
    return mask, t, g, 400


@pytest.mark.parametrize("kernel", ["p8w8k16", "p16w8k16", "p16w8k8"])
@pytest.mark.parametrize("limit", [-1, 37, 160])
def test_jobs_outside_the_quartered_range(kernel, limit):
    """Values that leave the range in which quartered sums are exact, within a
    run and between runs, and inputs that never were in it; ordinary jobs
    beside them."""
    from fpie_gb300.batch import BatchSolver

    jobs = [_decaying(100, 130), _job(90, 120, 171, 1), _decaying(40, 64)]
    for kind in ("huge", "inf", "nan", "tiny gradient", "tiny value"):
        mask, t, g, sweeps = _job(70, 150, 65, 3)
        mask[30:34, 40:50] = 0
        g[mask == 0] = 0
        if kind == "huge":
            t *= np.float32(1e36)
            g *= np.float32(1e35)
        elif kind == "inf":
            t[20, 30, 0], t[32, 45, 1] = np.inf, -np.inf
        elif kind == "nan":
            t[20, 30, 0] = np.nan
        elif kind == "tiny gradient":
            t[:] = 0
            g *= np.float32(1e-43)
        else:
            t[:] = np.float32(1e-37) * t
            g[:] = 0
        jobs.append((mask, t, g, sweeps))
    b = BatchSolver(4e9)
    b.set_kernel(kernel)
    ids = [b.add(*j) for j in jobs]
    for _ in range(400 // limit + 1 if limit > 0 else 1):
        b.run(limit)
    for jid, (mask, t, g, sweeps) in zip(ids, jobs):
        assert b.progress(jid) == (sweeps, sweeps)
        o = np_jacobi.GridJacobi(mask, t, g)
        o.sweep(sweeps)
        np.testing.assert_array_equal(b.state(jid), o.x)
