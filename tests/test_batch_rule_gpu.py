"""The batch's choice of tiles by the number of items, on both sides of its line.

States are compared for equality with the oracle (FP32) and with a
mixed-precision GridSolver (FP16): the tiles' shape does not enter a pixel's
arithmetic.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

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
