"""Repeated steps around the number of sweeps up to which they run as launches,
for grids of the shapes that differ in it: the oracle's states through every
change between launches and the resident kernel."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,few", [((38, 40), 5), ((194, 190), 16), ((300, 400), 17), ((333, 517), 20),
                                      ((176, 1457), 32), ((600, 610), 64), ((802, 802), 17)])
def test_states_around_the_line(size, few):
    from fpie_gb300 import backend

    rng = np.random.default_rng(few)
    mask = (rng.random(size) < 0.9).astype(np.int32)
    tgt = rng.uniform(0, 255, (*size, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (*size, 3)).astype(np.float32)
    grad[mask == 0] = 0
    s = backend.GridSolver(8, 8)
    for _ in range(2):
        s.reset(mask.size, mask, tgt, grad)
        assert s.resident
        o = cjacobi.CGrid(mask, tgt, grad)
        launches = []
        for k in (few, few, few + 1, few, 1, few + 1, few + 1):
            before = s.launches
            s.sweeps(k)
            launches.append(s.launches - before)
            o.sweep(k)
            np.testing.assert_array_equal(s.state(), o.x)
        # The reset's first short step and those over the line are one launch.
        assert launches[2] == launches[5] == launches[6] == 1
        assert launches[3] == -(-few // 16)
