"""Steps too short for the autotuner: launches at first, the flow kernel once
256 sweeps have been asked for since the reset; the oracle's states, bit for
bit, through the change and after a new reset."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

pytestmark = pytest.mark.gpu


def _inputs(n, m, seed):
    rng = np.random.default_rng(seed)
    mask = (rng.random((n, m)) < 0.97).astype(np.int32)
    mask[n // 2:, m // 3:] = 1
    mask[: n // 4, : m // 4] = 0
    tgt = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    grad[mask == 0] = 0
    return mask, tgt, grad


@pytest.mark.parametrize("size,flow", [((845, 850), True), ((100, 8000), True), ((1800, 1800), True),
                                       ((1801, 1800), False)])
def test_kernel_by_the_sweeps_since_the_reset(size, flow):
    from fpie_gb300 import backend

    s = backend.GridSolver(8, 8)
    late = "p16w8k12d" if flow else "p16w8k16"
    for seed in (1, 2):
        mask, tgt, grad = _inputs(*size, seed)
        s.reset(mask.size, mask, tgt, grad)
        assert s.resident == ""
        o = cjacobi.CGrid(mask, tgt, grad)
        for k, kernel in ((100, "p16w8k16"), (155, "p16w8k16"), (1, late), (13, late)):
            s.step(k)
            o.sweep(k)
            assert s.kernel == kernel
            np.testing.assert_array_equal(s.state(), o.x)
