"""solve() reports a device wait that gave up instead of a sweep count, and the
solver works again after a reset."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

pytestmark = pytest.mark.gpu


def _inputs(n, m, seed):
    rng = np.random.default_rng(seed)
    mask = np.zeros((n, m), np.int32)
    mask[1:-1, 1:-1] = 1
    tgt = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    grad[mask == 0] = 0
    return mask, tgt, grad


@pytest.mark.parametrize("kernel,size", [("auto", (300, 300)), ("p12w8x128k16r", (300, 300)),
                                         ("auto", (802, 802)), ("p16w8k16d", (500, 700))])
@pytest.mark.parametrize("max_sweeps", [1024, 4096])
def test_solve_raises_where_a_wait_gave_up(kernel, size, max_sweeps):
    from fpie_gb300 import _abi, backend

    mask, tgt, grad = _inputs(*size, 3)
    s = backend.GridSolver(8, 8)
    s.set_kernel(kernel)
    s.set_spin_limit(0)
    s.reset(mask.size, mask, tgt, grad)
    with pytest.raises(_abi.FpieTimeoutError):
        s.solve(1e-3, max_sweeps, 1024)
    s.sync()  # the error was reported once
    s.set_spin_limit(1 << 26)
    s.reset(mask.size, mask, tgt, grad)
    assert s.solve(1e-30, 100, 64) == 100
    o = cjacobi.CGrid(mask, tgt, grad)
    o.sweep(100)
    np.testing.assert_array_equal(s.state(), o.x)
