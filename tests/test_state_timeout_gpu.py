"""A device wait that gave up is raised by the next call that reads the state or
waits for the stream, once, for grids and equation systems."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(n, m):
    from fpie_gb300 import backend

    rng = np.random.default_rng(n)
    mask = np.zeros((n, m), np.int32)
    mask[1:-1, 1:-1] = 1
    tgt = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, np.zeros_like(tgt))
    return s, lambda: s.reset(mask.size, mask, tgt, np.zeros_like(tgt))


def _equ(n, m):
    from fpie_gb300 import backend

    rng = np.random.default_rng(n)
    src, tgt = (rng.integers(0, 256, (n, m, 3), dtype=np.uint8) for _ in range(2))
    mask = np.full((n, m), 255, np.uint8)
    s = backend.EquSolver(256)
    s.reset_images(src, mask, tgt, (0, 0), (0, 0), "max")
    return s, lambda: s.reset_images(src, mask, tgt, (0, 0), (0, 0), "max")


@pytest.mark.parametrize("make", [_grid, _equ])
@pytest.mark.parametrize("size", [(300, 300), (802, 802)])
@pytest.mark.parametrize("read", ["state", "sync", "step"])
def test_a_wait_that_gave_up_is_raised_once(make, size, read):
    from fpie_gb300 import _abi

    s, reset = make(*size)
    for _ in range(2):
        s.set_spin_limit(0)
        reset()
        s.sweeps(4000)
        with pytest.raises(_abi.FpieTimeoutError):
            {"state": s.state, "sync": s.sync, "step": lambda: s.step(0)}[read]()
        s.sync()
        s.state()
        s.set_spin_limit(1 << 26)
        reset()
        s.sweeps(100)
        s.sync()
        s.state()
        s.step(3)
