"""A batch job's range mark through runs on different kernels: a kernel that
does not look at the values it stores must not leave the next one, whose
quartered sums are exact in a range only, to trust them."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import np_jacobi

pytestmark = pytest.mark.gpu


def _islands(side, count, seed):
    """Islands of side x side unknowns on black; their values decay to the
    subnormals and, but for the smallest islands, stay there."""
    rng = np.random.default_rng(seed)
    n = count * (side + 1) + 1
    mask = np.zeros((n, n), np.int32)
    for r in range(1, n - 1, side + 1):
        for c in range(1, n - 1, side + 1):
            mask[r:r + side, c:c + side] = 1
    t = np.where(mask[..., None] != 0, rng.uniform(0, 255, (n, n, 3)), 0).astype(np.float32)
    return mask, t, np.zeros((n, n, 3), np.float32)


# Sweeps after which the islands' values are between 2^-149 and 2^-123.
@pytest.mark.parametrize("side,first", [(3, 264), (4, 430), (4, 520)])
@pytest.mark.parametrize("unlooked", ["p8w16k16", "p16w8k8"])
@pytest.mark.parametrize("then", ["auto", "p8w8k16", "p16w8k16", "p16w8k8"])
def test_runs_on_different_kernels_equal_the_oracle(side, first, unlooked, then):
    from fpie_gb300.batch import BatchSolver

    mask, t, g = _islands(side, 20, side)
    o = np_jacobi.GridJacobi(mask, t, g)
    o.sweep(first)
    least = np.abs(o.x[o.x != 0]).min()
    assert 2.0**-149 <= least < 2.0**-120  # where quartered sums round
    b = BatchSolver(1e9)
    job = b.add(mask, t, g, first + 48)
    b.set_kernel(unlooked)
    b.run(first)
    np.testing.assert_array_equal(b.state(job), o.x)
    b.set_kernel(then)
    for k in (16, 5, 27):
        b.run(k)
        o.sweep(k)
        np.testing.assert_array_equal(b.state(job), o.x)
