"""err is the float32 nearest to a sum that keeps a double's bits: residuals of
1, 2^-24 and 2^-49 sum to just above half way between two floats, so a sum that
drops the last of them rounds to 1 instead of 1 + 2^-23."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PARTS = (1.0, 2.0**-24, 2.0**-49)
EXPECTED = np.float32(np.sum(PARTS))


def _grid(places, shape=(70, 300)):
    """A grid whose residuals are |gradient| (the state is 0)."""
    mask = np.zeros(shape, np.int32)
    grad = np.zeros((*shape, 3), np.float32)
    for order, (i, j) in enumerate(places):
        mask[i, j] = 1
        for c in range(3):
            grad[i, j, c] = PARTS[(order + c) % 3]
    return mask, np.zeros((*shape, 3), np.float32), grad


# The three in one thread, in one warp, in different warps and blocks.
PLACES = [[(5, 8), (5, 9), (5, 10)], [(5, 8), (5, 40), (5, 77)], [(1, 1), (33, 200), (68, 298)],
          [(5, 8), (5, 9), (40, 8)]]


def test_the_premise():
    assert EXPECTED == np.float32(1 + 2.0**-23) != np.float32(PARTS[0] + PARTS[1])


@pytest.mark.parametrize("places", PLACES)
def test_grid(places):
    from fpie_gb300 import backend

    mask, tgt, grad = _grid(places)
    s = backend.GridSolver(8, 8)
    s.reset(mask.size, mask, tgt, grad)
    np.testing.assert_array_equal(s.step(0)[1], [EXPECTED] * 3)
    np.testing.assert_array_equal(s.residual_norms()[1], [np.sum(PARTS)] * 3)


@pytest.mark.parametrize("places", PLACES)
def test_batch(places):
    from fpie_gb300.batch import BatchSolver

    b = BatchSolver(1e9)
    job = b.add(*_grid(places), 0)
    np.testing.assert_array_equal(b.result(job)[1], [EXPECTED] * 3)


@pytest.mark.parametrize("unknowns", [(1, 2, 3), (1, 9, 40), (3, 300, 900)])
def test_equ(unknowns):
    from fpie_gb300 import backend

    A = np.zeros((1000, 4), np.int32)
    X = np.zeros((1000, 3), np.float32)
    B = np.zeros((1000, 3), np.float32)
    for order, k in enumerate(unknowns):
        for c in range(3):
            B[k, c] = PARTS[(order + c) % 3]
    s = backend.EquSolver(256)
    s.reset(1000, A, X, B)
    np.testing.assert_array_equal(s.step(0)[1], [EXPECTED] * 3)
