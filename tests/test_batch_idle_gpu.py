"""Batch jobs with strips of rows without unknowns, whose warps only take part in
the barriers: states equal to the oracle's, through even and odd remainders."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

pytestmark = pytest.mark.gpu


def _job(n, m, rows, seed):
    """Unknowns in the given spans of rows only; ordinary values everywhere."""
    rng = np.random.default_rng(seed)
    mask = np.zeros((n, m), np.int32)
    for a, b in rows:
        mask[a:b, 1:-1] = 1
    t = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    g = rng.uniform(-20, 20, (n, m, 3)).astype(np.float32)
    g[mask == 0] = 0
    return mask, t, g


@pytest.mark.parametrize("kernel", ["p8w8k16", "p16w8k16", "p16w8k8"])
def test_strips_without_unknowns(kernel):
    from fpie_gb300.batch import BatchSolver

    jobs = [_job(60, 60, [(1, 59)], 1), _job(128, 90, [(1, 17), (64, 65), (100, 127)], 2),
            _job(200, 130, [(95, 97)], 3), _job(300, 40, [(0, 1), (298, 300)], 4),
            _job(97, 97, [(48, 96)], 5)]
    b = BatchSolver(2e9)
    b.set_kernel(kernel)
    ids = [b.add(*j, 80) for j in jobs]
    oracles = [cjacobi.CGrid(*j) for j in jobs]
    for k in (1, 2, 17, 32, 28):
        b.run(k)
        for jid, o in zip(ids, oracles):
            o.sweep(k)
            np.testing.assert_array_equal(b.state(jid), o.x)
