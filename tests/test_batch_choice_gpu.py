"""Batches of more items than two per SM: tiles of 96x96 or of 112x112 by how the
jobs' sides divide, 16 warps for mixed jobs of one row of tiles; strips of jobs
without unknowns, whose warps do not sweep; states equal to the oracle's."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import cjacobi

pytestmark = pytest.mark.gpu


def _job(n, m, seed):
    rng = np.random.default_rng(seed)
    mask = np.zeros((n, m), np.int32)
    mask[1:-1, 1:-1] = 1
    if seed % 3 == 1:  # 16-row strips of a region without unknowns, between others
        mask[n // 3: n // 3 + 33] = 0
    t = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    g = rng.uniform(-20, 20, (n, m, 3)).astype(np.float32)
    g[mask == 0] = 0
    return mask, t, g


@pytest.mark.parametrize("sides,count,kernel", [((110, 110), 60, "p16w8k8"), ((100, 100), 60, "p16w8k8"),
                                                ((290, 300), 16, "p16w8k8"), ((90, 90), 120, "p16w8k16"),
                                                ((150, 150), 40, "p16w8k16"), ((96, 97), 120, "p16w8k16"),
                                                ((600, 600), 3, "p16w8k16")])
def test_choice_in_fp32(sides, count, kernel):
    from fpie_gb300.batch import BatchSolver

    jobs = [_job(*sides, k) for k in range(count)]
    b = BatchSolver(8e9)
    ids = [b.add(*j, 90) for j in jobs]
    b.run(33)
    assert b.kernel == kernel
    b.run()
    for jid, j in list(zip(ids, jobs))[:: max(1, count // 8)]:
        o = cjacobi.CGrid(*j)
        o.sweep(90)
        np.testing.assert_array_equal(b.state(jid), o.x)


@pytest.mark.parametrize("sides,count,kernel", [((96, 90), 120, "p8w16k16"), ((97, 90), 120, "p16w8k16"),
                                                ((110, 110), 60, "p16w8k8")])
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
def test_choice_in_mixed_precision(sides, count, kernel, precision):
    from fpie_gb300 import backend
    from fpie_gb300.batch import BatchSolver

    jobs = [_job(*sides, k) for k in range(count)]
    b = BatchSolver(8e9, precision=precision)
    ids = [b.add(*j, 150) for j in jobs]
    b.run()
    assert b.kernel == kernel
    for jid, j in list(zip(ids, jobs))[::20]:
        s = backend.GridSolver(8, 8)
        s.set_precision(precision)
        s.set_kernel(kernel)  # a 16-bit correction is rounded once per level
        s.reset(j[0].size, *j)
        s.step(150)
        np.testing.assert_array_equal(b.state(jid), s.state())


def test_epochs_of_an_emptying_batch():
    """The choice changes while jobs end; every state is the oracle's."""
    from fpie_gb300.batch import BatchSolver

    sizes = [(110, 110)] * 30 + [(33, 200), (60, 60), (230, 97), (130, 131)] * 6
    jobs = [(*_job(*z, k), 40 + 13 * k % 230) for k, z in enumerate(sizes)]
    b = BatchSolver(8e9)
    ids = [b.add(*j) for j in jobs]
    seen = set()
    for _ in range(8):
        b.run(37)
        seen.add(b.kernel)
    assert len(seen) > 1
    for jid, (mask, t, g, sweeps) in zip(ids, jobs):
        assert b.progress(jid) == (sweeps, sweeps)
        o = cjacobi.CGrid(mask, t, g)
        o.sweep(sweeps)
        np.testing.assert_array_equal(b.state(jid), o.x)


@pytest.mark.parametrize("sweeps,kernel", [(5120, "p16w8k8"), (5121, "p16w8k16")])
def test_levels_that_do_not_fit_the_queue_tables(sweeps, kernel):
    from fpie_gb300.batch import BatchSolver

    jobs = [_job(100, 105, k) for k in range(60)]
    b = BatchSolver(8e9)
    ids = [b.add(*j, sweeps) for j in jobs]
    b.run()
    assert b.kernel == kernel
    for k in (7, 30):
        o = cjacobi.CGrid(*jobs[k])
        o.sweep(sweeps)
        np.testing.assert_array_equal(b.state(ids[k]), o.x)
