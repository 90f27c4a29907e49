"""The look for inputs outside the quartered range: only where a resident step
follows, and then on the state that it starts from."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import np_jacobi

pytestmark = pytest.mark.gpu


def _inputs(n, m, seed):
    rng = np.random.default_rng(seed)
    mask = (rng.random((n, m)) < 0.9).astype(np.int32)
    mask[0] = mask[-1] = mask[:, 0] = mask[:, -1] = 0
    tgt = rng.uniform(0, 255, (n, m, 3)).astype(np.float32)
    grad = rng.uniform(-30, 30, (n, m, 3)).astype(np.float32)
    grad[mask == 0] = 0
    return mask, tgt, grad


def _wild(kind, mask, tgt, grad):
    if kind == "huge":
        tgt, grad = tgt * np.float32(1e36), grad * np.float32(1e35)
    elif kind == "inf":
        tgt = tgt.copy()
        tgt[20, 30, 0], tgt[0, 45, 1] = np.inf, -np.inf
    elif kind == "nan":
        tgt = tgt.copy()
        tgt[20, 30, 0] = np.nan
    else:
        tgt, grad = tgt * 0, grad * np.float32(1e-43)
    return mask, tgt, grad


@pytest.mark.parametrize("kind", ["huge", "inf", "nan", "tiny gradient"])
@pytest.mark.parametrize("first", ["p16w8k16", "sweep1", "few", "fp16 and back", "nothing"])
def test_inputs_out_of_range_after_other_kernels(kind, first):
    from fpie_gb300 import backend

    s = backend.GridSolver(8, 8)
    for seed, what in ((1, kind), (2, "ordinary"), (3, kind)):
        arrays = _inputs(70, 190, seed)
        if what != "ordinary":
            arrays = _wild(what, *arrays)
        s.reset(arrays[0].size, *arrays)
        o = np_jacobi.GridJacobi(*arrays)
        steps = [40, 21]
        if first == "few":
            steps = [1, 2, 3] + steps
        elif first == "fp16 and back":
            s.set_precision("fp16")
            s.set_precision("fp32")
        elif first != "nothing":
            s.set_kernel(first)
            s.step(9)
            s.set_kernel("auto")
            with np.errstate(all="ignore"):
                o.sweep(9)
        assert s.resident
        with np.errstate(all="ignore"):
            for k in steps:
                s.step(k)
                o.sweep(k)
                np.testing.assert_array_equal(s.state(), o.x)


def _launches(s, call):
    before = s.launches
    call()
    return s.launches - before


def test_only_a_resident_step_after_a_float_reset_looks():
    import torch

    from fpie_gb300 import backend

    s = backend.GridSolver(8, 8)
    for size in ((60, 90), (1900, 1800)):
        dev = [torch.from_numpy(a).cuda() for a in _inputs(*size, 4)]
        torch.cuda.synchronize()
        s.reset_tensors(*dev)
        assert _launches(s, lambda: s.reset_tensors(*dev)) == 1
    dev = [torch.from_numpy(a).cuda() for a in _inputs(60, 90, 4)]
    torch.cuda.synchronize()
    s.reset_tensors(*dev)
    assert [_launches(s, lambda: s.sweeps(100)) for _ in range(3)] == [2, 1, 1]


@pytest.mark.parametrize("kind", ["huge", "inf", "tiny gradient"])
def test_equation_systems_from_floats(kind):
    from fpie_gb300 import backend

    n, m = 60, 90
    mask = np.zeros((n, m), np.int32)
    mask[1:-1, 1:-1] = 1
    s = backend.EquSolver(256)
    ids = s.partition(mask)
    N = int(ids.max()) + 1
    A = np.zeros((N, 4), np.int32)
    A[1:] = np.stack([ids[:-2, 1:-1], ids[2:, 1:-1], ids[1:-1, :-2], ids[1:-1, 2:]], -1).reshape(-1, 4)
    rng = np.random.default_rng(6)
    X = rng.uniform(0, 255, (N, 3)).astype(np.float32)
    B = rng.uniform(-30, 30, (N, 3)).astype(np.float32)
    X[0] = B[0] = 0
    if kind == "huge":
        X, B = X * np.float32(1e36), B * np.float32(1e35)
    elif kind == "inf":
        X[700, 1] = np.inf
    else:
        X, B = X * 0, B * np.float32(1e-43)
    s.reset(N, A, X, B)
    assert s.kernel.startswith("grid:")
    o = np_jacobi.EquJacobi(A, X, B)
    with np.errstate(all="ignore"):
        for k in (40, 21):
            s.step(k)
            o.sweep(k)
            np.testing.assert_array_equal(s.state()[1:], o.X[1:])
